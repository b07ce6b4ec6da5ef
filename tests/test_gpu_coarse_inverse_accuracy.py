"""The FP32 coarse inverse against exact arithmetic: the mixed two-level solve
takes the iterations of a FP64 CG whose coarse matrix Z^T K Z is inverted in
FP64 (same boxes, same rigid-body modes), from one tile of the inverse to 59 a
side, on a compact block and on folded bars whose coarse operator is
ill-conditioned: there a lost symmetry of the elimination makes the
preconditioner indefinite long before its well-conditioned part shows it."""
import numpy as np
import pytest
import scipy.sparse as sp

from axia_gpu import _lib, meshgen

pytestmark = pytest.mark.gpu

MIXED = dict(precision=_lib.PREC_MIXED, refine_mode=_lib.REFINE_RELIABLE, matrix_format=_lib.FORMAT_BSR3,
             inner_rtol=0.1)


def folded_bar(cols, leg, w, gap):
    """A bar of width w folded through cols x cols legs along z, joined alternately at the top and the bottom,
    clamped at its start; the load pulls at its second and third layer of nodes."""
    p, n = w + gap, cols * w + (cols - 1) * gap
    m = meshgen.cantilever_c3d8(n, n, leg)
    x, y, z = m.coords[m.conn].mean(axis=1).T
    i, j = (x // p).astype(int), (y // p).astype(int)
    inx, iny = x - i * p < w, y - j * p < w
    odd = j % 2 == 1
    first = np.where(odd, cols - 2 - i, i) + j * cols  # of the two legs that a join connects
    joinx = ~inx & iny & np.where(first % 2 == 0, z > leg - w, z < w)
    last = j * cols + cols - 1
    joiny = inx & ~iny & (i == np.where(odd, 0, cols - 1)) & np.where(last % 2 == 0, z > leg - w, z < w)
    m.conn = m.conn[inx & iny | joinx | joiny]
    used = np.unique(m.conn)
    m.conn = np.searchsorted(used, m.conn).astype(np.int32)
    m.coords = m.coords[used]
    m.e_elem = np.full(len(m.conn), 210000.0)
    x, y, z = m.coords.T
    first_leg = (x <= w + 1e-9) & (y <= w + 1e-9)
    m.bc_dof = (3 * np.nonzero(first_leg & (z < 1e-9))[0][:, None] + np.arange(3)).ravel()
    m.bc_val = np.zeros(len(m.bc_dof))
    m.cload = np.zeros(m.ndof)
    m.cload[2::3] = first_leg & (z > 1.5) & (z < 3.5)
    return m


def subdomain_modes(m, target):
    """Orthonormal rigid-body modes of the boxes, on the free DOFs; and how many boxes hold nodes."""
    lo, ext = m.coords.min(0), np.ptp(m.coords, axis=0)
    h = np.cbrt(ext.prod() / target)
    while np.maximum(1, np.ceil(ext / h - 1e-9)).prod() > target:
        h *= 1.02
    n = np.maximum(1, np.ceil(ext / h - 1e-9)).astype(int)
    c = np.minimum(((m.coords - lo) / h).astype(int), n - 1)
    cells, sub = np.unique(np.ravel_multi_index(c.T, n), return_inverse=True)
    free = m.free_mask()
    number = np.cumsum(free) - 1
    data = []
    for k in range(len(cells)):
        a = np.nonzero(sub == k)[0]
        r = (m.coords[a] - m.coords[a].mean(0)) / h
        Z = np.zeros((len(a), 3, 6))
        Z[:, [0, 1, 2], [0, 1, 2]] = 1.0
        Z[:, 1, 3], Z[:, 2, 3] = -r[:, 2], r[:, 1]
        Z[:, 0, 4], Z[:, 2, 4] = r[:, 2], -r[:, 0]
        Z[:, 0, 5], Z[:, 1, 5] = -r[:, 1], r[:, 0]
        dof = (3 * a[:, None] + np.arange(3)).ravel()
        Z = Z.reshape(-1, 6)[free[dof]]
        w, V = np.linalg.eigh(Z.T @ Z)
        keep = w > 1e-9 * max(w.max(), 1e-300)
        data.append((number[dof[free[dof]]], Z @ (V[:, keep] / np.sqrt(w[keep]))))
    cols = np.cumsum([0] + [q.shape[1] for _, q in data])
    Z = sp.csr_matrix((np.concatenate([q.ravel() for _, q in data]),
                       (np.concatenate([np.repeat(d, q.shape[1]) for d, q in data]),
                        np.concatenate([np.tile(np.arange(c, c + q.shape[1]), len(d))
                                        for c, (d, q) in zip(cols, data)]))), shape=(int(free.sum()), cols[-1]))
    return Z, len(cells)


def exact_iterations(K, b, Z, rtol):
    dinv = 1.0 / K.diagonal()
    A = np.linalg.inv((Z.T @ (K @ Z)).toarray())
    x, r = np.zeros_like(b), b.copy()
    z = dinv * r + Z @ (A @ (Z.T @ r))
    p, rz = z.copy(), r @ z
    for it in range(1, 4000):
        q = K @ p
        alpha = rz / (p @ q)
        x += alpha * p
        r -= alpha * q
        if np.linalg.norm(r) <= rtol * np.linalg.norm(b):
            return it
        z = dinv * r + Z @ (A @ (Z.T @ r))
        rz, old = r @ z, rz
        p = z + rz / old * p
    raise AssertionError("no convergence")


def _check(ctx, m, target, rtol):
    ctx.setup(m)
    ctx.assemble_ex(_lib.ASM_CSR64 | _lib.ASM_BSR64 | _lib.ASM_BSR32)
    rp, col, val, _, _ = ctx.export_system()
    K = sp.csr_matrix((val, col, rp), shape=(len(rp) - 1,) * 2)
    free = m.free_mask()
    f = ctx.load_vector(m) * free
    nodes = m.n_nodes // target
    Z, n_sub = subdomain_modes(m, m.n_nodes // nodes)
    want = exact_iterations(K, f[free], Z, rtol)
    u, info = ctx.solve(f, rtol=rtol, preconditioner=_lib.PRECOND_COARSE, coarse_nodes=nodes,
                        max_iter=4 * want, **MIXED)
    assert abs(ctx.coarse_size()[0] - n_sub) <= 0.05 * n_sub  # nodes on the faces of boxes
    # FP32 recurrences cost some iterations, and one reliable update a few
    assert info.iters <= 1.25 * want + 5
    assert np.linalg.norm(K @ u[free] - f[free]) <= 1.01 * rtol * np.linalg.norm(f)


# 1, 1, 2, 5, 12 and 42 or more tiles of 64 unknowns
@pytest.mark.parametrize("target", [1, 8, 18, 48, 120, 640])
def test_compact_block(gpu_ctx, target):
    _check(gpu_ctx, meshgen.cantilever_c3d8(12, 10, 8), target, 1e-8)


@pytest.mark.parametrize("shape,target", [((3, 40, 2, 8), 2), ((4, 24, 2, 6), 4), ((3, 28, 4, 8), 8),
                                          ((3, 16, 4, 3), 27), ((2, 20, 5, 8), 21), ((3, 20, 5, 4), 48)])
def test_folded_bars(gpu_ctx, shape, target):
    _check(gpu_ctx, folded_bar(*shape), target, 1e-3)
