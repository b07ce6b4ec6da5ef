"""The automatic number of subdomains where FP32 limits it: slender, thin and
folded meshes fall back to at least 500 nodes per subdomain and converge, a
slender mesh within FP32's reach and a compact one keep the finer default, and
an operator that the FP32 elimination finds indefinite is no error of the call."""
import numpy as np
import pytest
import scipy.sparse as sp

from axia_gpu import _lib, meshgen
from test_gpu_coarse_inverse_accuracy import folded_bar

pytestmark = pytest.mark.gpu

MIXED = dict(precision=_lib.PREC_MIXED, refine_mode=_lib.REFINE_RELIABLE, matrix_format=_lib.FORMAT_BSR3,
             inner_rtol=0.1, preconditioner=_lib.PRECOND_COARSE)


def _assemble(ctx, m):
    ctx.setup(m)
    ctx.assemble_ex(_lib.ASM_CSR64 | _lib.ASM_BSR64 | _lib.ASM_BSR32)
    rp, col, val, _, _ = ctx.export_system()
    return sp.csr_matrix((val, col, rp), shape=(len(rp) - 1,) * 2)


def _axial(m):
    x = m.coords[:, 0]
    tip = np.nonzero(x > x.max() - 1e-9)[0]
    f = np.zeros(m.ndof)
    f[3 * tip] = 1000.0 / len(tip)
    return f


# (the longest bars are beyond FP32 with updates only every factor 100, whatever the subdomains)
@pytest.mark.parametrize("shape,rtol,inner,few", [
    ((120, 12, 12), 1e-8, 0.1, True), ((132, 12, 12), 1e-8, 0.1, True), ((144, 12, 12), 1e-6, 0.1, True),
    ((128, 8, 8), 1e-6, 0.1, True), ((112, 8, 8), 1e-8, 0.1, True), ((140, 10, 10), 1e-6, 0.1, True),
    ((60, 60, 1), 1e-5, 0.1, True), ((90, 10, 10), 1e-8, 0.1, True), ((72, 8, 8), 1e-8, 0.1, True),
    ((72, 8, 8), 1e-8, 0.01, True), ((80, 8, 8), 1e-8, 0.01, True), ((70, 10, 10), 1e-8, 0.1, False),
    ((40, 4, 4), 1e-8, 0.1, False), ((40, 40, 4), 1e-8, 0.01, False), ((40, 8, 8), 1e-8, 0.01, False)])
def test_bars_and_plates(gpu_ctx, shape, rtol, inner, few):
    m = meshgen.cantilever_c3d8(*shape)
    K, f, free = _assemble(gpu_ctx, m), _axial(m), m.free_mask()
    kw = dict(MIXED, inner_rtol=inner)
    u, info = gpu_ctx.solve(f, rtol=rtol, **kw)
    assert np.linalg.norm(K @ u[free] - f[free]) <= 1.01 * rtol * np.linalg.norm(f[free])
    assert (gpu_ctx.coarse_size()[0] <= m.n_nodes / 500 * 1.2) == few
    # the next assembly keeps the size
    n_sub = gpu_ctx.coarse_size()[0]
    gpu_ctx.assemble_ex(_lib.ASM_BSR64 | _lib.ASM_BSR32)
    again, _ = gpu_ctx.solve(f, rtol=rtol, **kw)
    assert gpu_ctx.coarse_size()[0] == n_sub and np.array_equal(u, again)


@pytest.mark.parametrize("shape", [(3, 28, 4, 8), (3, 40, 2, 8), (4, 24, 2, 6), (3, 40, 3, 9)])
def test_folded_into_a_compact_box(gpu_ctx, shape):
    m = folded_bar(*shape)
    K, free = _assemble(gpu_ctx, m), m.free_mask()
    f = gpu_ctx.load_vector(m) * free
    _, jac = gpu_ctx.solve(f, rtol=1e-3, **dict(MIXED, preconditioner=_lib.PRECOND_JACOBI))
    u, info = gpu_ctx.solve(f, rtol=1e-3, **MIXED)
    assert np.linalg.norm(K @ u[free] - f[free]) <= 1.01e-3 * np.linalg.norm(f)
    assert info.iters <= jac.iters / 2


def test_indefinite_default(gpu_ctx):
    """200x4x4: the FP32 elimination meets a negative pivot with the finer
    default; the call goes on with fewer subdomains and ends by its iterations."""
    m = meshgen.cantilever_c3d8(200, 4, 4)
    _assemble(gpu_ctx, m)
    f = _axial(m)
    with pytest.raises(_lib.AxiaError) as e:
        gpu_ctx.solve(f, rtol=1e-8, max_iter=20, **MIXED)
    assert e.value.code == _lib.ERR_NOT_CONVERGED
    assert 1 <= gpu_ctx.coarse_size()[0] <= m.n_nodes / 500
    with pytest.raises(_lib.AxiaError) as e:  # an explicit size keeps its error
        gpu_ctx.solve(f, rtol=1e-8, max_iter=20, coarse_nodes=100, **MIXED)
    assert e.value.code == _lib.ERR_ZERO_PIVOT


def test_one_slender_mesh_of_a_family(gpu_ctx):
    """A mesh out of reach takes fewer subdomains, its neighbours keep theirs."""
    ms = [meshgen.block_c3d8_pressure(n=14), meshgen.cantilever_c3d8(128, 8, 8), meshgen.block_c3d8_pressure(n=9)]
    ms[1].cload = _axial(ms[1])
    gpu_ctx.setup_multi(ms)
    gpu_ctx.assemble_ex(_lib.ASM_BSR64 | _lib.ASM_BSR32)
    f = np.concatenate([gpu_ctx.load_vector(m) for m in ms])
    u, _, rel, _ = gpu_ctx.solve_multi(f, rtol=1e-6, **MIXED)
    total = gpu_ctx.coarse_size()[0]
    assert (rel <= 1e-6).all() and np.isfinite(u).all()
    alone = []
    for m in ms:
        gpu_ctx.setup(m)
        gpu_ctx.assemble_ex(_lib.ASM_BSR64 | _lib.ASM_BSR32)
        gpu_ctx.solve(gpu_ctx.load_vector(m), rtol=1e-4, **MIXED)
        alone.append(gpu_ctx.coarse_size()[0])
    assert alone[1] <= ms[1].n_nodes / 500 < total
    # the mean row length of the family shifts a count by one box or so
    assert abs(total - sum(alone)) <= 0.35 * sum(alone)


def test_each_matrix_decides_for_itself(gpu_ctx):
    """Density designs of one bar, in reach of FP32 and, with a soft root, out of
    it: a design's subdomains and solution do not depend on the designs before it."""
    m = meshgen.simp_beam(48, 8, 8)
    x = m.coords[:, 0]
    f = np.zeros(m.ndof)
    f[0::3] = x > x.max() - 1e-9
    designs = np.ones((2, m.n_elem))
    designs[1, m.coords[m.conn].mean(axis=1)[:, 0] < 8.0] = 0.4

    def solve(k):
        u, _, info = gpu_ctx.compliance_forward(designs[k], 3.0, 1.0, f, **dict(MIXED, rtol=1e-6))
        return u, info.iters, gpu_ctx.coarse_size()[0]

    def fresh():
        gpu_ctx.setup(m)
        gpu_ctx.assemble_ex(_lib.ASM_BSR64 | _lib.ASM_BSR32)

    alone = []
    for k in (0, 1):
        fresh()
        alone.append(solve(k))
    assert alone[1][2] < alone[0][2]  # the second takes fewer subdomains
    fresh()
    for k in (0, 1, 1, 0, 1, 0, 0):
        u, iters, n_sub = solve(k)
        assert (iters, n_sub) == alone[k][1:]
        assert np.array_equal(u, alone[k][0])
