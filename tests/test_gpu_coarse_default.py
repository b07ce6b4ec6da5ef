"""The default size of the two-level preconditioner's subdomains: meshes on
both sides of its steps against the diagonal preconditioner, and the fallback
to larger subdomains where a node row reaches more of them than the operator's
item lists hold."""
import numpy as np
import pytest

from axia_gpu import _lib, meshgen

pytestmark = pytest.mark.gpu

MIXED = dict(precision=_lib.PREC_MIXED, refine_mode=_lib.REFINE_RELIABLE, inner_rtol=0.01,
             matrix_format=_lib.FORMAT_BSR3, rtol=1e-10)


def _both(ctx, m):
    ctx.setup(m)
    ctx.assemble_ex(_lib.ASM_BSR64 | _lib.ASM_BSR32)
    f = ctx.load_vector(m)
    ref, _ = ctx.solve(f, preconditioner=_lib.PRECOND_JACOBI, **MIXED)
    u, _ = ctx.solve(f, preconditioner=_lib.PRECOND_COARSE, **MIXED)
    return np.linalg.norm(u - ref) / np.linalg.norm(ref), ctx.coarse_size()[0]


# 2 and 36 nodes: one subdomain; 343: the 50-node floor; 4096: the power law
@pytest.mark.parametrize("n,subdomains", [(1, (1, 1)), (6, (1, 6)), (15, (8, 36))])
def test_default_subdomains(gpu_ctx, n, subdomains):
    err, n_sub = _both(gpu_ctx, meshgen.block_c3d8_pressure(n=n, perturb=0.1))
    assert subdomains[0] <= n_sub <= subdomains[1]
    assert err <= 1e-8  # both solutions to a residual of 1e-10


def test_row_reaching_many_subdomains(gpu_ctx):
    """A corner node joined to nodes all over the block by 24 more tetrahedra:
    its row reaches over 32 of the default's subdomains."""
    m = meshgen.block_tet(n=22, nn=4)
    x = m.coords
    rng = np.random.default_rng(3)
    extra = []
    far = np.nonzero(np.linalg.norm(x - x[0], axis=1) > 5.0)[0]
    while len(extra) < 24:
        a, b, c = rng.choice(far, 3, replace=False)
        v = np.linalg.det(x[[a, b, c]] - x[0])
        if abs(v) > 50.0:
            extra.append((0, a, b, c) if v > 0 else (0, b, a, c))
    m.conn = np.concatenate([m.conn, np.array(extra, np.int32)])
    m.e_elem = np.concatenate([m.e_elem, np.full(len(extra), 1.0)])
    err, n_sub = _both(gpu_ctx, m)
    assert 1 <= n_sub < 32
    assert err <= 1e-8
    # an explicit size keeps its error, and the context stays usable
    f = gpu_ctx.load_vector(m)
    with pytest.raises(_lib.AxiaError) as e:
        gpu_ctx.solve(f, preconditioner=_lib.PRECOND_COARSE, coarse_nodes=60, **MIXED)
    assert e.value.code == _lib.ERR_INVALID_ARG
    with pytest.raises(_lib.AxiaError):
        gpu_ctx.solve(f, preconditioner=_lib.PRECOND_COARSE, coarse_nodes=60, **MIXED)
    u, _ = gpu_ctx.solve(f, preconditioner=_lib.PRECOND_COARSE, **MIXED)
    assert np.isfinite(u).all()
