"""Systems that run as one thread-block cluster: from one block to the largest
cluster, and on both sides of the sizes where the whole grid takes over, in
FP64 (CSR) and mixed (node blocks, diagonal and two-level) against a direct
solve or each other."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

from axia_gpu import _lib, meshgen

pytestmark = pytest.mark.gpu

MIXED = dict(precision=_lib.PREC_MIXED, refine_mode=_lib.REFINE_RELIABLE, inner_rtol=0.01,
             matrix_format=_lib.FORMAT_BSR3)


# 12 .. 13,872 free DOFs: 1, 1, 2, 4, 8 and 16 blocks; 5.2 k and 6 k rows around
# 400,000 entries; 4,913 and 5,832 nodes around 130,000 node blocks
@pytest.mark.parametrize("n", [1, 2, 3, 5, 7, 10, 11, 12, 16, 17])
def test_one_cluster_and_whole_grid_agree(gpu_ctx, n):
    m = meshgen.block_c3d8_pressure(n=n, perturb=0.1)
    gpu_ctx.setup(m)
    gpu_ctx.assemble_ex(_lib.ASM_CSR64 | _lib.ASM_BSR64 | _lib.ASM_BSR32)
    f = gpu_ctx.load_vector(m)
    rp, col, val, _, _ = gpu_ctx.export_system()
    K = sp.csr_matrix((val, col, rp), shape=(len(rp) - 1,) * 2)
    free = m.free_mask()
    if n <= 12:
        ref = np.zeros(m.ndof)
        ref[free] = spla.spsolve(K.tocsc(), f[free])
    else:
        ref, _ = gpu_ctx.solve(f, rtol=1e-12, matrix_format=_lib.FORMAT_BSR3)
    for kw in (dict(), dict(spmv_lanes=8), MIXED, dict(MIXED, preconditioner=_lib.PRECOND_COARSE)):
        u, info = gpu_ctx.solve(f, rtol=1e-11, **kw)
        # the residual tolerance times the condition of the free system (under 1e3 in this norm)
        assert np.linalg.norm(u - ref) <= 1e-8 * np.linalg.norm(ref), kw
        assert np.linalg.norm(K @ u[free] - f[free]) <= 2e-11 * np.linalg.norm(f[free]), kw
        again, info2 = gpu_ctx.solve(f, rtol=1e-11, **kw)
        assert np.array_equal(u, again) and info.iters == info2.iters, kw


def test_failures_in_a_cluster(gpu_ctx):
    """The loop's exits: zero load, iteration cap, indefinite matrix."""
    m = meshgen.block_c3d8_pressure(n=4)
    gpu_ctx.setup(m)
    gpu_ctx.assemble_ex(_lib.ASM_CSR64 | _lib.ASM_BSR64 | _lib.ASM_BSR32)
    f = gpu_ctx.load_vector(m)
    for kw in (dict(), MIXED, dict(MIXED, preconditioner=_lib.PRECOND_COARSE)):
        u, info = gpu_ctx.solve(np.zeros_like(f), rtol=1e-10, **kw)
        assert not u.any() and info.iters == 0
        with pytest.raises(_lib.AxiaError) as e:
            gpu_ctx.solve(f, rtol=1e-10, max_iter=3, **kw)
        assert e.value.code == _lib.ERR_NOT_CONVERGED
        u, _ = gpu_ctx.solve(f, rtol=1e-10, **kw)
        assert np.isfinite(u).all()
    x = np.array([0, 1])
    with pytest.raises(_lib.AxiaError) as e:  # p.Ap = 0 in the first step
        gpu_ctx.solve_kff(2, (x, x, np.array([1.0, -1.0])), np.array([1.0, 1.0]))
    assert e.value.code == _lib.ERR_ZERO_PIVOT
