"""Many meshes solved as one system: the two-level preconditioner's subdomains
stay within what the CG kernel holds (682), at least one per mesh, and more
meshes than that are an error of the single solve, not of the batched one."""
import numpy as np
import pytest

from axia_gpu import _lib, meshgen

pytestmark = pytest.mark.gpu

MIXED = dict(precision=_lib.PREC_MIXED, refine_mode=_lib.REFINE_RELIABLE, inner_rtol=0.01,
             matrix_format=_lib.FORMAT_BSR3, rtol=1e-10)
MAX_SUBDOMAINS = 682


def _setup(ctx, sizes):
    ms = [meshgen.block_c3d8_pressure(n=n) for n in sizes]
    ctx.setup_multi(ms)
    ctx.assemble_ex(_lib.ASM_BSR64 | _lib.ASM_BSR32)
    return np.concatenate([ctx.load_vector(m) for m in ms])


# one-element meshes beside a large one, whose share alone would be 45 and 300 subdomains
@pytest.mark.parametrize("sizes,nodes", [([16] + [1] * 600, 0), ([16] + [1] * 660, 0), ([14, 14] + [1] * 650, 8),
                                         ([1] * MAX_SUBDOMAINS, 0)])
def test_large_and_tiny_meshes(gpu_ctx, sizes, nodes):
    f = _setup(gpu_ctx, sizes)
    ref, _ = gpu_ctx.solve(f, preconditioner=_lib.PRECOND_JACOBI, **MIXED)
    u, _ = gpu_ctx.solve(f, preconditioner=_lib.PRECOND_COARSE, coarse_nodes=nodes, **MIXED)
    assert len(sizes) <= gpu_ctx.coarse_size()[0] <= MAX_SUBDOMAINS
    assert np.linalg.norm(u - ref) <= 1e-8 * np.linalg.norm(ref)  # both to a residual of 1e-10


def test_more_meshes_than_subdomains(gpu_ctx):
    f = _setup(gpu_ctx, [1] * (MAX_SUBDOMAINS + 18))
    for _ in range(2):
        with pytest.raises(_lib.AxiaError) as e:
            gpu_ctx.solve(f, preconditioner=_lib.PRECOND_COARSE, **MIXED)
        assert e.value.code == _lib.ERR_TOO_LARGE
    ref, _ = gpu_ctx.solve(f, preconditioner=_lib.PRECOND_JACOBI, **MIXED)
    U, _, _ = gpu_ctx.solve_batched(np.stack([f, -f]), rtol=1e-10, preconditioner=_lib.PRECOND_COARSE)
    assert np.linalg.norm(U[0] - ref) <= 1e-8 * np.linalg.norm(ref)
    assert np.linalg.norm(U[1] + ref) <= 1e-8 * np.linalg.norm(ref)
