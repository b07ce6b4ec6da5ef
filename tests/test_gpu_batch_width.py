"""Load-case counts around the widths of the batched kernel (8, 16 and 32
columns, and a remainder after 32), meshes around its row tiles, with and
without the FP32 low parts and the two-level preconditioner, against single
solves of the same cases."""
import numpy as np
import pytest

from axia_gpu import _lib, meshgen

pytestmark = pytest.mark.gpu

RTOL = 1e-10


@pytest.mark.parametrize("low", [0, _lib.ASM_BSR32LO])
@pytest.mark.parametrize("pre", [_lib.PRECOND_JACOBI, _lib.PRECOND_COARSE])
@pytest.mark.parametrize("n,nrhs", [(2, 1), (5, 8), (5, 9), (7, 16), (7, 17), (9, 34)])
def test_widths_match_single_solves(gpu_ctx, n, nrhs, pre, low):
    m = meshgen.block_c3d8_multiload(n=n, nrhs=nrhs)
    if nrhs > 2:
        m.cload_batch[1] = 0.0  # an idle case
    gpu_ctx.setup(m)
    gpu_ctx.assemble_ex(_lib.ASM_BSR64 | _lib.ASM_BSR32 | low)
    U, info, rel = gpu_ctx.solve_batched(m.cload_batch, rtol=RTOL, preconditioner=pre)
    assert U.shape == m.cload_batch.shape and rel.shape == (nrhs,)
    assert (rel <= RTOL).all()
    U2, _, _ = gpu_ctx.solve_batched(m.cload_batch, rtol=RTOL, preconditioner=pre)
    assert np.array_equal(U, U2)  # fixed summation orders
    for k in sorted({0, 1 if nrhs > 1 else 0, nrhs // 2, nrhs - 1}):
        u, _ = gpu_ctx.solve(m.cload_batch[k], rtol=1e-12, matrix_format=_lib.FORMAT_BSR3)
        # both within their residual tolerances: errors of cond(K) 1e-10 at most
        assert np.linalg.norm(U[k] - u) <= 1e-7 * max(np.linalg.norm(u), 1e-300)


def test_long_rows(gpu_ctx):
    """C3D20 rows (up to 81 blocks) are longer than the kernel's row staging."""
    m = meshgen.block_c3d20_traction(n=4)
    gpu_ctx.setup(m)
    gpu_ctx.assemble_ex(_lib.ASM_BSR64 | _lib.ASM_BSR32 | _lib.ASM_BSR32LO)
    f = gpu_ctx.load_vector(m)
    F = np.stack([f, -2.0 * f, 0.5 * f])
    U, _, rel = gpu_ctx.solve_batched(F, rtol=RTOL, preconditioner=_lib.PRECOND_COARSE)
    u, _ = gpu_ctx.solve(f, rtol=1e-12, matrix_format=_lib.FORMAT_BSR3)
    assert (rel <= RTOL).all()
    for k, s in enumerate((1.0, -2.0, 0.5)):
        assert np.linalg.norm(U[k] - s * u) <= 1e-7 * np.linalg.norm(s * u)
