"""A load that is not finite, handed over on the device where no host check sees
it, is AXIA_ERR_NONFINITE in every form of the solve, not a zero load; the next
call is unharmed."""
import numpy as np
import pytest
import torch

from axia_gpu import _lib, meshgen

pytestmark = pytest.mark.gpu

MIX = dict(precision=_lib.PREC_MIXED, refine_mode=_lib.REFINE_RELIABLE, inner_rtol=0.1)
BSR = dict(matrix_format=_lib.FORMAT_BSR3)
FORMS = {
    "csr64": dict(), "bsr64": BSR, "csr_mixed": MIX, "bsr_mixed": dict(MIX, **BSR),
    "csr_restart": dict(precision=_lib.PREC_MIXED, refine_mode=_lib.REFINE_RESTART),
    "two_level": dict(MIX, preconditioner=_lib.PRECOND_COARSE, **BSR),
    "sym": dict(MIX, matrix_format=_lib.FORMAT_BSR3_SYM),
}


@pytest.fixture(scope="module", params=[6, 18])  # one cluster, the whole grid
def block(gpu_ctx, request):
    m = meshgen.block_c3d8_multiload(n=request.param, nrhs=9)
    gpu_ctx.setup(m)
    gpu_ctx.assemble_ex(_lib.ASM_CSR64 | _lib.ASM_CSR32 | _lib.ASM_BSR64 | _lib.ASM_BSR32 | _lib.ASM_SYM32 |
                        _lib.ASM_BSR32LO)
    return m, int(np.nonzero(m.free_mask())[0][-1])


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("form", FORMS)
def test_single(gpu_ctx, block, form, bad):
    m, dof = block
    f = torch.from_numpy(m.cload_batch[0]).cuda()
    u = torch.zeros_like(f)
    gpu_ctx.solve_device(f.data_ptr(), u.data_ptr(), rtol=1e-8, **FORMS[form])
    ref = u.clone()
    g = f.clone()
    g[dof] = bad
    with pytest.raises(_lib.AxiaError) as e:
        gpu_ctx.solve_device(g.data_ptr(), u.data_ptr(), rtol=1e-8, **FORMS[form])
    assert e.value.code == _lib.ERR_NONFINITE
    gpu_ctx.solve_device(f.data_ptr(), u.data_ptr(), rtol=1e-8, **FORMS[form])
    assert torch.equal(u, ref)
    info = gpu_ctx.solve_device((0.0 * f).data_ptr(), u.data_ptr(), rtol=1e-8, **FORMS[form])  # a zero load stays one
    assert info.iters == 0 and not u.any()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("krylov", [_lib.KRYLOV_PER_CASE, _lib.KRYLOV_BLOCK])
@pytest.mark.parametrize("pre", [_lib.PRECOND_JACOBI, _lib.PRECOND_COARSE])
def test_batched(gpu_ctx, block, pre, krylov, bad):
    m, dof = block
    F = torch.from_numpy(m.cload_batch).cuda()
    F[3] = 0.0  # an idle case beside it
    U = torch.zeros_like(F)
    kw = dict(rtol=1e-8, preconditioner=pre, krylov=krylov)
    gpu_ctx.solve_batched_device(9, F.data_ptr(), U.data_ptr(), **kw)
    ref = U.clone()
    G = F.clone()
    G[5, dof] = bad
    with pytest.raises(_lib.AxiaError) as e:
        gpu_ctx.solve_batched_device(9, G.data_ptr(), U.data_ptr(), **kw)
    assert e.value.code == _lib.ERR_NONFINITE
    gpu_ctx.solve_batched_device(9, F.data_ptr(), U.data_ptr(), **kw)
    assert torch.equal(U, ref)
