"""A load case that is not finite in a wide batched launch leaves nothing behind
for the launches after it, whatever their widths, within a call or in the next."""
import numpy as np
import pytest
import torch

from axia_gpu import _lib, meshgen

pytestmark = pytest.mark.gpu

RTOL = 1e-10


def _solve(ctx, F, **kw):
    Fd = torch.from_numpy(np.ascontiguousarray(F)).cuda()
    U = torch.full_like(Fd, 7.0)
    info, rel = ctx.solve_batched_device(F.shape[0], Fd.data_ptr(), U.data_ptr(), rtol=RTOL,
                                         preconditioner=_lib.PRECOND_COARSE, **kw)
    return U.cpu().numpy(), rel


@pytest.mark.parametrize("bad", [np.nan, np.inf, 1e300])
@pytest.mark.parametrize("low", [0, _lib.ASM_BSR32LO])
@pytest.mark.parametrize("n", [7, 12])  # 48 and 162 coarse unknowns: 16 and 30 rows of padding
def test_later_launches(gpu_ctx, n, low, bad):
    m = meshgen.block_c3d8_multiload(n=n, nrhs=34)
    F = m.cload_batch
    free = np.nonzero(m.free_mask())[0]
    gpu_ctx.setup(m)
    gpu_ctx.assemble_ex(_lib.ASM_BSR64 | _lib.ASM_BSR32 | low)
    ref = {k: _solve(gpu_ctx, F[:k])[0] for k in (1, 7, 16, 34)}
    assert gpu_ctx.coarse_size()[1] % 64 != 0
    wide = F[:32].copy()
    wide[:, free] = bad  # every case and every coarse unknown of a wide launch
    for k in (1, 7, 16, 34):
        try:
            _solve(gpu_ctx, np.concatenate([wide, F[:2]]))
        except _lib.AxiaError:
            pass
        U, rel = _solve(gpu_ctx, F[:k])
        assert (rel <= RTOL).all()
        assert np.array_equal(U, ref[k])
