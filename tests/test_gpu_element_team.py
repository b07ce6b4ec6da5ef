"""C3D20 / C3D20R batches on both sides of the size where a team of warps shares
an element: the same bits per element whatever the batch, and the oracle's
stiffness."""
import numpy as np
import pytest

from axia_gpu import meshgen
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _elements(n, seed):
    rng = np.random.default_rng(seed)
    xi = meshgen.HEX20_XI.astype(np.float64)
    return 0.5 * xi[None] + rng.uniform(-0.08, 0.08, (n, 20, 3)), rng.uniform(1e3, 2e5, n)


@pytest.mark.parametrize("reduced", [False, True])
def test_batches_agree(gpu_ctx, reduced):
    xyz, e = _elements(4 * 152 + 1, 5)
    big, vbig = gpu_ctx.element_ke(xyz, e, 0.3, reduced=reduced)  # one warp per element
    for n in (1, 7, 153, 4 * 152):  # a team per element: 1, part of and all the SMs, several per SM
        ke, vol = gpu_ctx.element_ke(xyz[:n], e[:n], 0.3, reduced=reduced)
        assert np.array_equal(ke, big[:n]) and np.array_equal(vol, vbig[:n])
    ref, vref = O.element_ke(xyz[3], float(e[3]), 0.3, reduced=reduced)
    assert np.abs(big[3] - ref).max() <= 1e-12 * np.abs(ref).max()
    assert abs(vbig[3] - vref) <= 1e-12 * vref
