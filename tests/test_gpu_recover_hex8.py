"""The C3D8 recovery kernel takes four elements per warp: element counts around
that, distorted elements of several sizes far from the origin, several moduli,
against the oracle."""
import numpy as np
import pytest

from axia_gpu import meshgen
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(1, 1, 1), (3, 1, 1), (2, 2, 1), (5, 1, 1), (3, 3, 4)])
@pytest.mark.parametrize("h,offset", [(1.0, 0.0), (1e-3, 10.0), (100.0, -3e3)])
def test_counts_and_placements(gpu_ctx, nx, ny, nz, h, offset):
    rng = np.random.default_rng(nx * 100 + ny * 10 + nz)
    m = meshgen.cantilever_c3d8(nx, ny, nz, h=h)
    m.coords = m.coords + rng.uniform(-0.15, 0.15, m.coords.shape) * h + offset
    m.e_elem = rng.uniform(1e3, 2e5, m.n_elem)
    u = rng.standard_normal(m.ndof) * 1e-3 * h
    f = rng.standard_normal(m.ndof)
    gpu_ctx.setup(m)
    stress, strain, vm, rf, emean = gpu_ctx.recover(u, f)
    s_ref, vm_ref, em_ref = O.nodal_stress(m, u, elem_mean=True)
    eps_ref = O.nodal_strain(s_ref, float(m.e_elem[0]), m.nu)
    rf_ref = O.reactions(m, u, f)
    # the oracle's own rounding: coordinates |offset| / h ulps, a few dozen operations
    tol = 1e-14 * (1.0 + abs(offset) / h) * 100
    for a, b in ((stress, s_ref), (vm, vm_ref), (emean, em_ref), (strain, eps_ref), (rf, rf_ref)):
        assert np.abs(a - b).max() <= tol * np.abs(b).max()
