"""The C3D8 energy kernel takes four elements per warp: element counts around
four, distorted elements of several sizes and places, against the oracle's
element stiffness; and the gradient, where u and v are one vector."""
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
    u = rng.standard_normal(m.ndof) * h
    v = rng.standard_normal(m.ndof) * h
    gpu_ctx.setup(m)
    s_uv, s_uu = gpu_ctx.element_energy(u, v), gpu_ctx.element_energy(u)
    # the oracle's own rounding: coordinates |offset| / h ulps, a few dozen operations
    tol = 1e-14 * (1.0 + abs(offset) / h) * 100
    for k in range(m.n_elem):
        ke, _ = O.element_ke(m.coords.reshape(-1, 3)[m.conn[k]], 1.0, m.nu)
        d = (3 * m.conn[k][:, None] + np.arange(3)).ravel()
        for s, w in ((s_uv, v), (s_uu, u)):
            scale = np.abs(u[d]) @ np.abs(ke) @ np.abs(w[d])
            assert abs(s[k] - u[d] @ ke @ w[d]) <= tol * scale


@pytest.mark.parametrize("nx,ny,nz", [(3, 1, 1), (5, 3, 2)])
def test_gradient_is_the_energy_of_u_with_itself(gpu_ctx, nx, ny, nz):
    m = meshgen.simp_beam(nx=nx, ny=ny, nz=nz)
    rho = np.random.default_rng(nx).uniform(0.3, 1.0, m.n_elem)
    gpu_ctx.setup(m)
    u, _, _ = gpu_ctx.compliance_forward(rho, m.pexp, m.e0, gpu_ctx.load_vector(m), rtol=1e-12)
    g = gpu_ctx.compliance_backward()
    ref = -m.pexp * rho ** (m.pexp - 1.0) * m.e0 * gpu_ctx.element_energy(u)
    assert np.abs(g - ref).max() <= 1e-13 * np.abs(ref).max()
