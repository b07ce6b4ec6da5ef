"""Nodal means and shear strains are rounded as the divisions of their
definition round them: bitwise those of the element stresses, on tetrahedra with
2 to 24 elements at a node and on hexahedra with 1 to 8."""
import numpy as np
import pytest

from axia_gpu import meshgen

pytestmark = pytest.mark.gpu

E, NU = 210000.0, 0.3


def _recover(ctx, m):
    ctx.setup(m)
    u = np.random.default_rng(11).standard_normal(m.ndof)
    return ctx.recover(u, e_strain=E)


def test_means_of_tetrahedra(gpu_ctx):
    m = meshgen.block_tet(n=3, nn=4, e=E, nu=NU, perturb=0.2)
    stress, strain, _, _, emean = _recover(gpu_ctx, m)
    want = np.zeros_like(stress)
    cnt = np.zeros(m.n_nodes)
    for e, nodes in enumerate(m.conn):  # one point: an element's stress is that of its nodes
        want[nodes] += emean[e]
        cnt[nodes] += 1.0
    assert {6.0, 12.0, 24.0} <= set(cnt)  # not powers of two
    assert np.array_equal(stress, want / cnt[:, None])
    assert np.array_equal(strain[:, 3:], stress[:, 3:] / (E / (1.0 + NU)))


@pytest.mark.parametrize("n", [1, 5])
def test_shear_strains_of_hexahedra(gpu_ctx, n):
    m = meshgen.block_c3d8_pressure(n=n, e=E, nu=NU, perturb=0.2)
    stress, strain, _, _, _ = _recover(gpu_ctx, m)
    assert np.array_equal(strain[:, 3:], stress[:, 3:] / (E / (1.0 + NU)))
    tr = stress[:, :3].sum(axis=1, keepdims=True)
    want = ((1.0 + NU) * stress[:, :3] - NU * tr) / E
    # the numerator's rounding differs by a fused multiply-add: a few ulp of its terms
    assert np.abs(strain[:, :3] - want).max() <= 4 * 2.0**-53 * np.abs(stress[:, :3]).max() * 3 / E


def test_not_finite(gpu_ctx):
    """Infinities and NaN of the stresses go through as a division passes them."""
    m = meshgen.block_c3d8_pressure(n=3, e=E, nu=NU, perturb=0.2)
    gpu_ctx.setup(m)
    u = np.random.default_rng(3).standard_normal(m.ndof) * 3e302  # strains of 1e303, E times that overflows
    stress, strain, _, _, _ = gpu_ctx.recover(u, e_strain=E)
    assert np.isinf(stress[:, 3:]).any()
    with np.errstate(all="ignore"):
        assert np.array_equal(strain[:, 3:], stress[:, 3:] / (E / (1.0 + NU)), equal_nan=True)
