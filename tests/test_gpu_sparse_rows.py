"""Matrices with a few entries per row on both sides of the line between one
cluster and the whole grid (rows count there as well as entries): chains, plane
and space grids against a direct solve."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

pytestmark = pytest.mark.gpu


def grid_matrix(dims):
    K = sp.identity(1)
    for d in dims:
        T = sp.diags([-np.ones(d - 1), 2.0 * np.ones(d), -np.ones(d - 1)], [-1, 0, 1])
        K = sp.kron(K, sp.identity(d)) + sp.kron(sp.identity(K.shape[0]), T)
    return K.tocoo()  # the first identity leaves a shift of 1 on the diagonal


@pytest.mark.parametrize("lanes", [0, 8])
# 19,642 / 19,643 rows: the line for 3 entries per row and 4 lanes; 130 / 137 squared; 25 / 27 cubed
@pytest.mark.parametrize("dims", [(2,), (700,), (19642,), (19643,), (130000,), (130, 130), (137, 137), (25, 25, 25),
                                  (27, 27, 27)])
def test_grid_matrices(gpu_ctx, dims, lanes):
    K = grid_matrix(dims)
    n = K.shape[0]
    b = np.random.default_rng(7).standard_normal(n)
    x, info = gpu_ctx.solve_kff(n, (K.row, K.col, K.data), b, rtol=1e-12, spmv_lanes=lanes)
    Kc = K.tocsc()
    ref = spla.spsolve(Kc, b)
    # smallest eigenvalue above 1: the error is at most the residual
    assert np.linalg.norm(x - ref) <= 1.1e-12 * np.linalg.norm(b)
    again, info2 = gpu_ctx.solve_kff(n, (K.row, K.col, K.data), b, rtol=1e-12, spmv_lanes=lanes)
    assert np.array_equal(x, again) and info.iters == info2.iters
