"""The coarse inverse works on 64 x 64 tiles on and below the diagonal: from one
tile to 59 a side, with the last one nearly empty or full.  The mixed
solve has to reach the direct solution, and a coarse space that is inverted
correctly never costs iterations against the diagonal alone."""
import numpy as np
import pytest

from axia_gpu import _lib, meshgen
from oracle import oracle as O

pytestmark = pytest.mark.gpu

MIXED = dict(precision=_lib.PREC_MIXED, refine_mode=_lib.REFINE_RELIABLE, matrix_format=_lib.FORMAT_BSR3,
             inner_rtol=0.1, rtol=1e-10)


@pytest.fixture(scope="module")
def block():
    m = meshgen.cantilever_c3d8(12, 10, 8)
    ref = O.solve_static(m, solver=O.SOLVER_PCG, tol=1e-6, keep_csr=True)
    u = np.zeros(m.ndof)
    u[m.bc_dof] = m.bc_val
    u[m.free_mask()] = O.direct_solve(ref.indptr, ref.indices, ref.data, ref.rhs)
    return m, u


@pytest.mark.parametrize("nodes", [2000, 264, 60, 24, 16, 8, 4, 2])
def test_tiles(gpu_ctx, block, nodes):
    m, u_ref = block
    gpu_ctx.setup(m)
    gpu_ctx.assemble_ex(_lib.ASM_BSR64 | _lib.ASM_BSR32)
    f = gpu_ctx.load_vector(m)
    _, jac = gpu_ctx.solve(f, **MIXED)
    u, info = gpu_ctx.solve(f, preconditioner=_lib.PRECOND_COARSE, coarse_nodes=nodes, **MIXED)
    # a reliable update more or less may cost an iteration or two
    assert info.iters <= jac.iters + 2
    assert np.linalg.norm(u - u_ref) <= 1e-8 * np.linalg.norm(u_ref)
