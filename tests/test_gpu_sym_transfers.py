"""FP64 residual-restriction of symmetric stencils against the sparse
operators: f_c = R (f - A_0 x) through level 1's right hand side of a
noise-free cycle with no smoothing, at window edges (rows of 255, 256 and 257
or more columns), short rows, 2D and 3D."""
import numpy as np
import pytest

import multigridmc_gb300 as M

pytestmark = pytest.mark.gpu

SHAPES = [(4, 4, 4), (16, 6, 8), (34, 12, 6), (256, 4, 4), (258, 6, 4), (4, 4), (30, 10), (256, 8), (510, 6), (512, 4)]


@pytest.mark.parametrize("op", ["fd", "fem"])
@pytest.mark.parametrize("shape", SHAPES)
def test_resid_restrict_sym(shape, op):
    A = (M.LinearOperator.shifted_laplace_fd if op == "fd" else M.LinearOperator.shifted_laplace_fem)(shape, 10.0)
    prm = M.MultigridParameters(nlevel=2, npresmooth=0, npostsmooth=0)
    s = M.MultigridMCSampler(A, prm, precision=M.FP64)
    # without smoothing a noise-free cycle is x = R^T (R A R^T)^{-1} R b
    rng = np.random.default_rng(3)
    b = rng.standard_normal(A.n)
    R = M.intergrid_to_sparse(shape).toarray()
    As = A.to_scipy()
    Ac = R @ (As @ R.T)
    want = R.T @ np.linalg.solve(Ac, R @ b)
    got = s.precondition(b)
    # sums of at most 27 terms, and the coarse solve's condition number
    tol = 200 * np.finfo(float).eps * np.linalg.cond(Ac)
    assert np.linalg.norm(got - want) < tol * np.linalg.norm(want)
    s.close()
    # one pre-smoothing sweep: x' = x + P (b - A x) with x = M^{-1} b
    prm = M.MultigridParameters(nlevel=2, smoother="SOR", npresmooth=1, npostsmooth=0)
    s = M.MultigridMCSampler(A, prm, precision=M.FP64)
    x = np.zeros(A.n)
    s.sor(0, M.FORWARD, b, x, with_noise=False)
    want = x + R.T @ np.linalg.solve(Ac, R @ (b - As @ x))
    got = s.precondition(b)
    assert np.linalg.norm(got - want) < tol * np.linalg.norm(want)
    s.close()
