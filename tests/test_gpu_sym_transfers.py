"""Residual-restriction of symmetric FP64 stencils, and of per-vertex stencils
and 2D FP32 levels (one coarse row segment per CTA), against the sparse
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
    _check(A, shape, M.FP64)


@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
@pytest.mark.parametrize("shape", [(4, 4), (30, 10), (66, 8), (68, 6), (4, 4, 4), (34, 12, 6), (66, 6, 4)])
@pytest.mark.parametrize("op", ["fd", "fd_periodic", "fem_periodic"])
def test_resid_restrict_rows(shape, op, precision):
    if op == "fd":
        A = M.LinearOperator.shifted_laplace_fd(shape, 10.0)
    elif op == "fd_periodic":
        A = M.LinearOperator.shifted_laplace_fd_periodic(shape, 0.12, 0.23)
    else:
        A = M.LinearOperator.shifted_laplace_fem_periodic(shape, 0.12, 0.23)
    _check(A, shape, precision)


def _check(A, shape, precision):
    prm = M.MultigridParameters(nlevel=2, npresmooth=0, npostsmooth=0)
    s = M.MultigridMCSampler(A, prm, precision=precision)
    # without smoothing a noise-free cycle is x = R^T (R A R^T)^{-1} R b
    rng = np.random.default_rng(3)
    b = rng.standard_normal(A.n)
    R = M.intergrid_to_sparse(shape).toarray()
    As = A.to_scipy()
    Ac = R @ (As @ R.T)
    want = R.T @ np.linalg.solve(Ac, R @ b)
    got = s.precondition(b)
    # sums of at most 27 terms, and the coarse solve's condition number
    tol = 200 * np.finfo(float if precision == M.FP64 else np.float32).eps * np.linalg.cond(Ac)
    assert np.linalg.norm(got - want) < tol * np.linalg.norm(want)
    s.close()
    # one pre-smoothing sweep: x' = x + P (b - A x) with x = M^{-1} b
    prm = M.MultigridParameters(nlevel=2, smoother="SOR", npresmooth=1, npostsmooth=0)
    s = M.MultigridMCSampler(A, prm, precision=precision)
    x = np.zeros(A.n)
    s.sor(0, M.FORWARD, b, x, with_noise=False)
    want = x + R.T @ np.linalg.solve(Ac, R @ (b - As @ x))
    got = s.precondition(b)
    assert np.linalg.norm(got - want) < tol * np.linalg.norm(want)
    s.close()
