"""Prolongation (FP64: sums of the parents direction by direction) in one to
three dimensions at the smallest and at ragged sizes, and the coarse Cholesky
product at coarse grids whose rows end within, at and beyond the vectors that
a warp loads ahead."""
import numpy as np
import pytest

import multigridmc_gb300 as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
@pytest.mark.parametrize("shape", [(4,), (512,), (4, 4), (6, 260), (260, 6), (4, 4, 4), (258, 6, 4), (20, 12, 36)])
def test_prolongation(shape, precision):
    s = M.MultigridMCSampler(M.LinearOperator.shifted_laplace_fd(shape, 10.0), M.MultigridParameters(nlevel=2),
                             precision=precision)
    R = M.intergrid_to_sparse(shape)
    rng = np.random.default_rng(5)
    xc, x = rng.standard_normal(R.shape[0]), rng.standard_normal(R.shape[1])
    got = s.prolongate_add(0, 0.7, xc, x.copy())
    # at most 8 parents and one update, each rounded once
    eps = np.finfo(np.float64 if precision == M.FP64 else np.float32).eps
    assert np.max(np.abs(got - (x + 0.7 * (R.T @ xc)))) <= 12 * eps * (np.max(np.abs(x)) + np.max(np.abs(xc)))
    s.close()


# unknowns of the coarse grid: 1, 9, 127 to 129, 256 to 258, 511 to 513 and 1023 to 1025 of its rows
@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
@pytest.mark.parametrize("cells", [4, 20, 256, 258, 260, 514, 516, 518, 1024, 1026, 1028, 2048, 2050, 2052])
def test_coarse_product(cells, precision):
    op = M.LinearOperator.shifted_laplace_fd((cells,), 1e4)
    s = M.MultigridMCSampler(op, M.MultigridParameters(nlevel=2, smoother="SOR", npresmooth=1, npostsmooth=0),
                             precision=precision)
    b = np.random.default_rng(7).standard_normal(op.n)
    x = np.zeros(op.n)
    s.sor(0, M.FORWARD, b, x, with_noise=False)
    R, A = M.intergrid_to_sparse(op.shape), op.to_scipy()
    Ac = (R @ A @ R.T).toarray()
    want = x + R.T @ np.linalg.solve(Ac, R @ (b - A @ x))
    got = s.precondition(b)
    # rounding of the sweep, residual and factors times the coarse matrix' condition
    eps = np.finfo(np.float64 if precision == M.FP64 else np.float32).eps
    assert np.linalg.norm(got - want) <= 100 * eps * np.linalg.cond(Ac) * np.linalg.norm(want)
    s.close()
