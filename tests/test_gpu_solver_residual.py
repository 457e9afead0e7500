"""The solver's residual kernel: the residual norm it reports and the right
hand side it hands to the preconditioner, at rows just below, at and beyond
the segments a warp takes, for each kind of stencil, with and without
low-rank rows."""
import numpy as np
import pytest

import multigridmc_gb300 as M

pytestmark = pytest.mark.gpu


def _fd(shape):
    return M.LinearOperator.shifted_laplace_fd(shape, 10.0)


def _centre(shape):
    st = M.fd_stencil(shape, 10.0)
    n = int(np.prod([c - 1 for c in shape]))
    return M.LinearOperator(shape, st, centre=st.ravel()[13] * np.random.default_rng(1).uniform(1.0, 1.5, n))


def _fem(shape):
    return M.LinearOperator.shifted_laplace_fem(shape, 10.0)


def _field(shape):
    return M.LinearOperator.shifted_laplace_fem_periodic(shape, 0.12, 0.23)


CASES = [(_fd, (4, 4, 4)), (_fd, (128, 8, 4)), (_fd, (130, 12, 6)), (_fd, (258, 20)), (_centre, (132, 8, 4)),
         (_fem, (130, 8, 4)), (_fem, (256, 16)), (_field, (256, 16)), (_fd, (514,))]


@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
@pytest.mark.parametrize("lowrank", [False, True])
@pytest.mark.parametrize("make,shape", CASES)
def test_second_iteration(make, shape, lowrank, precision):
    op = make(shape)
    if lowrank:
        rows = np.arange(op.n)
        op = op.with_lowrank([(rows[::3], np.ones(rows[::3].size) / rows.size), (rows[:5], np.ones(rows[:5].size))],
                             np.array([0.01, 0.02]))
    s = M.MultigridMCSampler(op, M.MultigridParameters(nlevel=2), precision=precision)
    b = np.random.default_rng(3).standard_normal(op.n)
    x1, _, r0, _ = s.solve(b, maxiter=1)
    x2, _, r1, _ = s.solve(b, maxiter=2)
    A = op.to_scipy()
    r = b - A @ x1
    # the residual's own rounding: 29 terms of size |A| |x|, added per row
    scale = 29 * np.finfo(float).eps * np.linalg.norm(abs(A) @ np.abs(x1) + np.abs(b))
    assert abs(r0 - np.linalg.norm(b)) <= 1e-13 * np.linalg.norm(b)
    assert abs(r1 - np.linalg.norm(r)) <= scale
    # P is linear and bounded by |P b| / |b| up to the condition of the vector
    # (below 1e3); in FP32 its own rounding
    tol = 1e3 * scale * np.linalg.norm(x1) / np.linalg.norm(b)
    if precision == M.FP32_MIXED:
        tol += 1e-4 * np.linalg.norm(x2 - x1)
    assert np.linalg.norm(x2 - x1 - s.precondition(r)) <= tol + 1e-12 * np.linalg.norm(x1)
    s.close()
