"""Gradients of FP32-mixed chains against those of FP64 chains on the same
noise: they lose no bits to cancelling sums, to the low-rank correction of
accurate measurements, or to weights of several terms."""
import numpy as np
import pytest

import multigridmc_gb300 as M
from problems import fem_posterior, posterior

pytestmark = pytest.mark.gpu


def _points():
    op = M.LinearOperator.shifted_laplace_fd((24, 24, 24), 10.0)
    idx = np.random.default_rng(0).permutation(op.n)[:100]
    return op.with_lowrank([(np.array([i]), np.ones(1)) for i in idx], 0.01 * np.ones(100))


# Relative errors (x-bar, f-bar) with u from two sweeps per reversed sweep, a
# correction in FP64 between them and A_0 u summed in FP32 in stencil order,
# as measured; the bound is 1.1 times that.
CASES = {
    "fem": (lambda: fem_posterior((32, 16, 48), periodic=False, m=6, radius=0.15)[1], 6.93e-7, 1.52e-7),
    "points": (_points, 5.23e-7, 7.82e-8),
    "balls": (lambda: posterior((32, 32, 32), m=8, radius=0.1, variance=1.0)[1], 9.09e-7, 7.13e-8),
    "prior": (lambda: posterior((32, 32, 32))[1], 1.04e-6, 6.98e-8),
}


@pytest.mark.parametrize("name", CASES)
def test_state_gradient(name):
    make, tol_x, tol_f = CASES[name]
    op = make()
    prm = M.MultigridParameters(nlevel=3)
    a, b = (M.MultigridMCSampler(op, prm, precision=p, seed=4) for p in (M.FP64, M.FP32_MIXED))
    rng, err = np.random.default_rng(0), []
    for k in range(8):
        v = rng.standard_normal(op.n).astype(np.float32).astype(float) if k < 4 else (np.arange(op.n) % 97 == k).astype(float)
        out = []
        for s in (a, b):
            xbar, fbar = v.copy(), np.zeros(op.n)
            s.adjoint_step(xbar, fbar)
            out.append((xbar, fbar))
        err.append([np.linalg.norm(q - p) / np.linalg.norm(p) for p, q in zip(*out)])
    ex, ef = np.exp(np.log(err).mean(0))
    assert ex <= 1.1 * tol_x and ef <= 1.1 * tol_f, (ex, ef)
    a.close()
    b.close()
