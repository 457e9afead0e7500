"""Observables: values past the staging buffer, long supports shared by
several CTAs, the count and its reset, and the error of a non-finite value."""
import numpy as np
import pytest

import multigridmc_gb300 as M
from problems import posterior

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
@pytest.mark.parametrize("nnz", [1, 1024, 1025, 5000, 40000])
def test_observable_sum(nnz, precision):
    """z = b^T x of the state, for supports of one CTA and of several."""
    op = M.LinearOperator.shifted_laplace_fd((36, 36, 36), 10.0)
    s = M.MultigridMCSampler(op, M.MultigridParameters(nlevel=2), precision=precision, seed=3)
    rng = np.random.default_rng(1)
    idx = np.sort(rng.choice(op.n, nnz, replace=False))
    val = rng.standard_normal(nnz)
    s.set_probes([(idx, val), (idx[:1], val[:1])], 4)
    s.step(2)
    z = s.read_observations(4)
    x = s.get_state()
    want = np.array([val @ x[idx], val[0] * x[idx[0]]])
    # sums of nnz terms in FP64
    assert z.shape == (2, 2) and np.all(np.abs(z[1] - want) <= 1e-15 * nnz * np.abs(val).max() * np.abs(x).max())
    s.close()


def test_observations_past_the_staging_buffer():
    _, op = posterior((8, 8), m=2, radius=0.2)
    probes = [(np.array([k]), np.ones(1)) for k in range(5)]
    a = M.MultigridMCSampler(op, M.MultigridParameters(nlevel=2), seed=5)
    b = M.MultigridMCSampler(op, M.MultigridParameters(nlevel=2), seed=5)
    for s in (a, b):
        s.set_probes(probes, 1000)
    a.step(1000)
    za = a.read_observations(1000)
    zb = []
    for _ in range(10):
        b.step(100)
        zb.append(b.read_observations(100))
    assert za.shape == (1000, 5) and np.array_equal(za, np.concatenate(zb))
    a.step(3)
    assert np.array_equal(a.read_observations(1000)[-1], a.get_state()[:5])
    a.close()
    b.close()


def test_non_finite_observable_is_reported():
    op = M.LinearOperator.shifted_laplace_fd((8, 8), 10.0)
    s = M.MultigridMCSampler(op, M.MultigridParameters(nlevel=2))
    s.set_observable(np.arange(op.n), np.ones(op.n), 4)
    s.step(1)
    assert np.isfinite(s.read_observations(4)).all()
    s.set_state(np.full(op.n, np.nan))
    s.step(1)
    with pytest.raises(M.MGMCError) as e:
        s.read_observations(4)
    assert e.value.name == "MGMC_ERR_NONFINITE"
    s.close()
