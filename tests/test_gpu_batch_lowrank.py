"""Low-rank corrections of batched chains, bit for bit those of the chains
stepped alone: groups whose chains correct in different ways (few separate
columns, overlapping columns, more columns than a CTA's S^{-1}, none), and
supports whose rows a CTA of the batch takes in several parts."""
import numpy as np
import pytest

import multigridmc_gb300 as M
from problems import posterior

pytestmark = pytest.mark.gpu


def _same(make, nsteps=4):
    solo, chains = make(), make()
    for s in solo:
        s.step(nsteps)
    batch = M.MultigridMCBatch(chains)
    assert batch.groups == (1, len(chains))
    batch.step(nsteps)
    batch.synchronize()
    for k, (a, b) in enumerate(zip(solo, chains)):
        xa, xb = a.get_state(), b.get_state()
        assert np.all(np.isfinite(xa)) and np.array_equal(xa, xb), f"chain {k}: {np.abs(xa - xb).max():.3e}"
    batch.close()
    for s in solo + chains:
        s.close()


def _points(shape, m, seed):
    op = M.LinearOperator.shifted_laplace_fd(shape, 10.0)
    idx = np.random.default_rng(seed).permutation(op.n)[:m]
    return op.with_lowrank([(np.array([i]), np.ones(1)) for i in idx], 0.01 * np.ones(m))


def _chain(op, nlevel, seed):
    s = M.MultigridMCSampler(op, M.MultigridParameters(nlevel=nlevel), precision=M.FP32_MIXED, seed=seed)
    s.fix_rhs(np.random.default_rng(seed).standard_normal(op.n))
    return s


def test_chains_of_different_modes():
    shape = (32, 16, 24)
    _same(lambda: [_chain(op, 3, 20 + k) for k, op in enumerate([
        posterior(shape)[1],
        posterior(shape, m=4, radius=0.08, seed=3)[1],
        posterior(shape, m=12, radius=0.4, seed=4)[1],
        _points(shape, 64, 5),
        _points(shape, 65, 6),
        _points(shape, 300, 7),
        posterior(shape, m=1, radius=0.1, seed=8)[1],
    ])])


def test_rows_in_several_parts():
    """Three slabs of vertices, about 340,000 rows of C: more than 1024 rows a
    CTA when the chain steps alone."""
    shape = (72, 72, 72)
    op = M.LinearOperator.shifted_laplace_fd(shape, 10.0)
    c = np.arange(op.n) // 71 ** 2
    slabs = [np.flatnonzero((c >= lo) & (c < hi)) for lo, hi in ((0, 23), (25, 47), (49, 71))]
    op = op.with_lowrank([(i, np.full(len(i), 1e-3)) for i in slabs], np.full(3, 0.1))
    _same(lambda: [_chain(op, 3, 30 + k) for k in range(2)])
