"""The low-rank Cholesky sampler's block kernels against the oracle at the
edges of their sizes: blocks of one value, of odd and even length, of more
values than a row keeps in registers, two blocks and many."""
import numpy as np
import pytest

import multigridmc_gb300 as M
import oracle as O
from problems import posterior

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,m,radius", [((12,), 2, 0.2), ((5, 3), 0, 0.1), ((9, 40), 3, 0.1), ((34, 4), 2, 0.2),
                                            ((1030, 3), 2, 0.1), ((7, 9, 5), 5, 0.25), ((4, 4, 30), 35, 0.2)])
def test_blocks_equal_oracle(shape, m, radius):
    op_o, op = posterior(shape, m=m, radius=radius, variance=1e-2)
    noise = O.CLCG().draw_normal(2 * op.n)
    orc = O.lowrank_cholesky_sampler(op_o, O.Source(noise))
    gpu = M.LowRankCholeskySampler(op, noise=M.INJECTED)
    gpu.inject_noise(noise)
    f = np.random.default_rng(3).standard_normal(op.n)
    # the factors are unique; rounding in either is amplified by the condition number
    tol = 64 * np.finfo(float).eps * np.linalg.cond(op.to_scipy().toarray())
    xo, xg = np.zeros(op.n), np.zeros(op.n)
    for _ in range(2):
        orc.apply(f, xo)
        gpu.apply(f, xg)
        assert np.linalg.norm(xg - xo) < tol * np.linalg.norm(xo)
    gpu.close()
