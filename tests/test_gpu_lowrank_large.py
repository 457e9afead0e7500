"""Low-rank corrections of many or widely overlapping columns, whose solve is a
launch of its own, against their formula on the library's own noise-free
sweeps: x'' = x' - C S^{-1} B^T x' with x' and the columns of C swept by a
sampler without the low-rank term."""
import numpy as np
import pytest
import scipy.sparse as sp

import multigridmc_gb300 as M

pytestmark = pytest.mark.gpu


def _balls(shape, m, radius):
    pts = np.indices([c - 1 for c in shape][::-1]).reshape(len(shape), -1)[::-1]
    xs = [(p + 1.0) / c for p, c in zip(pts, shape)]
    cols = []
    for x0 in np.random.default_rng(4).uniform(0.1, 0.9, (m, len(shape))):
        i = np.nonzero(sum((a - b) ** 2 for a, b in zip(xs, x0)) <= radius ** 2)[0]
        cols.append((i, np.full(i.size, 1.0 / i.size)))
    return cols


# shape, columns, radius: the first three differ in the terms a lane takes (one
# block, its edge, several); then overlapping columns on more CTAs than the SMs
# hold, in runs of 256 and of 1024 rows; then few wide ones
CASES = [((20, 20), 65, 0.15), ((24, 24), 128, 0.15), ((24, 24), 129, 0.1), ((40, 40), 300, 0.1), ((64, 64, 64), 20, 0.3),
         ((128, 128, 128), 6, 0.4), ((160, 160, 160), 2, 0.45)]


@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
@pytest.mark.parametrize("shape,m,radius", CASES)
def test_correction(shape, m, radius, precision):
    prior = M.LinearOperator.shifted_laplace_fd(shape, 10.0)
    op = prior.with_lowrank(_balls(shape, m, radius), 0.01 * np.ones(m))
    s, p = M.SSORSampler(op, precision=precision), M.SSORSampler(prior, precision=M.FP64)
    B = sp.csc_matrix((op.B_val, op.B_idx, op.B_ptr), shape=(op.n, m))
    rng = np.random.default_rng(6)
    f = rng.standard_normal(op.n)
    # rounding of m products and of an m x m solve of condition below 1e3, in the state's precision
    tol = 1e-11 if precision == M.FP64 else 2e-5
    for d in (M.FORWARD, M.BACKWARD):
        C = np.zeros((op.n, m))
        for j in range(m):
            c = np.zeros(op.n)
            p.sor(0, d, B[:, j].toarray().ravel(), c, with_noise=False)
            C[:, j] = c
        S = np.diag(op.Sigma) + B.T @ C
        x = rng.standard_normal(op.n)
        want = x.copy()
        p.sor(0, d, f, want, with_noise=False)
        want -= C @ np.linalg.solve(S, B.T @ want)
        s.sor(0, d, f, x, with_noise=False)
        assert np.max(np.abs(x - want)) < tol * np.max(np.abs(want))
    s.close()
    p.close()
