"""The low-rank correction of a sweep against its formula in numpy, for each
way its rows are shared out: few columns per CTA, overlapping columns, more
than 64 columns, and supports of up to two and three rows of four per thread;
and the low-rank term of a residual-restriction."""
import numpy as np
import pytest

import multigridmc_gb300 as M

pytestmark = pytest.mark.gpu

# shape, ball centres (or how many at random), radius
CASES = {
    "few": ((32, 32, 32), [(x, y, z) for x in (0.25, 0.75) for y in (0.25, 0.75) for z in (0.25, 0.75)], 0.12),
    "overlapping": ((16, 16, 16), 20, 0.25),
    "one_column": ((16, 12), 1, 0.2),
    "sixty_four": ((40, 40), 64, 0.06),
    "many": ((24, 24), 70, 0.1),
    "empty_rows": ((24, 24), [(0.3, 0.3), (0.3, 0.3), (0.7, 0.6)], 0.1),
    "two_quads": ((1400, 1400), [(0.25, 0.5), (0.75, 0.5)], 0.2),
    "three_quads": ((1400, 1400), [(0.25, 0.5), (0.75, 0.5)], 0.24),
}


def _operator(name):
    shape, centres, radius = CASES[name]
    if isinstance(centres, int):
        centres = np.random.default_rng(4).uniform(0.1, 0.9, (centres, len(shape)))
    N = [c - 1 for c in shape]
    pts = np.indices(N[::-1]).reshape(len(shape), -1)[::-1]  # x fastest
    xs = [(p + 1.0) / c for p, c in zip(pts, shape)]
    cols = []
    for x0 in centres:
        i = np.nonzero(sum((a - b) ** 2 for a, b in zip(xs, x0)) <= radius ** 2)[0]
        cols.append((i, np.full(i.size, 1.0 / i.size)))
    return M.LinearOperator.shifted_laplace_fd(shape, 10.0).with_lowrank(cols, 0.01 * np.ones(len(cols)))


def _sweep(op, x, f, forward):
    """Red-black sweep of A_0, the arrays as (..., rows, x)."""
    N = [c - 1 for c in op.shape][::-1]
    x, f = x.reshape(N).copy(), f.reshape(N)
    colour = sum(np.indices(N)) & 1
    w = op.stencil.reshape(3, 3, 3)
    for k in (0, 1) if forward else (1, 0):
        off = np.zeros(N)
        for d in range(len(N)):  # array axis d is direction len(N) - 1 - d
            o = [1, 1, 1]
            o[2 - (len(N) - 1 - d)] = 0
            lo = [slice(None)] * len(N)
            hi = [slice(None)] * len(N)
            lo[d], hi[d] = slice(0, -1), slice(1, None)
            off[tuple(hi)] += w[tuple(o)] * x[tuple(lo)]
            off[tuple(lo)] += w[tuple(o)] * x[tuple(hi)]
        x = np.where(colour == k, (f - off) / w[1, 1, 1], x)
    return x.reshape(-1)


@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
@pytest.mark.parametrize("name", list(CASES))
def test_lowrank_correction(name, precision):
    op = _operator(name)
    s = M.SSORSampler(op, precision=precision)
    rng = np.random.default_rng(6)
    f = rng.standard_normal(op.n)
    # the formula's own rounding: a sweep, m products and an m x m solve of
    # condition below 1e3, in the state's precision
    tol = 1e-11 if precision == M.FP64 else 2e-5
    import scipy.sparse as sp
    B = sp.csc_matrix((op.B_val, op.B_idx, op.B_ptr), shape=(op.n, op.m))
    for forward in (True, False):
        C = np.stack([_sweep(op, np.zeros(op.n), B[:, j].toarray().ravel(), forward) for j in range(op.m)], 1)
        S = np.diag(op.Sigma) + B.T @ C
        x = rng.standard_normal(op.n)
        want = _sweep(op, x, f, forward)
        want = want - C @ np.linalg.solve(S, B.T @ want)
        s.sor(0, M.FORWARD if forward else M.BACKWARD, f, x, with_noise=False)
        assert np.max(np.abs(x - want)) < tol * np.max(np.abs(want))
    s.close()


@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
@pytest.mark.parametrize("name", ["few", "overlapping", "many"])
def test_residual_lowrank(name, precision):
    op = _operator(name)
    s = M.MultigridMCSampler(op, M.MultigridParameters(nlevel=2, smoother="SOR", npresmooth=1, npostsmooth=0),
                             precision=precision)
    b = np.random.default_rng(7).standard_normal(op.n)
    x = np.zeros(op.n)
    s.sor(0, M.FORWARD, b, x, with_noise=False)
    R, A = M.intergrid_to_sparse(op.shape), op.to_scipy()
    Ac = (R @ A @ R.T).toarray()
    want = x + R.T @ np.linalg.solve(Ac, R @ (b - A @ x))
    got = s.precondition(b)
    # the coarse solve amplifies the residual's rounding by its condition number (below 1e4)
    tol = 1e-10 if precision == M.FP64 else 1e-3
    assert np.linalg.norm(got - want) < tol * np.linalg.norm(want)
    s.close()
