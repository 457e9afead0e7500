"""FP64 sweeps with in-kernel noise: constant symmetric stencils (neighbours
added in pairs or by classes) against the same stencil given per vertex, whose
kernels add weight by weight.  Both draw the same normals, so the results
differ by rounding only."""
import numpy as np
import pytest

import multigridmc_gb300 as M

pytestmark = pytest.mark.gpu


def _axis_stencil(dim):
    st = np.zeros(27)
    for d in range(dim):
        st[13 - 3 ** d] = st[13 + 3 ** d] = -0.2 / (d + 1)
    st[13] = 1.0 - st.sum()
    return st


def _full_stencil(dim):
    st = np.zeros(27)
    for k in range(27):
        d = [abs(k % 3 - 1), abs((k // 3) % 3 - 1), abs(k // 9 - 1)]
        if not any(d[dim:]):
            st[k] = -0.1 / (1 + d[0] + 2 * d[1] + 4 * d[2])
    st[13] = 1.0 - st.sum() + st[13]
    return st


@pytest.mark.parametrize("omega", [1.0, 1.2])
@pytest.mark.parametrize("full", [False, True])
@pytest.mark.parametrize("shape", [(9, 8), (33, 6), (129, 5), (2, 3, 4), (8, 5, 4), (34, 6, 5), (65, 9, 4), (130, 4, 4)])
def test_noisy_sweeps(shape, full, omega):
    st = (_full_stencil if full else _axis_stencil)(len(shape))
    n = int(np.prod([c - 1 for c in shape]))
    const = M.LinearOperator(shape, st)
    if full:
        vertex = M.LinearOperator(shape, st, field=np.repeat(st[:, None], n, axis=1))
    else:
        vertex = M.LinearOperator(shape, st, centre=np.full(n, st[13]))
    a, b = (M.SSORSampler(op, omega=omega, precision=M.FP64, seed=9) for op in (const, vertex))
    rng = np.random.default_rng(1)
    f, x0 = rng.standard_normal(n), rng.standard_normal(n)
    for direction in (M.FORWARD, M.BACKWARD):
        x, y, z = x0.copy(), x0.copy(), x0.copy()
        a.sor(0, direction, f, x, with_noise=True)
        b.sor(0, direction, f, y, with_noise=True)
        a.sor(0, direction, f, z, with_noise=False)
        assert np.max(np.abs(x - z)) > 0.1  # there is noise
        # at most 29 roundings of terms below 8 in each, carried through at most 8 colours
        assert np.max(np.abs(x - y)) < 2 * 29 * 8 * 8 * 2.0 ** -52
    a.close()
    b.close()
