"""FP64 levels with per-vertex or unsymmetric 27-point stencils are swept two
colours or one colour per launch, whichever set-up finds faster: the state does
not depend on the choice (nor on the CTA shapes), bit for bit."""
import numpy as np
import pytest

import multigridmc_gb300 as M

pytestmark = pytest.mark.gpu


def _operator(shape, kind):
    st = np.zeros(27)
    for k in range(27):
        d = [k % 3 - 1, (k // 3) % 3 - 1, k // 9 - 1]
        st[k] = -0.1 / (1 + abs(d[0]) + 2 * abs(d[1]) + 4 * abs(d[2])) * (1 + 0.1 * d[0] - 0.05 * d[1] + 0.02 * d[2])
    st[13] = 1.0 - st.sum() + st[13]
    n = int(np.prod([c - 1 for c in shape]))
    if kind == "constant":
        return M.LinearOperator(shape, st)
    scale = np.random.default_rng(0).uniform(1.0, 1.2, n)
    fld = np.repeat(st[:, None], n, axis=1)
    fld[13] *= scale
    return M.LinearOperator(shape, st, field=fld)


@pytest.mark.parametrize("noise", [M.PHILOX, M.INJECTED])
@pytest.mark.parametrize("kind", ["constant", "field"])
@pytest.mark.parametrize("shape", [(66, 64, 67), (80, 66, 64), (130, 48, 48)])
def test_choice_does_not_change_the_state(shape, kind, noise, monkeypatch):
    op = _operator(shape, kind)
    f = np.random.default_rng(1).standard_normal(op.n)
    out = []
    for autotune in "01":
        monkeypatch.setenv("MGMC_AUTOTUNE", autotune)
        s = M.SSORSampler(op, omega=1.1, precision=M.FP64, noise=noise, seed=2)
        s.fix_rhs(f)
        if noise == M.INJECTED:
            s.inject_noise(np.random.default_rng(3).standard_normal(2 * s.noise_per_step))
        s.step(2)
        out.append(s.get_state())
        s.close()
    assert np.all(np.isfinite(out[0])) and np.array_equal(*out)
