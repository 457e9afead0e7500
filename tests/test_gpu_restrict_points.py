"""Residual-restriction of levels large enough for one coarse point per thread:
a noise-free two-level cycle -- one sweep, the coarse sweeps of R (f - A x), its
prolongation -- restated with the sparse operators and the samplers' own sweeps."""
import numpy as np
import pytest

import multigridmc_gb300 as M

pytestmark = pytest.mark.gpu


def _operator(shape, kind):
    st = np.zeros(27)
    dim, n = len(shape), int(np.prod([c - 1 for c in shape]))
    for k in range(27):
        d = [abs(k % 3 - 1), abs((k // 3) % 3 - 1), abs(k // 9 - 1)]
        if any(d[dim:]) or (kind.startswith("axis") and sum(d) > 1):
            continue
        st[k] = -0.1 / (1 + d[0] + 2 * d[1] + 4 * d[2])
    st[13] = 1.0 - st.sum() + st[13]
    scale = np.random.default_rng(0).uniform(1.0, 1.2, n)
    if kind.endswith("centre"):
        return M.LinearOperator(shape, st, centre=st[13] * scale)
    if kind.endswith("field"):
        fld = np.repeat(st[:, None], n, axis=1)
        fld[13] *= scale
        return M.LinearOperator(shape, st, field=fld)
    return M.LinearOperator(shape, st)


@pytest.mark.parametrize("precision,shape,kind", [
    (M.FP64, (32768,), "axis"), (M.FP32_MIXED, (24578,), "axis"), (M.FP32_MIXED, (258, 256), "axis"),
    (M.FP32_MIXED, (1026, 64), "axis-centre"), (M.FP32_MIXED, (364, 360), "full"), (M.FP32_MIXED, (360, 364), "full-centre"),
    (M.FP32_MIXED, (456, 460), "full-field"), (M.FP64, (1030, 1010), "axis-centre"), (M.FP64, (1010, 1030), "full-field"),
    (M.FP32_MIXED, (96, 96, 98), "axis-centre")])
def test_two_level_cycle(precision, shape, kind):
    op = _operator(shape, kind)
    prm = M.MultigridParameters(nlevel=2, smoother="SOR", coarse_solver="SSOR", npresmooth=1, npostsmooth=0)
    s = M.MultigridMCSampler(op, prm, precision=precision, noise=M.INJECTED)
    s.inject_noise(np.zeros(s.noise_per_step))
    f, got = np.random.default_rng(1).standard_normal(op.n), np.zeros(op.n)
    s.apply(f, got)
    s.close()
    R, A = M.intergrid_to_sparse(shape), op.to_scipy()
    fine, coarse = M.SSORSampler(op, precision=M.FP64), M.SSORSampler(op.coarsen(), precision=M.FP64)
    x = np.zeros(op.n)
    fine.sor(0, M.FORWARD, f, x, with_noise=False)
    fc = R @ (f - A @ x)
    y = np.zeros(fc.size)
    for d in (M.FORWARD, M.BACKWARD):
        coarse.sor(0, d, fc, y, with_noise=False)
    fine.close()
    coarse.close()
    want = x + R.T @ y
    # a few hundred roundings of terms below 10
    eps = 2.0 ** -52 if precision == M.FP64 else 2.0 ** -23
    assert np.max(np.abs(got - want)) < 300 * 10 * eps
