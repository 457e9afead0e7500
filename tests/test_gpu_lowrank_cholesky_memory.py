"""The low-rank Cholesky sampler's two forms: with the products E and G of the
factor's blocks (three arrays of the blocks' size) and compact (two), which
lattices whose three arrays do not fit fall back to; any number of columns."""
import ctypes as C

import numpy as np
import pytest

import multigridmc_gb300 as M
import oracle as O
from gpu_helpers.build import build as gpu_build
from problems import posterior

pytestmark = pytest.mark.gpu


def _bytes(monkeypatch, compact, shape):
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("MGMC_LRCHOL_COMPACT", "1" if compact else "0")
    op = posterior(shape, m=2, radius=0.1)[1]
    f, x = np.ones(op.n), np.zeros(op.n)
    M.LowRankCholeskySampler(op).apply(f, x)  # modules and graph memory of the first one
    before = torch.cuda.mem_get_info()[0]
    s = M.LowRankCholeskySampler(op)
    s.apply(f, x)
    after = torch.cuda.mem_get_info()[0]
    s.close()
    return before - after


@pytest.mark.parametrize("compact,arrays", [(False, 3), (True, 2)])
def test_resident_memory(compact, arrays, monkeypatch):
    shape = (25, 25, 25)
    p, nb = 24 * 24, 24
    block_bytes = 8 * nb * p * p
    # vectors, Q and allocation granules: a few per cent of one array
    assert _bytes(monkeypatch, compact, shape) <= (arrays + 0.5) * block_bytes


@pytest.mark.parametrize("shape,m,radius", [((12,), 2, 0.2), ((5, 3), 0, 0.1), ((9, 40), 3, 0.1), ((34, 4), 2, 0.2),
                                            ((1030, 3), 2, 0.1), ((7, 9, 5), 5, 0.25), ((4, 4, 30), 35, 0.2)])
def test_compact_form_equals_oracle(shape, m, radius, monkeypatch):
    monkeypatch.setenv("MGMC_LRCHOL_COMPACT", "1")
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


def test_both_forms_draw_the_same(monkeypatch):
    _, op = posterior((17, 16, 9), m=3, radius=0.15)
    f = np.random.default_rng(1).standard_normal(op.n)
    out = []
    for compact in "01":
        monkeypatch.setenv("MGMC_LRCHOL_COMPACT", compact)
        s = M.LowRankCholeskySampler(op, seed=7)
        x = np.zeros(op.n)
        for _ in range(3):
            s.apply(f, x)
        out.append(x.copy())
        s.close()
    # the same normals; 64 eps per unit of the prior's condition number, below 1e4 here
    assert np.linalg.norm(out[0] - out[1]) < 64 * np.finfo(float).eps * 1e4 * np.linalg.norm(out[0])


@pytest.mark.parametrize("m", [1, 32, 33, 300, 6200, 28672, 28673, 30000])
def test_columns_beyond_shared_memory(m):
    """m x m and Q products up to and beyond the columns that one CTA and that
    shared memory take (W = 0 where it would be gigabytes of host data)."""
    lib = C.CDLL(gpu_build("chol_wide_check"))
    rng = np.random.default_rng(m)
    part, Q = rng.standard_normal((3, m)), rng.standard_normal((130, m))
    W = rng.standard_normal((m, m)) if m <= 300 else None
    g, xi0 = rng.standard_normal(130), rng.standard_normal(130)
    P = lambda a: a.ctypes.data_as(C.POINTER(C.c_double)) if a is not None else None
    out = []
    for wide in (-1, 1):
        xi, v = xi0.copy(), np.zeros(m)
        assert lib.chol_wide_check(P(part), 3, m, P(W), P(Q), 130, P(g), P(xi), P(v), wide) == 0
        out.append((xi, v))
    t = part.sum(0)
    want = (W.T @ t if W is not None else 0.0) - t
    # sums of m products of size below 6 x 18 in FP64
    for xi, v in out:
        assert np.max(np.abs(v - want)) < 1e-15 * 110 * (m if W is not None else 3)
        assert np.max(np.abs(xi - (xi0 + g + Q @ want))) < 1e-15 * m * 6 * max(1.0, np.abs(want).max())
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("m", [31, 32, 33, 100, 400])
def test_many_columns_equal_oracle(m):
    op_o, op = posterior((9, 9, 9))
    B = np.zeros((op.n, m))
    B[np.random.default_rng(2).permutation(op.n)[:m], np.arange(m)] = 1.0
    sig = 0.5 * np.ones(m)
    op_o.set_lowrank(B, sig)
    op = op.with_lowrank(B, sig)
    noise = O.CLCG().draw_normal(2 * op.n)
    orc = O.lowrank_cholesky_sampler(op_o, O.Source(noise))
    gpu = M.LowRankCholeskySampler(op, noise=M.INJECTED)
    gpu.inject_noise(noise)
    f = np.random.default_rng(3).standard_normal(op.n)
    tol = 64 * np.finfo(float).eps * np.linalg.cond(op.to_scipy().toarray())
    xo, xg = np.zeros(op.n), np.zeros(op.n)
    for _ in range(2):
        orc.apply(f, xo)
        gpu.apply(f, xg)
        assert np.linalg.norm(xg - xo) < tol * np.linalg.norm(xo)
    gpu.close()
