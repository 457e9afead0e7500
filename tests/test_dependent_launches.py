"""Source rules of kernels that start while the launch before is still running
(programmatic dependent launches), and the same chains with and without such
launches."""
import os
import re

import numpy as np
import pytest

import multigridmc_gb300 as M
from problems import fem_posterior, periodic_posterior, posterior

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "multigridmc_gb300", "csrc")

# operands that no launch of a step writes: operators, factors, index lists, tables of pointers
CONSTANT = {"vd", "jobcols", "jobs", "rows", "ptr", "col", "val", "sigma_inv", "sigma_sqrt", "L", "Linv", "LinvT", "row",
            "A", "Q", "W", "la", "lrs", "ca", "bq"}
WAIT, TRIGGER = r"\bpdl_begin(_trigger)?\(", r"\bpdl_trigger\("


def _functions():
    """name -> (parameters, body) of every device function of kernels.cuh."""
    s = open(os.path.join(CSRC, "kernels.cuh")).read()
    s = re.sub(r"//[^\n]*|__launch_bounds__\([^()]*\)|=\s*VarField<T>\{nullptr, 0\}", "", s)
    out = {}
    for m in re.finditer(r"(?:__global__|__device__ __forceinline__)([^;{(]*?)(\w+)\s*\(([^{;]*?)\)\s*(?:const\s*)?\{", s):
        depth, end = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(s[end], 0)
            end += 1
        old = out.get(m.group(2), ("", ""))  # overloads together
        out[m.group(2)] = (old[0] + " " + m.group(3), old[1] + s[m.end():end])
    return out


def _waiting(fns):
    """Functions that wait, and the ones that those call."""
    calls = {f: {g for g in fns if g != f and re.search(r"\b%s\s*[<(]" % g, body)} for f, (_, body) in fns.items()}
    waits = {f for f, (_, body) in fns.items() if re.search(WAIT, body)} - {"pdl_begin", "pdl_begin_trigger"}
    for step in (lambda w: {f for f in fns if calls[f] & w}, lambda w: {g for f in w for g in calls[f]}):
        while step(waits) - waits:
            waits |= step(waits)
    return waits


def test_the_parser_sees_the_kernels():
    fns = _functions()
    names = _waiting(fns)
    for k in ("k_sweep_rb_vec", "sweep_rb_vec_body", "k_sweep_row_pair", "k_lr_correct", "lr_correct_body", "k_chol_gemv_lower",
              "chol_gemv_lower_body", "k_prolong_add", "k_resid_restrict_tiled", "rr_tile_compute", "k_add_Bq", "sor_point",
              "ld8_stream", "k_step_end", "k_chol_step"):
        assert k in names, k
    assert "k_unpack" in fns and "k_unpack" not in names


def test_no_promises_on_memory_that_a_launch_writes():
    fns = _functions()
    for name in sorted(_waiting(fns)):
        params, body = fns[name]
        promised = set(re.findall(r"__restrict__\s*(\w+)", params + body))
        assert promised <= CONSTANT, f"{name}: {sorted(promised - CONSTANT)}"
        assert "ld.global.nc" not in body, name
        for asm in re.findall(r"asm(.*?);\s*\n", body, re.S):
            if "ld.global" in asm:
                assert "volatile" in asm and '"memory"' in asm, name


def test_a_kernel_waits_before_it_lets_the_next_one_start():
    fns = _functions()
    for name, (_, body) in fns.items():
        t = re.search(TRIGGER, body)
        if t and name != "pdl_trigger":
            w = re.search(WAIT, body)
            assert w and w.start() < t.start(), name


def _chain(make, prm, precision, seed=3):
    op = make()
    s = M.MultigridMCSampler(op, prm, precision=precision, seed=seed)
    s.fix_rhs(np.random.default_rng(1).standard_normal(op.n))
    s.set_observable(np.arange(min(op.n, 3000)), np.ones(min(op.n, 3000)), 8)
    return s


def _points(shape, m, seed=0):
    """m single-vertex measurements."""
    op = M.LinearOperator.shifted_laplace_fd(shape, 10.0)
    idx = np.random.default_rng(seed).permutation(op.n)[:m]
    return op.with_lowrank([(np.array([i]), np.ones(1)) for i in idx], 0.01 * np.ones(m))


V3, W3 = M.MultigridParameters(nlevel=3), M.MultigridParameters(nlevel=4, cycle=2)
CASES = {
    "fd-2d": (lambda: posterior((48, 80))[1], V3),
    "fd-2d-m5": (lambda: posterior((48, 80), m=5, radius=0.1)[1], V3),
    "fd-3d-m6": (lambda: posterior((40, 32, 24), m=6, radius=0.1)[1], V3),
    "fd-3d-m70": (lambda: _points((24, 24, 24), 70), V3),
    "fem-3d-w": (lambda: fem_posterior((32, 16, 48), periodic=False, m=4, radius=0.15)[1], W3),
    "fields-3d": (lambda: periodic_posterior((24, 16, 32), m=4, radius=0.15)[1], V3),
    "fields-2d": (lambda: fem_posterior((40, 24), m=3, radius=0.1)[1], V3),
}


def _on_and_off(monkeypatch, run):
    monkeypatch.delenv("MGMC_NO_PDL", raising=False)
    on = run()
    monkeypatch.setenv("MGMC_NO_PDL", "1")
    off = run()
    assert len(on) == len(off)
    for a, b in zip(on, off):
        assert np.all(np.isfinite(a)) and np.array_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
@pytest.mark.parametrize("name", CASES)
def test_steps_with_and_without_dependent_launches(name, precision, monkeypatch):
    def run():
        s = _chain(*CASES[name], precision)
        s.step(12)
        out = [s.get_state(), s.read_observations(8)]
        b = np.random.default_rng(2).standard_normal(s.n)
        out.append(s.solve(b)[0])
        s.step(3)
        out.append(s.get_state())
        s.close()
        return out
    _on_and_off(monkeypatch, run)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
@pytest.mark.parametrize("name", ["fd-2d-m5", "fd-3d-m6", "fd-3d-m70", "fem-3d-w"])
def test_adjoint_with_and_without_dependent_launches(name, precision, monkeypatch):
    def run():
        s = _chain(*CASES[name], precision)
        r = np.random.default_rng(4)
        x, out = r.standard_normal(s.n), []
        for k in range(3):  # issued, then captured, then replayed
            xbar, fbar = r.standard_normal(s.n), np.zeros(s.n)
            gc, gs = s.adjoint_params(x, xbar, fbar, k)
            out += [xbar, fbar, np.array([gc]), np.asarray(gs)]
        s.close()
        return out
    _on_and_off(monkeypatch, run)


@pytest.mark.gpu
def test_batch_with_and_without_dependent_launches(monkeypatch):
    shape = (16, 24, 16)

    def run():
        ch = [_chain(lambda m=m, k=k: _points(shape, m, k) if m else posterior(shape)[1], V3, M.FP32_MIXED, 10 + k)
              for k, m in enumerate((0, 4, 70, 9))]
        ch.append(_chain(*CASES["fd-2d-m5"], M.FP32_MIXED))
        b = M.MultigridMCBatch(ch)
        b.step(8)
        b.synchronize()
        out = [v for s in ch for v in (s.get_state(), s.read_observations(8))]
        b.close()
        for s in ch:
            s.close()
        return out
    _on_and_off(monkeypatch, run)
