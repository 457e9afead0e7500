"""The work that users of this framework have it do, as cases that can be timed.

A case is a dict of plain values.  ``prepare`` builds what a program holds
before the call (operator, sampler, right hand side, state), ``run`` makes one
pass through the public entry points, ``work`` says what a pass cannot do
without, and ``exact`` restates the pass in plain torch in 64 bits: the same
multicolour Gibbs sweeps, Galerkin hierarchy, low-rank terms and Philox
normals, without this package's code.

Ranges that ``draw`` covers and the listed cases stand for:

* chains in 2D (16 to 800 cells per direction) and 3D (16 to 160, the listed
  256^3 chain being the largest), FP64 and, in 3D, FP32-mixed, FD, FEM and periodic
  (variable) priors, 0 to 64 ball measurements, SOR and SSOR smoothers, V- and
  W-cycles, Cholesky and SSOR coarse samplers, unequal extents;
* the one-level SSOR (Gibbs) sampler, which the experiments compare with;
* ``apply(f, x)`` on page-locked host vectors (the call a drop-in makes);
* batches of chains of uneven sizes;
* the loop solver, the parameter adjoint and the low-rank Cholesky sampler.

FP32-mixed chains hand their FP32 state over in float64 vectors; ``run``
returns those states in float32, which loses nothing.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

import multigridmc_gb300 as M

RADIUS, VARIANCE = 0.05, 1e-4  # the local measurements of the benchmark
LAMBDA = (0.12, 0.23)          # the periodic correlation length of the reference's tests


# ------------------------------------------------------------------ cases
def _chain(name=None, **kw):
    case = dict(kind="chain", op="fd", kappa_sq=10.0, nx=32, ny=32, nz=32, m=0, nlevel=3, precision="fp64",
                smoother="SSOR", cycle=1, coarse="Cholesky", omega=1.0, steps=4)
    case.update(kw)
    return dict(case, name=name) if name else case


def listed():
    return [
        # the reference's default experiment: 2D prior, FP64, many tiny kernels
        _chain("chain_2d_64_fp64", nx=64, ny=64, nz=0, nlevel=4, steps=10),
        # a large oblong 2D posterior
        _chain("chain_2d_768x480_fp64", nx=768, ny=480, nz=0, nlevel=5, m=12, steps=8),
        # the middle of the published 16^3 - 64^3 comparison, FP64 posterior
        _chain("chain_3d_32_fp64", nx=32, ny=32, nz=32, nlevel=3, m=32, steps=8),
        # ragged 3D lattice, FEM prior (27-point fine level), SOR smoother, W-cycle
        _chain("chain_fem_96x48x80_fp32", op="fem", nx=96, ny=48, nz=80, nlevel=4, m=20, precision="fp32",
               smoother="SOR", cycle=2, kappa_sq=25.0, steps=4),
        # periodic correlation length: per-vertex stencils on every level
        _chain("chain_periodic_64_fp32", op="fd_periodic", nx=64, ny=64, nz=64, nlevel=4, m=32, precision="fp32",
               steps=4),
        # the FP64 posterior that MGMC, Gibbs and exact samplers are compared on
        _chain("chain_3d_128_fp64", nx=128, ny=128, nz=128, nlevel=5, m=32, steps=4),
        # the headline chain: FP32-mixed posterior
        _chain("chain_3d_256_fp32", nx=256, ny=256, nz=256, nlevel=5, m=64, precision="fp32", steps=8),
        # the drop-in's call: Sampler::apply(f, x) on host vectors, FP64
        _chain("apply_host_96x80x112_fp64", kind="apply", nx=96, ny=80, nz=112, nlevel=4, m=16, steps=2),
        # many chains of uneven sizes, one launch sequence
        dict(name="batch_20_chains_fp32", kind="batch", chains=20, sizes="32,48,64", mmax=16, steps=4),
        # Q x = f to 1e-10 (posterior means, exact moments, exact draws)
        _chain("solve_128_fp32", kind="solve", nx=128, ny=128, nz=128, nlevel=5, m=32, precision="fp32", steps=1),
        # pathwise gradients: two steps in reverse, FP64
        _chain("adjoint_64_fp64", kind="adjoint", nx=64, ny=64, nz=64, nlevel=4, m=16, steps=2),
        # the reference's own exact comparator
        _chain("lrchol_32_fp64", kind="lrchol", nx=32, ny=32, nz=32, m=32, nlevel=1, steps=2),
    ]


def _log(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def _cells(rng, lo, hi, nlevel):
    """A cell count of about log-uniform size that can be coarsened nlevel - 1 times."""
    q = 2 ** (nlevel - 1)
    return max(2, round(_log(rng, lo, hi) / q)) * q


def draw(rng):
    kind = rng.choice(["chain"] * 6 + ["apply", "batch", "solve", "adjoint", "lrchol", "gibbs"])
    precision = rng.choice(["fp64", "fp32"])
    kappa_sq = round(_log(rng, 1.0, 100.0), 3)
    if kind == "batch":
        return dict(kind="batch", chains=rng.randint(3, 20), sizes=rng.choice(["32", "32,48", "48,64", "32,64"]),
                    mmax=rng.randint(0, 24), steps=rng.randint(1, 6))
    if kind == "lrchol":
        nx, ny, nz = (rng.randint(8, 26) for _ in range(3))
        return _chain(kind="lrchol", nx=nx, ny=ny, nz=nz, m=rng.randint(0, 24), nlevel=1, kappa_sq=kappa_sq,
                      steps=rng.randint(1, 3))
    if kind == "adjoint":
        nlevel = rng.randint(2, 3)
        nx, ny, nz = (_cells(rng, 16, 56, nlevel) for _ in range(3))
        return _chain(kind="adjoint", nx=nx, ny=ny, nz=nz, nlevel=nlevel, m=rng.randint(1, 16), kappa_sq=kappa_sq,
                      steps=rng.randint(1, 2))
    if rng.random() < 0.3 and kind != "solve":
        nlevel = 1 if kind == "gibbs" else rng.randint(3, 5)
        nx, ny, nz = _cells(rng, 16, 800, nlevel), _cells(rng, 16, 800, nlevel), 0
        top, precision = 800 * 800, "fp64"  # mixed precision is for 3D lattices, where it pays
    else:
        nlevel = 1 if kind == "gibbs" else rng.randint(3, 4)  # one level takes odd cell counts too
        nx, ny, nz = (_cells(rng, 16, 160, nlevel) for _ in range(3))
        top = 160 ** 3
    op = rng.choice(["fd", "fd", "fd", "fem", "fd_periodic"]) if kind == "chain" else "fd"
    coarse, q = "Cholesky", 2 ** (nlevel - 1)
    if math.prod(c // q for c in (nx, ny, nz) if c) > 2000 or rng.random() < 0.15:
        coarse = "SSOR"
    if op != "fd":  # per-vertex stencils are assembled on the host
        top = min(top, 64 ** 3)
    if kind == "solve":  # cells of about equal sides, as a multigrid solver wants
        nx = min(nx, 12 * q)
        ny, nz = nx + rng.choice([0, q]), nx + rng.choice([0, q])
        return _chain(kind=kind, kappa_sq=kappa_sq, nx=nx, ny=ny, nz=nz, nlevel=nlevel, precision=precision,
                      m=rng.choice([0, rng.randint(1, 8), rng.randint(8, 48)]), steps=1)
    while math.prod(c for c in (nx, ny, nz) if c) > top:
        nx, ny = max(nx // 2 // q, 2) * q, max(ny // 2 // q, 2) * q
        nz = max(nz // 2 // q, 2) * q if nz else 0
    case = _chain(kind=kind, op=op, kappa_sq=kappa_sq, nx=nx, ny=ny, nz=nz, nlevel=nlevel, precision=precision,
                  m=rng.choice([0, rng.randint(1, 8), rng.randint(8, 48)]), smoother=rng.choice(["SSOR", "SSOR", "SOR"]),
                  cycle=rng.choice([1, 1, 2]), coarse=coarse, omega=rng.choice([1.0, 1.0, 1.2, 0.9]),
                  steps=rng.randint(1, 8))
    if kind == "gibbs":
        case.update(coarse="SSOR", cycle=1, smoother="SSOR")
    return case


# ------------------------------------------------------------------ inputs
def _shape(case):
    return tuple(c for c in (case["nx"], case["ny"], case["nz"]) if c)


def _balls(shape, centres):
    """Local measurements: (vertex indices, weights) of the mean over the
    lattice points within RADIUS of each centre (the nearest vertex where the
    lattice is too coarse for any)."""
    cols = []
    N = [c - 1 for c in shape]
    for x0 in centres:
        near = [min(max(int(round(x * c)), 1), c - 1) for x, c in zip(x0, shape)]
        lo = [max(1, math.ceil((x - RADIUS) * c)) for x, c in zip(x0, shape)]
        hi = [min(c - 1, math.floor((x + RADIUS) * c)) for x, c in zip(x0, shape)]
        axes = [np.arange(a, b + 1) for a, b in zip(lo, hi)]
        grid = np.meshgrid(*axes[::-1], indexing="ij")[::-1]  # x fastest
        ok = sum((g / c - x) ** 2 for g, c, x in zip(grid, shape, x0)) <= RADIUS * RADIUS
        pts = [g[ok] for g in grid] if ok.any() else [np.array([v]) for v in near]
        idx = np.zeros(pts[0].size, np.int64)
        stride = 1
        for p, k in zip(pts, N):
            idx += (p - 1) * stride
            stride *= k
        cols.append((np.sort(idx), np.full(idx.size, 1.0 / idx.size)))
    return cols


def _inputs(case, seed):
    """Columns of B, Sigma, right hand side, initial state and Philox seed."""
    rng = np.random.default_rng(seed)
    shape = _shape(case)
    n = math.prod(c - 1 for c in shape)
    cols = _balls(shape, rng.uniform(0.1, 0.9, (case["m"], len(shape))))
    sigma = VARIANCE * np.ones(case["m"])
    if case["m"]:  # f = B Sigma^{-1} y of measured values y
        f = np.zeros(n)
        for (i, v), y, s in zip(cols, rng.standard_normal(case["m"]), sigma):
            f[i] += v * (y / s)
    else:
        f = 0.1 * rng.standard_normal(n)
    x = rng.standard_normal(n)
    return dict(cols=cols, sigma=sigma, f=f, x=x, noise_seed=int(rng.integers(1 << 31)))


def _operator(case, inp):
    shape = _shape(case)
    if case["op"] == "fem":
        op = M.LinearOperator.shifted_laplace_fem(shape, case["kappa_sq"])
    elif case["op"] == "fd_periodic":
        op = M.LinearOperator.shifted_laplace_fd_periodic(shape, *LAMBDA)
    else:
        op = M.LinearOperator.shifted_laplace_fd(shape, case["kappa_sq"])
    return op.with_lowrank(inp["cols"], inp["sigma"]) if case["m"] else op


def _sampler(case, inp, precision=None):
    prm = M.MultigridParameters(nlevel=case["nlevel"], smoother=case["smoother"], cycle=case["cycle"],
                                coarse_solver=case["coarse"], omega=case["omega"])
    return M.MultigridMCSampler(_operator(case, inp), prm, seed=inp["noise_seed"],
                                precision=M.FP32_MIXED if (precision or case["precision"]) == "fp32" else M.FP64)


def _batch_cases(case, seed):
    """The chains of a batch: sizes in turn, kappa^2 log-uniform, uneven measurement counts."""
    rng = np.random.default_rng([seed, 1])
    sizes = [int(s) for s in case["sizes"].split(",")]
    out = []
    for k in range(case["chains"]):
        c = sizes[k % len(sizes)]
        out.append(_chain(nx=c, ny=c, nz=c, nlevel=4 if c >= 64 else 3, m=int(rng.integers(0, case["mmax"] + 1)),
                          kappa_sq=float(10.0 ** rng.uniform(0, 2)), precision="fp32", steps=case["steps"]))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        chains = []
        for k, c in enumerate(_batch_cases(case, seed)):
            inp = _inputs(c, [seed, 2, k])
            s = _sampler(c, inp)
            s.fix_rhs(inp["f"])
            s.set_state(inp["x"])
            chains.append(s)
        outs = [torch.empty(s.n, dtype=torch.float64, device="cuda") for s in chains]
        return dict(case=case, batch=M.MultigridMCBatch(chains), chains=chains, outs=outs)
    inp = _inputs(case, seed)
    if kind == "lrchol":
        s = M.LowRankCholeskySampler(_operator(case, inp), seed=inp["noise_seed"])
        f = torch.from_numpy(inp["f"]).cuda()
        outs = [torch.empty(s.n, dtype=torch.float64, device="cuda") for _ in range(case["steps"])]
        torch.cuda.synchronize()
        return dict(case=case, s=s, f=f, outs=outs)
    s = _sampler(case, inp)
    st = dict(case=case, s=s)
    if kind == "apply":
        st["f"] = torch.from_numpy(inp["f"]).pin_memory()
        st["x"] = torch.from_numpy(inp["x"]).pin_memory()
        return st
    if kind == "solve":
        st["b"] = torch.from_numpy(inp["f"]).cuda()
        st["x"] = torch.empty(s.n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        return st
    s.fix_rhs(inp["f"])
    s.set_state(inp["x"])
    st["x"] = torch.empty(s.n, dtype=torch.float64, device="cuda")
    if kind == "adjoint":  # the checkpointed forward chain and the adjoint of its last state
        st["states"] = []
        for _ in range(case["steps"]):
            x = torch.empty(s.n, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            s.get_state_device(x.data_ptr())
            st["states"].append(x)
            s.step(1)
        st["xbar0"] = torch.from_numpy(_xbar(case, seed)).cuda()
        st["xbar"], st["fbar"] = torch.empty_like(st["x"]), torch.empty_like(st["x"])
    else:  # chains record the mean over the central ball, as the experiments do
        i, v = _centre_ball(_shape(case))
        s.set_observable(i, v, case["steps"])
    torch.cuda.synchronize()
    return st


def _centre_ball(shape):
    return _balls(shape, [[0.5] * len(shape)])[0]


def _xbar(case, seed):
    return np.random.default_rng([seed, 3]).standard_normal(math.prod(c - 1 for c in _shape(case)))


# ------------------------------------------------------------------ a pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        state["batch"].step(case["steps"])
        state["batch"].synchronize()
        for s, x in zip(state["chains"], state["outs"]):
            s.get_state_device(x.data_ptr())
        return [x.float() for x in state["outs"]]
    s = state["s"]
    if kind == "lrchol":
        for x in state["outs"]:
            s.apply_device(state["f"].data_ptr(), x.data_ptr())
        return state["outs"]
    if kind == "apply":
        f, x = state["f"].numpy(), state["x"].numpy()
        for _ in range(case["steps"]):
            s.apply(f, x)
        return x if case["precision"] == "fp64" else x.astype(np.float32)
    if kind == "solve":
        _, _, converged = s.solve_device(state["b"].data_ptr(), state["x"].data_ptr(), 1e-10, math.inf, 100)
        return {"x": state["x"], "converged": converged}
    if kind == "adjoint":
        state["xbar"].copy_(state["xbar0"])
        state["fbar"].zero_()
        torch.cuda.current_stream().synchronize()  # the sampler works on a stream of its own
        gc, gs = 0.0, 0.0
        for k in reversed(range(case["steps"])):
            c, g = s.adjoint_params_device(state["states"][k].data_ptr(), state["xbar"].data_ptr(),
                                           state["fbar"].data_ptr(), k)
            gc, gs = gc + c, gs + g
        return {"xbar": state["xbar"], "fbar": state["fbar"], "centre": gc, "log_sigma": gs}
    s.step(case["steps"])
    z = s.read_observations(case["steps"])
    s.get_state_device(state["x"].data_ptr())
    if case["precision"] == "fp32":
        return {"x": state["x"].float(), "z": z.astype(np.float32)}
    return {"x": state["x"], "z": z}


# ------------------------------------------------------------------ work
def work(case):
    """Bytes and operations of a pass: per sweep of a level its state read and
    written and its right hand side read once (per-vertex stencils too), per
    transfer the fine vectors once, the coarse factor once per half, the
    entries of B and of its support once per low-rank correction.  Noise is
    generated and costs no bytes."""
    if case["kind"] == "batch":
        parts = [work(c) for c in _batch_cases(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    shape, size = _shape(case), 8 if case["precision"] == "fp64" else 4
    dim, m = len(shape), case["m"]
    n0 = math.prod(c - 1 for c in shape)
    if case["kind"] == "lrchol":
        nb, p = shape[-1] - 1, n0 // (shape[-1] - 1)
        entries = nb * p * (p + 1) // 2 + (nb - 1) * p * p  # one block row of L, both solves read it
        return {"bytes": case["steps"] * 8.0 * (2 * entries + 3 * n0 * m + 2 * n0),
                "flops": case["steps"] * (4.0 * entries + 8.0 * n0 * m)}
    ball = math.pi * RADIUS ** 2 if dim == 2 else 4 / 3 * math.pi * RADIUS ** 3
    total = {"bytes": 0.0, "flops": 0.0}

    def add(nbytes, flops):
        total["bytes"] += nbytes
        total["flops"] += flops

    def level(l):
        n = math.prod((c >> l) - 1 for c in shape)
        npt = 2 * dim + 1 if l == 0 and case["op"] != "fem" else 3 ** dim
        var = 0 if case["op"] != "fd_periodic" else 1 if l == 0 else npt
        nnz = m * max(1.0, ball * n)

        def sweep():
            add((3 + var) * n * size, (2 * npt + 6) * n)
            add(nnz * (4 + size) + nnz * (8 + 3 * size), 4 * nnz + 2 * m * m)

        last = l == case["nlevel"] - 1
        if last and case["coarse"] == "Cholesky":
            add(n * (n + 1) * size, 2 * n * (n + 1))
            return
        if last:
            sweep(), sweep()
            return
        for _ in range(case["cycle"] if l else 1):
            for _ in range(2 if case["smoother"] == "SSOR" else 1):
                sweep(), sweep()
            nc = math.prod((c >> (l + 1)) - 1 for c in shape)
            add((4 + var) * n * size + 2 * nc * size, (2 * npt + 8) * n)
            level(l + 1)

    level(0)
    if case["kind"] == "solve":  # ten cycles to 1e-10, each with its FP64 residual and update
        return {"bytes": 10 * (total["bytes"] + 48.0 * n0), "flops": 10 * (total["flops"] + 20.0 * n0)}
    if case["kind"] == "adjoint":  # the step again, and two transposed sweeps for each sweep
        return {"bytes": 3 * case["steps"] * total["bytes"], "flops": 3 * case["steps"] * total["flops"]}
    return {"bytes": case["steps"] * total["bytes"] + (2 * 8.0 * n0 if case["kind"] == "apply" else 8.0 * n0),
            "flops": case["steps"] * total["flops"]}


# ------------------------------------------------- the same in 64-bit torch
_M0, _M1, _W0, _W1, _MASK = 0xD2511F53, 0xCD9E8D57, 0x9E3779B9, 0xBB67AE85, 0xFFFFFFFF
_DEV = "cuda"


def _mulhilo(a, m):
    """High and low 32 bits of a * m for 32-bit a in int64."""
    hi = (a * (m >> 16) + ((a * (m & 0xFFFF)) >> 16)) >> 16
    return hi & _MASK, (a * m) & _MASK


def _normals(x, y, sc, seed, lane):
    """Philox4x32-10 (Salmon et al. 2011) and Box-Muller: normal `lane` of the block of counter (x, y, sc)."""
    a, b = x & _MASK, y & _MASK
    c, d = torch.full_like(a, sc & _MASK), torch.full_like(a, sc >> 32)
    k0, k1 = seed & _MASK, seed >> 32
    for _ in range(10):
        h0, l0 = _mulhilo(a, _M0)
        h1, l1 = _mulhilo(c, _M1)
        a, b, c, d = h1 ^ b ^ k0, l1, h0 ^ d ^ k1, l0
        k0, k1 = (k0 + _W0) & _MASK, (k1 + _W1) & _MASK
    r, t = torch.where(lane < 2, a, c).double(), torch.where(lane < 2, b, d).double()
    rad = torch.sqrt(-2.0 * torch.log(r * 2.0 ** -32 + 2.0 ** -33))
    ang = (t * 2.0 ** -32 - 0.5) * (2.0 * math.pi)
    return rad * torch.where(lane % 2 == 0, torch.cos(ang), torch.sin(ang))


def _vec_normals(count, purpose, level, sc, seed):
    i = torch.arange(count, device=_DEV)
    return _normals(i >> 2, torch.full_like(i, (purpose << 24) | (level << 8)), sc, seed, i & 3)


def _restrict1(x, d):
    def every_second(first):
        return x.narrow(d, first, x.shape[d] - 2).index_select(d, at)
    at = torch.arange(0, x.shape[d] - 2, 2, device=x.device)
    return 0.5 * every_second(0) + every_second(1) + 0.5 * every_second(2)


def _prolong1(x, d):
    d = d % x.dim()
    pad = [0, 0] * (x.dim() - 1 - d) + [1, 1]
    xp = F.pad(x, pad)
    nc = x.shape[d]
    even = 0.5 * (xp.narrow(d, 0, nc + 1) + xp.narrow(d, 1, nc + 1))
    both = torch.stack([even.narrow(d, 0, nc), x], d + 1).flatten(d, d + 1)
    return torch.cat([both, even.narrow(d, nc, 1)], d)


class _Level64:
    """One level: weights by offset (numbers or arrays), colours, B."""

    def __init__(self, dim, N, weights, ncol, index):
        self.dim, self.N, self.w, self.ncol, self.index = dim, N, weights, ncol, index  # N = (N2, N1, N0)
        g = torch.meshgrid(*(torch.arange(k, device=_DEV) for k in N), indexing="ij")
        self.c, self.b, self.a = g
        self.colour = (self.a + self.b + self.c) & 1 if ncol == 2 else (self.a & 1) | (self.b & 1) << 1 | (self.c & 1) << 2

    def apply(self, x):
        xp = F.pad(x, (1, 1) * 3)
        y = 0.0
        for (dz, dy, dx), w in self.w.items():
            y = y + w * xp[..., 1 + dz:1 + dz + self.N[0], 1 + dy:1 + dy + self.N[1], 1 + dx:1 + dx + self.N[2]]
        return y

    def sweep(self, x, f, omega, forward):
        """One SOR sweep of the level's sparse part, colour by colour."""
        order = range(self.ncol) if forward else reversed(range(self.ncol))
        d = self.w[0, 0, 0]
        for k in order:
            x = torch.where(self.colour == k, x + omega / d * (f - self.apply(x)), x)
        return x

    def restrict(self, x):
        for d in range(self.dim):
            x = _restrict1(x, -1 - d)
        return x

    def prolong(self, x):
        for d in range(self.dim):
            x = _prolong1(x, -1 - d)
        return x

    def coarse(self):
        """R A P, read off from its products with 3^dim indicator vectors."""
        act = [1 if self.dim > 2 else 0, 1 if self.dim > 1 else 0, 1]
        Nc = tuple((k - 1) // 2 if a else 1 for k, a in zip(self.N, act))
        g = torch.meshgrid(*(torch.arange(k, device=_DEV) for k in Nc), indexing="ij")
        r3 = [range(3) if a else range(1) for a in act]
        offs = [(dz, dy, dx) for dz in ((-1, 0, 1) if act[0] else (0,)) for dy in ((-1, 0, 1) if act[1] else (0,))
                for dx in (-1, 0, 1)]
        w = {}
        for p in [(i, j, k) for i in r3[0] for j in r3[1] for k in r3[2]]:
            e = torch.ones(Nc, dtype=torch.bool, device=_DEV)
            for gi, pi, a in zip(g, p, act):
                if a:
                    e = e & (gi % 3 == pi)
            y = self.restrict(self.apply(self.prolong(e.double())))
            for o in offs:
                at = torch.ones(Nc, dtype=torch.bool, device=_DEV)
                for gi, pi, oi, a in zip(g, p, o, act):
                    if a:
                        at = at & ((gi + oi) % 3 == pi)
                w[o] = torch.where(at, y, w[o]) if o in w else torch.where(at, y, torch.zeros_like(y))
        return _Level64(self.dim, Nc, w, 2 ** self.dim, self.index + 1)

    def point_normals(self, sc, seed):
        N2, N1, N0 = self.N
        p = self.a + 1 if self.ncol == 2 else self.a
        groups = ((N0 + 1) >> 3) + 1 if self.ncol == 2 else (N0 + 7) >> 3
        return _normals((self.c * N1 + self.b) * groups + (p >> 3), (self.index << 8) | (p & 1), sc, seed, (p & 7) >> 1)

    def dense(self):
        n = math.prod(self.N)
        idx = torch.arange(n, device=_DEV).reshape(self.N)
        A = torch.zeros(n * n, dtype=torch.float64, device=_DEV)
        for o, w in self.w.items():
            src = tuple(slice(max(0, -k), m - max(0, k)) for k, m in zip(o, self.N))
            dst = tuple(slice(max(0, k), m + min(0, k)) for k, m in zip(o, self.N))
            rows, cols = idx[src].reshape(-1), idx[dst].reshape(-1)
            A = A.index_put((rows * n + cols,), (w + torch.zeros(self.N, dtype=torch.float64, device=_DEV))[src].reshape(-1))
        return A.reshape(n, n)


class _Chain64:
    """The chain of a case in 64-bit torch."""

    def __init__(self, case, inp, centre=None, log_sigma=None):
        self.case, self.seed = case, inp["noise_seed"]
        shape = _shape(case)
        self.dim = len(shape)
        N = tuple([1] * (3 - self.dim) + [c - 1 for c in reversed(shape)])
        fine = _Level64(self.dim, N, _fine_weights(case, centre), 2 ** self.dim if case["op"] == "fem" else 2, 0)
        self.L = [fine]
        for _ in range(case["nlevel"] - 1):
            self.L.append(self.L[-1].coarse())
        self.m = case["m"]
        if self.m:
            sigma = torch.from_numpy(inp["sigma"]).to(_DEV)
            self.sigma = sigma if log_sigma is None else torch.exp(log_sigma)
            B = torch.zeros((self.m, math.prod(N)), dtype=torch.float64, device=_DEV)
            for j, (i, v) in enumerate(inp["cols"]):
                B[j, torch.from_numpy(i).to(_DEV)] = torch.from_numpy(v).to(_DEV)
            B = B.reshape((self.m,) + N)
            for lv in self.L:
                lv.B = B
                lv.C, lv.S = [], []
                for fwd in (True, False):
                    C = torch.cat([lv.sweep(torch.zeros_like(b), b, case["omega"], fwd) for b in B.split(8)])
                    lv.C.append(C)
                    lv.S.append(torch.diag(self.sigma) + B.flatten(1) @ C.flatten(1).T)
                B = lv.restrict(B) if lv is not self.L[-1] else None
        last = self.L[-1]
        if case["coarse"] == "Cholesky" or case["kind"] == "solve":
            Q = last.dense()
            if self.m:
                Bc = last.B.flatten(1)
                Q = Q + Bc.T @ (Bc / self.sigma[:, None])
            self.chol = torch.linalg.cholesky(Q)

    def A(self, lv, x):
        y = lv.apply(x)
        if self.m:
            q = (lv.B.flatten(1) @ x.reshape(-1)) / self.sigma
            y = y + (lv.B.flatten(1).T @ q).reshape(x.shape)
        return y

    def sor(self, lv, x, f, forward, noisy):
        sc, omega, d = self.step_index * 4096 + self.inv, self.case["omega"], lv.w[0, 0, 0]
        if noisy:
            sd = (d * (2.0 - omega) / omega) ** 0.5
            x = lv.sweep(x, f + sd * lv.point_normals(sc, self.seed), omega, forward)
        else:
            x = lv.sweep(x, f, omega, forward)
        if self.m:
            k = 0 if forward else 1
            u = -(lv.B.flatten(1) @ x.reshape(-1))
            if noisy:
                u = u + torch.sqrt(self.sigma) * _vec_normals(self.m, 1, lv.index, sc, self.seed)
            z = torch.linalg.solve(lv.S[k], u)
            x = x + (lv.C[k].flatten(1).T @ z).reshape(x.shape)
        self.inv += noisy
        return x

    def cycle(self, l, x, f, noisy):
        lv, case = self.L[l], self.case
        if l == len(self.L) - 1:
            if case["coarse"] == "Cholesky" or not noisy:
                g = torch.linalg.solve_triangular(self.chol, f.reshape(-1, 1), upper=False)
                if noisy:
                    g = g + _vec_normals(g.shape[0], 2, lv.index, self.step_index * 4096 + self.inv, self.seed)[:, None]
                    self.inv += 1
                return torch.linalg.solve_triangular(self.chol.T, g, upper=True).reshape(x.shape)
            return self.sor(lv, self.sor(lv, x, f, True, noisy), f, False, noisy)
        ssor = case["smoother"] == "SSOR"
        for _ in range(case["cycle"] if l else 1):
            x = self.sor(lv, x, f, True, noisy)
            x = self.sor(lv, x, f, False, noisy) if ssor else x
            fc = lv.restrict(f - self.A(lv, x))
            x = x + lv.prolong(self.cycle(l + 1, torch.zeros_like(fc), fc, noisy))
            x = self.sor(lv, x, f, True, noisy) if ssor else x
            x = self.sor(lv, x, f, False, noisy)
        return x

    def step(self, k, x, f):
        self.step_index, self.inv = k, 0
        return self.cycle(0, x, f, 1)

    def solve(self, b):
        """Q x = b by noise-free cycles to the limit of 64 bits."""
        self.step_index, self.inv = 0, 0
        x, best = torch.zeros_like(b), math.inf
        for _ in range(60):
            r = b - self.A(self.L[0], x)
            rn = float(r.norm())
            if rn > 0.97 * best:
                break
            best = rn
            x = x + self.cycle(0, torch.zeros_like(b), r, 0)
        return x


def _fine_weights(case, centre=None):
    """Level 0's weights by offset (dz, dy, dx): FD, FD with the periodic correlation length, or Q1 elements."""
    shape = _shape(case)
    dim, vol = len(shape), math.prod(1.0 / c for c in shape)
    if case["op"] == "fem":  # tensor products of the 1D mass and stiffness matrices
        mass = [[1 / (6 * c), 4 / (6 * c), 1 / (6 * c)] for c in shape]
        stiff = [[-c, 2 * c, -c] for c in shape]
        w = {}
        for o in [(i, j, k) for i in ((-1, 0, 1) if dim > 2 else (0,)) for j in (-1, 0, 1) for k in (-1, 0, 1)]:
            off = [o[2], o[1], o[0]][:dim]
            v = case["kappa_sq"] * math.prod(mass[d][off[d] + 1] for d in range(dim))
            for s in range(dim):
                v += math.prod((stiff if d == s else mass)[d][off[d] + 1] for d in range(dim))
            w[o] = v
        return w
    w, diag = {}, sum(2.0 * vol * c * c for c in shape)
    for d, c in enumerate(shape):
        for s in (-1, 1):
            o = [0, 0, 0]
            o[2 - d] = s
            w[tuple(o)] = -vol * c * c
    if case["op"] == "fd_periodic":
        lam = torch.ones((), dtype=torch.float64, device=_DEV)
        for c in reversed(shape):  # x fastest
            lam = lam[..., None] * torch.cos(math.pi * torch.arange(1, c, dtype=torch.float64, device=_DEV) / c)
        lam = 0.5 * (LAMBDA[1] + LAMBDA[0]) + 0.5 * (LAMBDA[1] - LAMBDA[0]) * lam
        w[0, 0, 0] = (diag + vol / lam ** 2).reshape((1,) * (3 - dim) + tuple(lam.shape))
    else:
        w[0, 0, 0] = diag + vol * case["kappa_sq"] if centre is None else centre
    return w


def _exact_chain(case, inp):
    c = _Chain64(case, inp)
    x, f = (torch.from_numpy(inp[k]).to(_DEV).reshape(c.L[0].N) for k in ("x", "f"))
    i, v = (torch.from_numpy(a).to(_DEV) for a in _centre_ball(_shape(case)))
    z = []
    for k in range(case["steps"]):
        x = c.step(k, x, f)
        z.append((x.reshape(-1)[i] * v).sum())
    return x.reshape(-1), torch.stack(z)


def _exact_lrchol(case, inp):
    """Block Cholesky of A_0 along the last direction, thin QR of L^{-1} B (positive diagonal of R)."""
    lv = _Level64(len(_shape(case)), tuple([1] * (3 - len(_shape(case))) + [c - 1 for c in reversed(_shape(case))]),
                  _fine_weights(case), 2, 0)
    nb, p, n, m = lv.N[0], lv.N[1] * lv.N[2], math.prod(lv.N), case["m"]
    plane = _Level64(lv.dim, (2,) + lv.N[1:], lv.w, 2, 0).dense()
    Ain, Aoff = plane[:p, :p], plane[p:, :p]
    D, O, S = [], [], Ain
    for k in range(nb):
        D.append(torch.linalg.cholesky(S))
        if k + 1 < nb:
            O.append(torch.linalg.solve_triangular(D[k], Aoff.T, upper=False).T)
            S = Ain - O[k] @ O[k].T

    def lower(v):  # L^{-1} v
        out = []
        for k, b in enumerate(v.split(p)):
            out.append(torch.linalg.solve_triangular(D[k], b - O[k - 1] @ out[-1] if k else b, upper=False))
        return torch.cat(out)

    def upper(v):  # L^{-T} v
        out, v = [None] * nb, v.split(p)
        for k in reversed(range(nb)):
            b = v[k] - O[k].T @ out[k + 1] if k + 1 < nb else v[k]
            out[k] = torch.linalg.solve_triangular(D[k].T, b, upper=True)
        return torch.cat(out)

    g0 = lower(torch.from_numpy(inp["f"]).to(_DEV)[:, None])
    if m:
        B = torch.zeros((n, m), dtype=torch.float64, device=_DEV)
        for j, (i, v) in enumerate(inp["cols"]):
            B[torch.from_numpy(i).to(_DEV), j] = torch.from_numpy(v).to(_DEV)
        V = lower(B)
        Q, R = torch.linalg.qr(V)
        s = torch.sign(torch.diagonal(R))
        Q, R = Q * s, R * s[:, None]
        eye = torch.eye(m, dtype=torch.float64, device=_DEV)
        W = torch.linalg.cholesky(eye - R @ torch.linalg.solve(torch.diag(torch.from_numpy(inp["sigma"]).to(_DEV)) + V.T @ V, R.T))
        g0 = g0 + Q @ ((W.T - eye) @ (Q.T @ g0))
    out = []
    for k in range(case["steps"]):
        xi = _vec_normals(n, 4, 0, k * 4096, inp["noise_seed"])[:, None] + g0
        if m:
            xi = xi + Q @ ((W - eye) @ (Q.T @ xi))
        out.append(upper(xi).reshape(-1))
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return [_exact_chain(c, _inputs(c, [seed, 2, k]))[0] for k, c in enumerate(_batch_cases(case, seed))]
    inp = _inputs(case, seed)
    if kind == "lrchol":
        return _exact_lrchol(case, inp)
    if kind == "solve":
        c = _Chain64(case, inp)
        return {"x": c.solve(torch.from_numpy(inp["f"]).to(_DEV).reshape(c.L[0].N)).reshape(-1), "converged": None}
    if kind == "adjoint":
        s = _fine_weights(case)[0, 0, 0]
        s = torch.tensor(s, dtype=torch.float64, device=_DEV, requires_grad=True)
        ls = torch.log(torch.from_numpy(inp["sigma"]).to(_DEV)).requires_grad_()
        c = _Chain64(case, inp, s, ls)
        x0, f = (torch.from_numpy(inp[k]).to(_DEV).reshape(c.L[0].N).requires_grad_() for k in ("x", "f"))
        x = x0
        for k in range(case["steps"]):
            x = c.step(k, x, f)
        grads = torch.autograd.grad((x.reshape(-1) * torch.from_numpy(_xbar(case, seed)).to(_DEV)).sum(), [x0, f, s, ls])
        return {"xbar": grads[0].reshape(-1), "fbar": grads[1].reshape(-1), "centre": float(grads[2]), "log_sigma": grads[3]}
    x, z = _exact_chain(case, inp)
    return x if kind == "apply" else {"x": x, "z": z}
