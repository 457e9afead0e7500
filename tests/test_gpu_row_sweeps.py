"""Colour passes against a plain numpy sweep in 64 bits: 9- and 27-point levels
(two colours of a row per launch) at the edges of their row widths -- rows of
one point, of odd and even length, one CTA's longest row and one point more
(which runs one colour per launch) -- and red-black levels with pitches that
take the vector pass and ones that do not."""
import numpy as np
import pytest

import multigridmc_gb300 as M

pytestmark = pytest.mark.gpu


def _stencil(dim, symmetric):
    """A diagonally dominant 3^dim-point stencil, equal or unequal at +-offsets."""
    st = np.zeros(27)
    for k in range(27):
        d = [k % 3 - 1, (k // 3) % 3 - 1, k // 9 - 1]
        if any(d[dim:]):
            continue
        st[k] = -0.1 / (1 + abs(d[0]) + 2 * abs(d[1]) + 4 * abs(d[2]))
        if not symmetric:
            st[k] *= 1 + 0.1 * d[0] - 0.05 * d[1] + 0.02 * d[2]
    st[13] = 1.0 - st.sum() + st[13]
    return st


def _normals(a, b, c, N, level, sc, seed, axis=False):
    """Philox4x32-10 and Box-Muller in 64 bits: the normal of point (a, b, c)
    of a 3^dim-point level, or of a red-black one (axis)."""
    m = np.uint64(0xFFFFFFFF)
    groups = ((N[0] + 1) >> 3) + 1 if axis else (N[0] + 7) >> 3
    a = a + 1 if axis else a
    grp = ((c * N[1] + b) * groups + (a >> 3)).astype(np.uint64)
    ctr = [grp, (np.uint64(level << 8) | (a & 1).astype(np.uint64)), np.full_like(grp, sc & 0xFFFFFFFF),
           np.full_like(grp, sc >> 32)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = ctr[0] * np.uint64(0xD2511F53), ctr[2] * np.uint64(0xCD9E8D57)
        ctr = [(p1 >> np.uint64(32)) ^ ctr[1] ^ np.uint64(k0), p1 & m, (p0 >> np.uint64(32)) ^ ctr[3] ^ np.uint64(k1), p0 & m]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    lane = (a & 7) >> 1
    u = np.where(lane < 2, ctr[0], ctr[2]).astype(float) * 2.0 ** -32 + 2.0 ** -33
    ang = (np.where(lane < 2, ctr[1], ctr[3]).astype(float) * 2.0 ** -32 - 0.5) * 2 * np.pi
    return np.sqrt(-2 * np.log(u)) * np.where(lane % 2 == 0, np.cos(ang), np.sin(ang))


def _sweep(st, dim, x, f, omega, forward):
    """One multicolour SOR sweep (colour = parities of a, b, c) of x[c, b, a]."""
    c, b, a = np.indices(x.shape)
    axis = np.count_nonzero(st) <= 2 * dim + 1
    colour = (a + b + c) & 1 if axis else (a & 1) | (b & 1) << 1 | (c & 1) << 2
    ncol = 2 if axis else 2 ** dim
    order = range(ncol) if forward else reversed(range(ncol))
    for k in order:
        xp = np.pad(x, 1)
        y = sum(st[(dz + 1) * 9 + (dy + 1) * 3 + dx + 1] *
                xp[1 + dz:1 + dz + x.shape[0], 1 + dy:1 + dy + x.shape[1], 1 + dx:1 + dx + x.shape[2]]
                for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1))
        x = np.where(colour == k, x + omega / st[13] * (f - y), x)
    return x


SHAPES = [(2, 4, 4), (9, 3, 2), (16, 6, 5), (66, 5, 4), (33, 8), (130, 6), (131, 4), (513, 4), (514, 4), (513, 4, 3)]


@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("shape", SHAPES)
def test_row_sweeps(shape, symmetric, precision):
    _check(shape, _stencil(len(shape), symmetric), 1.2, precision)


@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
@pytest.mark.parametrize("omega", [1.0, 1.2])
@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("shape", [(2, 3, 4), (8, 5, 4), (12, 8, 3), (33, 4, 5), (9,), (8, 6), (7, 5), (200, 16, 16)])
def test_red_black_sweeps(shape, symmetric, omega, precision):
    st = _stencil(len(shape), symmetric)
    for k in range(27):
        if sum(d != 1 for d in (k % 3, (k // 3) % 3, k // 9)) > 1:
            st[k] = 0.0
    _check(shape, st, omega, precision)


def _check(shape, st, omega, precision):
    dim, seed = len(shape), 5
    N = [s - 1 for s in shape] + [1] * (3 - dim)
    axis = np.count_nonzero(st) <= 2 * dim + 1
    op = M.LinearOperator(shape, st)
    s = M.SSORSampler(op, omega=omega, precision=precision, seed=seed)
    rng = np.random.default_rng(2)
    f = rng.standard_normal(op.n)
    # per point 27 terms of size <= 1 and a diagonal >= 1: 27 roundings in a
    # sum, carried through at most 2^dim colours; the in-kernel normals are
    # FP32 approximations, off by up to 2e-4 where u is within 1e-7 of 1
    eps = 2.0 ** -52 if precision == M.FP64 else 2.0 ** -23
    c, b, a = np.indices(N[::-1])
    for forward in (True, False):
        for noisy in (False, True):
            x = rng.standard_normal(op.n)
            cval = f.reshape(N[::-1])
            if noisy:
                sd = np.sqrt(st[13] * (2 - omega) / omega)
                cval = cval + sd * _normals(a, b, c, N, 0, 4095, seed, axis)
            want = _sweep(st, dim, x.reshape(N[::-1]), cval, omega, forward).reshape(-1)
            s.sor(0, M.FORWARD if forward else M.BACKWARD, f, x, with_noise=noisy)
            assert np.max(np.abs(x - want)) < (5e-4 if noisy else 27 * 8 * 4 * eps)
    s.close()
