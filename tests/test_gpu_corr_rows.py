"""A CTA of the low-rank correction whose rows lie beyond 2^31 in the row lists
of a level (the lists' earlier part is allocated, not filled)."""
import ctypes as C

import numpy as np
import pytest

from gpu_helpers.build import build as gpu_build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("base", [0, 512, 2 ** 31 - 300, 2 ** 31 + 512])
def test_rows_from(base):
    lib = C.CDLL(gpu_build("corr_rows_check"))
    n, nx = 700, 1000
    rng = np.random.default_rng(3)
    rows = rng.permutation(nx)[:n].astype(np.uint32)
    cols = rng.integers(0, 2, n).astype(np.int32)
    vals = rng.integers(-8, 9, n).astype(np.float32)
    x = rng.integers(-8, 9, nx).astype(np.float32)
    want = x.copy()
    want[rows] += vals * np.where(cols == 0, np.float32(3.0), np.float32(-5.0))  # small integers: exact
    P = lambda a, t: a.ctypes.data_as(C.POINTER(t))
    assert lib.corr_rows_check(C.c_longlong(base), n, P(rows, C.c_uint), P(cols, C.c_int), P(vals, C.c_float), C.c_float(3.0),
                               C.c_float(-5.0), P(x, C.c_float), nx) == 0
    assert np.array_equal(x, want)
