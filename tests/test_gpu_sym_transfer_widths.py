"""Residual-restriction of symmetric FP64 stencils at row lengths between the
powers of two: CTAs of every multiple of 32 threads up to 256, and windows of
longer rows that share the columns evenly (test_gpu_sym_transfers has the
edges at the powers of two)."""
import pytest

import multigridmc_gb300 as M
from test_gpu_sym_transfers import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("op", ["fd", "fem"])
@pytest.mark.parametrize("shape", [(36, 4, 6), (66, 6, 4), (98, 4, 4), (130, 8), (164, 6), (194, 6), (226, 6), (260, 4),
                                   (272, 4, 4), (300, 6), (508, 4), (760, 4), (762, 4)])
def test_widths(shape, op):
    A = (M.LinearOperator.shifted_laplace_fd if op == "fd" else M.LinearOperator.shifted_laplace_fem)(shape, 10.0)
    _check(A, shape, M.FP64)
