"""A single non-finite state entry is not overwritten by a sweep: whatever its
colour, an observable over it raises MGMC_ERR_NONFINITE (omega = 1, where the
new value of a point could be formed without its old one, included)."""
import numpy as np
import pytest

import multigridmc_gb300 as M

pytestmark = pytest.mark.gpu

OPS = {"fd-2d": lambda: M.LinearOperator.shifted_laplace_fd((12, 10), 10.0),
       "fd-3d": lambda: M.LinearOperator.shifted_laplace_fd((8, 12, 10), 10.0),
       "fem-2d": lambda: M.LinearOperator.shifted_laplace_fem((12, 10), 10.0),
       "fem-3d": lambda: M.LinearOperator.shifted_laplace_fem((8, 12, 10), 10.0)}


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("omega", [1.0, 1.3])
@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
@pytest.mark.parametrize("name", OPS)
def test_one_entry(name, precision, omega, bad):
    op = OPS[name]()
    nx, ny = op.shape[0] - 1, op.shape[1] - 1
    s = M.SSORSampler(op, omega=omega, precision=precision)
    f = np.ones(op.n)
    for colour in range(2 ** len(op.shape)):  # an interior point of every colour
        k = 2 + (colour & 1) + (2 + (colour >> 1 & 1)) * nx + (2 + (colour >> 2) if len(op.shape) == 3 else 0) * nx * ny
        for direction in (M.FORWARD, M.BACKWARD):
            x = np.zeros(op.n)
            x[k] = bad
            s.sor(0, direction, f, x, with_noise=True)
            assert not np.isfinite(x[k]), (colour, direction)
    s.close()


@pytest.mark.parametrize("precision", [M.FP64, M.FP32_MIXED])
@pytest.mark.parametrize("name", OPS)
def test_reported(name, precision):
    op = OPS[name]()
    for k in (0, 1, op.shape[0] - 1, op.shape[0]):
        s = M.MultigridMCSampler(op, M.MultigridParameters(nlevel=2), precision=precision)
        s.set_observable(np.array([k]), np.ones(1), 4)
        x = np.zeros(op.n)
        x[k] = np.nan
        s.set_state(x)
        s.step(1)
        with pytest.raises(M.MGMCError) as e:
            s.read_observations(4)
        assert e.value.name == "MGMC_ERR_NONFINITE"
        s.close()
