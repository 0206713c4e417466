"""GPU: complex64 square grids at grid steps so large that the stencil's weights vanish beside everything
else (they are the unit in which the kernels carry their slopes)."""

import numpy as np
import pytest

from test_gpu_parity import _device_solve, _spec_2d, gpu, rel  # noqa: F401

pytestmark = pytest.mark.gpu


# one register tile an SM, streaming, one register tile a launch, tiles in shared memory
@pytest.mark.parametrize("order,variant", [(3, -1), (3, 15), (3, 10), (5, -1), (5, 10), (5, 1)])
@pytest.mark.parametrize("dx", [1e3, 1e9, 1e12, 1e20, 1e60, 1e170])
def test_large_grid_steps(gpu, oracle_lib, order, variant, dx):  # noqa: F811
    s = _spec_2d(64, order, seed=3)
    rng = np.random.default_rng(4)
    s.u0 = 0.5 * (rng.normal(size=(64, 64)) + 1j * rng.normal(size=(64, 64)))
    s.dx, s.dt, steps = dx, 1e-2, 20
    got = _device_solve(gpu, s, steps, np.complex64, variant)
    want = oracle_lib.solve(s.dt, dx, order, steps, s.pumping, s.coeffs, s.u0, dtype=np.float64)
    assert rel(got, want) <= 3e-5
