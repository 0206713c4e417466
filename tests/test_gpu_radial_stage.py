"""GPU: radial complex128 grids by stage kernels, which form a node's operator row for every stage, against
the kernels that form it once a launch: the same operations, bit for bit."""

import numpy as np
import pytest

from test_gpu_parity import _device_solve, _spec_1d, gpu, rel  # noqa: F401

pytestmark = pytest.mark.gpu


# a few nodes beyond the near-axis rows, ragged last blocks of threads, one that several blocks hold
@pytest.mark.parametrize("order", [3, 5, 7])
@pytest.mark.parametrize("n,dx", [(8, 0.04), (255, 0.1), (257, 0.04), (1000, 0.04), (2501, 0.3)])
def test_stage_kernels_equal_the_spread_solve(gpu, oracle_lib, order, n, dx):  # noqa: F811
    s = _spec_1d(n, order, seed=n, dx=dx)
    stage = _device_solve(gpu, s, 19, np.complex128, 0)
    assert np.array_equal(stage, _device_solve(gpu, s, 19, np.complex128, -1))
    assert rel(stage, oracle_lib.solve(s.dt, s.dx, order, 19, s.pumping, s.coeffs, s.u0, dtype=np.float64)) <= 1e-12
