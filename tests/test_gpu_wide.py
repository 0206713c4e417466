"""GPU: single solves spread over the whole GPU (k1d_wide.cuh, k2d_wide.cuh,
k2d_wide_reg.cuh) against the kernels that
batches
take, which compute every node with the same operations: bit for bit."""

import numpy as np
import pytest

from test_gpu_parity import _device_solve, _spec_1d, gpu, rel  # noqa: F401

pytestmark = pytest.mark.gpu


def _batch(s, steps, dtype):
    from nls_gb300.batch import BatchSolver
    b = BatchSolver([s], dtype=dtype)
    b.run(steps)
    return b.get(0)


# sizes around one CTA's segment and its halo, ragged last segments, the largest of one and of
# several CTAs an SM, step counts below, at and beyond the steps per exchange
@pytest.mark.parametrize("order", [3, 5, 7])
@pytest.mark.parametrize("n,steps", [(64, 1), (65, 3), (257, 8), (300, 9), (1000, 33), (2501, 17), (8192, 20)])
@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
def test_radial_equals_the_batch_kernels(gpu, order, n, steps, dtype):  # noqa: F811
    s = _spec_1d(n, order, seed=n)
    got = _device_solve(gpu, s, steps, dtype, -1)
    assert np.array_equal(got, _batch(s, steps, dtype))


@pytest.mark.parametrize("n,dtype", [(29000, np.complex64), (20001, np.complex128)])
def test_radial_large_grids(gpu, n, dtype):  # noqa: F811
    s = _spec_1d(n, 5, seed=1)
    assert np.array_equal(_device_solve(gpu, s, 21, dtype, -1), _batch(s, 21, dtype))


@pytest.mark.parametrize("kind", ["1d c64", "1d c128", "2d c64", "2d c128"])
def test_exchange_timeout_is_reported_and_the_context_recovers(gpu, oracle_lib, kind):  # noqa: F811
    """Waits for tags that nobody publishes (test control): they give up after about a second, the
    context's synchronize reports NLS_ERR_TIMEOUT, and the next solve is correct."""
    from nls_gb300 import _lib, device
    s = _spec_1d(700, 5)
    dtype = np.complex64 if kind.endswith("c64") else np.complex128
    assert _lib.lib().nls_test_set_exchange_tag_extra(0, 1 << 20) == _lib.NLS_OK
    try:
        _device_solve(gpu, s, 6, dtype, -1)
        with pytest.raises(_lib.NativeError) as err:
            device.context(0).synchronize()
        assert err.value.status == _lib.NLS_ERR_TIMEOUT
    finally:
        assert _lib.lib().nls_test_set_exchange_tag_extra(0, 0) == _lib.NLS_OK
    got = _device_solve(gpu, s, 40, dtype, -1)
    want = oracle_lib.solve(s.dt, s.dx, s.order, 40, s.pumping, s.coeffs, s.u0,
                            dtype=np.float32 if dtype == np.complex64 else np.float64)
    assert rel(got, want) <= (3e-5 if dtype == np.complex64 else 1e-10)
