"""GPU: single solves spread over the whole GPU (k1d_wide.cuh, k2d_wide.cuh,
k2d_wide_reg.cuh) against the kernels that
batches
take, which compute every node with the same operations: bit for bit."""

import numpy as np
import pytest

from test_gpu_parity import _device_solve, _spec_1d, _spec_2d, gpu, rel  # noqa: F401

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


# one CTA, tiles without an interior, tiles of unequal size, one and two lanes a node, the largest
# grid held on chip and the smallest beyond it
@pytest.mark.parametrize("order", [3, 5])
@pytest.mark.parametrize("n,steps", [(5, 3), (7, 1), (16, 2), (41, 9), (100, 6), (173, 5), (256, 7), (333, 4), (520, 3),
                                     (530, 3)])
def test_square_complex128_equals_the_stage_kernels(gpu, order, n, steps):  # noqa: F811
    s = _spec_2d(n, order, seed=n)
    assert np.array_equal(_device_solve(gpu, s, steps, np.complex128, -1),
                          _device_solve(gpu, s, steps, np.complex128, 0))


# every region height, odd sides, one tile and the most, narrow last tiles, the largest grids held in
# registers (order 3: 840, order 5: 720) and the smallest beyond them
@pytest.mark.parametrize("order,variant,sizes", [(3, 15, (3, 41, 57, 64, 113, 200, 400, 555, 777, 840, 841)),
                                                 (5, 10, (5, 37, 97, 128, 241, 333, 512, 719, 720, 721))])
def test_square_complex64_equals_the_batch_kernels(gpu, order, variant, sizes):  # noqa: F811
    for n in sizes:
        s = _spec_2d(n, order, seed=n)
        for steps in (1, 2, 7):
            assert np.array_equal(_device_solve(gpu, s, steps, np.complex64, -1),
                                  _device_solve(gpu, s, steps, np.complex64, variant)), (n, steps)


def test_different_sizes_and_types_share_the_exchange_slots(gpu):  # noqa: F811
    """Launches of other layouts on the same slots, one after the other without a wait."""
    specs = [(_spec_1d(900, 5), np.complex64), (_spec_2d(120, 3), np.complex128), (_spec_1d(3000, 7), np.complex128),
             (_spec_2d(60, 5), np.complex128), (_spec_2d(150, 3), np.complex64), (_spec_1d(900, 3), np.complex64),
             (_spec_2d(300, 5), np.complex64)]
    first = [_device_solve(gpu, s, 13, dt, -1) for s, dt in specs]
    for _ in range(3):
        for (s, dt), want in zip(specs, first):
            assert np.array_equal(_device_solve(gpu, s, 13, dt, -1), want)


@pytest.mark.parametrize("case", ["nan", "inf", "zero", "huge", "long"])
def test_values_outside_the_float_pairs(gpu, case):  # noqa: F811
    """Nodes whose values leave the float pairs' range take the plain FP64 forms: non-finite values
    spread as in the stage kernels, a zero state stays zero, and steps so long that dt |b| exceeds
    the pairs' limit agree with the oracle."""
    from oracle import oracle
    s = _spec_2d(48, 3, seed=2)
    steps = 3
    if case in ("nan", "inf"):
        s.u0[20, 23] = complex(float(case), 0.0)
    if case == "zero":
        s.u0 = s.u0 * 0.0
    if case == "huge":
        s.u0 = s.u0 * 1e9
        s.dt = 1e-16
    if case == "long":
        s.dx, s.dt, s.u0 = 2.0, 0.05, s.u0 * 1e3
    got = _device_solve(gpu, s, steps, np.complex128, -1)
    stage = _device_solve(gpu, s, steps, np.complex128, 0)
    assert np.array_equal(got, stage, equal_nan=True)
    if case == "nan":
        # three steps of four stages spread it by 12 nodes along the axes, less along the diagonals
        assert np.isnan(got[20, 23]) and np.isnan(got[8, 23]) and np.isfinite(got[7, 23]) and np.isfinite(got[20, 36])
    elif case != "inf":
        want = oracle.solve(s.dt, s.dx, 3, steps, s.pumping, s.coeffs, s.u0, dtype=np.float64)
        assert rel(got, want) <= 1e-10 if case != "zero" else np.array_equal(got, want)


@pytest.mark.parametrize("kind", ["1d c64", "1d c128", "2d c64", "2d c128"])
def test_exchange_timeout_is_reported_and_the_context_recovers(gpu, oracle_lib, kind):  # noqa: F811
    """Waits for tags that nobody publishes (test control): they give up after about a second, the
    context's synchronize reports NLS_ERR_TIMEOUT, and the next solve is correct."""
    from nls_gb300 import _lib, device
    s = _spec_1d(700, 5) if kind[0] == "1" else _spec_2d(64, 3)
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
