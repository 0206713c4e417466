"""GPU: solves spread over the whole GPU beside other work on the GPU, what their results hold when a
wait between their CTAs has expired, and the kernels that take them where they cannot run."""

import ctypes
import threading
import time

import numpy as np
import pytest

from test_gpu_parity import _device_solve, _spec_1d, _spec_2d, gpu  # noqa: F401

pytestmark = pytest.mark.gpu

# (spec, type); the square grids of the last two need more SMs than the blocker leaves
CASES = {"1d c64": (lambda: _spec_1d(4096, 5), np.complex64), "1d c128": (lambda: _spec_1d(2501, 7), np.complex128),
         "2d c128": (lambda: _spec_2d(256, 3), np.complex128), "2d c64": (lambda: _spec_2d(840, 3), np.complex64)}


def _tensors(torch, s, dtype):
    c = dtype == np.complex128
    u = torch.tensor(np.ascontiguousarray(np.asarray(s.u0).T), dtype=torch.complex128 if c else torch.complex64, device="cuda")
    P = torch.tensor(np.ascontiguousarray(np.asarray(s.pumping).T), dtype=torch.float64 if c else torch.float32, device="cuda")
    return u, P


def _solve_on(ctx, s, u, P, iters):
    from nls_gb300 import _lib
    pr = _lib.make_problem(u.dim(), u.shape[0], s.order, s.dt, s.dx, s.coeffs, -1)
    code = _lib.dtype_code(np.complex64 if "64" in str(u.dtype) else np.complex128)
    _lib.check(_lib.lib().nls_solve_device(ctx.handle, code, ctypes.byref(pr), iters, ctypes.c_void_p(P.data_ptr()),
                                           ctypes.c_void_p(u.data_ptr())), "nls_solve_device", ctx.handle)


def test_beside_a_kernel_that_outlasts_the_bound_of_a_wait(gpu):  # noqa: F811
    """24 SMs are held for longer than a wait between CTAs may take by a batch of radial grids on the
    default context; solves on another context wait for them or run beside them, and are right."""
    torch = gpu
    from nls_gb300 import _lib
    from nls_gb300.batch import BatchSolver
    blocker = BatchSolver([_spec_1d(4096, 5) for _ in range(24)], dtype=np.complex64)
    blocker.run(20000)
    blocker.synchronize()
    t = time.perf_counter()
    blocker.run(20000)
    blocker.synchronize()
    steps = int(20000 * 4.0 / (time.perf_counter() - t))
    other = _lib.Context(0)
    todo = []
    for make, dtype in CASES.values():
        s = make()
        want = _device_solve(torch, s, 40, dtype, -1)
        todo.append((s, want) + _tensors(torch, s, dtype))
    torch.cuda.synchronize()
    blocker.run(steps)
    time.sleep(0.1)
    t = time.perf_counter()
    for s, _, u, P in todo:
        _solve_on(other, s, u, P, 40)
    other.synchronize()
    waited = time.perf_counter() - t
    blocker.synchronize()
    assert waited > 3.0, "the blocker did not hold the SMs for the time this test is about"
    for s, want, u, _ in todo:
        got = u.cpu().numpy()
        assert np.array_equal(got.T if s.dim == 2 else got, want)


def test_two_contexts_at_once(gpu):  # noqa: F811
    """Two threads, each with a context, solve grids that need most SMs at the same time."""
    torch = gpu
    from nls_gb300 import _lib
    jobs, bad = [], []
    for name in ("2d c64", "2d c128"):
        make, dtype = CASES[name]
        s = make()
        want = _device_solve(torch, s, 200, dtype, -1).T
        jobs.append((s, np.ascontiguousarray(want), _tensors(torch, s, dtype), _lib.Context(0)))
    torch.cuda.synchronize()

    def work(s, want, uP, ctx):
        try:
            for _ in range(20):
                u = uP[0].clone()
                torch.cuda.current_stream().synchronize()
                _solve_on(ctx, s, u, uP[1], 200)
                ctx.synchronize()
                if not np.array_equal(u.cpu().numpy(), want):
                    bad.append("wrong state")
        except Exception as e:
            bad.append(repr(e))
    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


@pytest.mark.parametrize("kind", list(CASES))
def test_expired_waits_leave_nan_where_the_state_is_not_right(gpu, kind):  # noqa: F811
    """Waits for tags that nobody publishes (test control): what did not depend on them is right bit
    for bit, everything else is NaN, and nodes next to the other CTAs' are among the latter."""
    from nls_gb300 import _lib, device
    s, dtype = (_spec_1d(700, 5) if kind[0] == "1" else _spec_2d(100, 3)), CASES[kind][1]
    for steps in (1, 2, 40):
        want = _device_solve(gpu, s, steps, dtype, -1)
        assert _lib.lib().nls_test_set_exchange_tag_extra(0, 1 << 20) == _lib.NLS_OK
        try:
            got = _device_solve(gpu, s, steps, dtype, -1)
            with pytest.raises(_lib.NativeError) as err:
                device.context(0).synchronize()
            assert err.value.status == _lib.NLS_ERR_TIMEOUT
        finally:
            assert _lib.lib().nls_test_set_exchange_tag_extra(0, 0) == _lib.NLS_OK
        bad = np.isnan(got)
        assert bad.any() and np.array_equal(got[~bad], want[~bad])
        assert np.array_equal(_device_solve(gpu, s, steps, dtype, -1), want)


@pytest.mark.parametrize("call", ["norm", "chemical_potential", "damping_integral", "density_errors"])
@pytest.mark.parametrize("kind", ["1d c128", "2d c64"])
def test_a_diagnostic_after_an_expired_solve_reports_it(gpu, kind, call):  # noqa: F811
    """The usual loop of solving in place and logging: the first blocking call says that the state is
    not valid, the next is the ordinary one again."""
    torch = gpu
    from nls_gb300 import _lib, device
    s, dtype = (_spec_1d(700, 5) if kind[0] == "1" else _spec_2d(100, 3)), CASES[kind][1]
    u, P = _tensors(torch, s, dtype)
    kw = dict(order=s.order, dt=s.dt, dx=s.dx, coeffs=s.coeffs, iters=1)

    def diagnostic(v):
        if call == "norm":
            return device.norm(v)
        if call == "density_errors":
            return device.density_errors(v, u.to(torch.complex128), P.double(), s.coeffs)
        return getattr(device, call)(v, P, dx=s.dx, coeffs=s.coeffs)
    want = diagnostic(device.solve_(u.clone(), P, **kw))
    assert _lib.lib().nls_test_set_exchange_tag_extra(0, 1 << 20) == _lib.NLS_OK
    try:
        v = device.solve_(u.clone(), P, **kw)
        with pytest.raises(_lib.NativeError) as err:
            diagnostic(v)
        assert err.value.status == _lib.NLS_ERR_TIMEOUT
    finally:
        assert _lib.lib().nls_test_set_exchange_tag_extra(0, 0) == _lib.NLS_OK
    device.context(0).synchronize()
    assert diagnostic(device.solve_(u.clone(), P, **kw)) == want


@pytest.mark.parametrize("decline", [1, 2])
@pytest.mark.parametrize("kind", list(CASES))
def test_without_memory_or_room_the_other_kernels_take_the_solve(gpu, kind, decline):  # noqa: F811
    """No memory for the exchange slots (1), no room for all CTAs at once (2): the same bits, by other
    launches, and by the first ones again afterwards."""
    from nls_gb300 import _lib, device
    s, dtype = (_spec_1d(700, 5) if kind[0] == "1" else _spec_2d(100, 3)), CASES[kind][1]
    want = _device_solve(gpu, s, 23, dtype, -1)
    ctx = device.context(0)
    assert _lib.lib().nls_test_set_exchange_state(ctx.handle, 0, decline) == _lib.NLS_OK
    try:
        before = ctx.launches
        assert np.array_equal(_device_solve(gpu, s, 23, dtype, -1), want)
        # one launch for all steps on a single CTA or cluster, else one or four a step
        assert ctx.launches - before == {"1d c64": 1, "1d c128": 1, "2d c128": 4 * 23, "2d c64": 23}[kind]
    finally:
        assert _lib.lib().nls_test_set_exchange_state(ctx.handle, 0, 0) == _lib.NLS_OK
    before = ctx.launches
    assert np.array_equal(_device_solve(gpu, s, 23, dtype, -1), want)
    assert ctx.launches - before == 1


@pytest.mark.parametrize("kind", list(CASES))
def test_tags_start_again_when_they_run_out(gpu, kind):  # noqa: F811
    """Solves of a few steps across the end of the tags, with the slots full of the largest ones."""
    from nls_gb300 import _lib
    s, dtype = (_spec_1d(700, 5) if kind[0] == "1" else _spec_2d(100, 3)), CASES[kind][1]
    want = _device_solve(gpu, s, 9, dtype, -1)
    u, P = _tensors(gpu, s, dtype)
    gpu.cuda.synchronize()
    ctx = _lib.Context(0)
    _solve_on(ctx, s, u.clone(), P, 1)      # allocates the slots
    assert _lib.lib().nls_test_set_exchange_state(ctx.handle, (1 << 31) - 1 - 100, 0) == _lib.NLS_OK
    for _ in range(40):
        v = u.clone()
        gpu.cuda.synchronize()
        _solve_on(ctx, s, v, P, 9)
        ctx.synchronize()
        got = v.cpu().numpy()
        assert np.array_equal(got.T if s.dim == 2 else got, want)


def test_under_capture_the_stage_kernels_take_the_solve(gpu):  # noqa: F811
    """A graph replays its launches with the same arguments, tags included: a captured solve takes the
    kernels without an exchange, and every replay advances the state."""
    torch = gpu
    from nls_gb300 import device
    s = _spec_2d(100, 3)
    u, P = _tensors(torch, s, np.complex128)
    kw = dict(order=s.order, dt=s.dt, dx=s.dx, coeffs=s.coeffs)
    want = device.solve_(u.clone(), P, iters=9, **kw)
    v = u.clone()
    device.solve_(v, P, iters=3, variant=0, **kw)      # allocates the stage buffers
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(side):
        graph.capture_begin()
        device.solve_(v, P, iters=3, **kw)
        graph.capture_end()
    torch.cuda.synchronize()
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(v, want)
