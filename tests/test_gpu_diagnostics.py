"""GPU: the FP64 diagnostics of device states against exactly rounded sums on the host.

The sums' error bound: float-pair groups and FP64 additions each stay below 2^-46 of the sum of the
terms' sizes, so 1e-13 of it; H(u) of a complex64 state is single precision, about 20 roundings of
2^-24 of the terms' sizes."""

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(n, dtype, kind):
    rng = np.random.default_rng(n)
    x = np.linspace(-1, 1, n)
    r2 = x[:, None] ** 2 + x[None, :] ** 2
    u = (0.8 * np.exp(-3 * r2) + 1e-3 * rng.normal(size=(n, n))) * np.exp(1j * r2)
    if kind == "tails":                    # rows of values the pairs cannot hold
        u = u * np.exp(-200.0 * r2)
        u[: n // 4] = 0.0
    if kind == "large":
        u = u * 1e15
    P = 6.0 * np.exp(-((np.sqrt(r2) - 0.5) ** 2) / 0.02)
    return u.astype(dtype), P.astype(np.float32 if dtype == np.complex64 else np.float64)


# one group, ragged groups and columns, around the size from which pairs are used, several passes a block
@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("kind,sizes", [("plain", (5, 17, 33, 255, 256, 257, 1000)), ("tails", (300,)), ("large", (300,))])
def test_square_grids(dtype, kind, sizes):
    import torch
    from nls_gb300 import device, workloads as w
    c = w.coeffs()
    dx = 0.15625
    for n in sizes:
        u, P = _state(n, dtype, kind)
        tu, tP = torch.tensor(u, device="cuda"), torch.tensor(P, device="cuda")
        U, Q = u.astype(np.complex128), P.astype(np.float64)
        d = U.real ** 2 + U.imag ** 2
        assert abs(device.norm(tu) - math.fsum(d.ravel())) <= 1e-13 * math.fsum(d.ravel())
        res = c[11] * Q / (c[12] + c[13] * d)
        term = (res - 1.0) * d * dx ** 2
        size = math.fsum(((res + 1.0) * d * dx ** 2).ravel())
        assert abs(device.damping_integral(tu, tP, dx=dx, coeffs=c) - math.fsum(term.ravel())) <= 1e-13 * size
        if kind == "large" and dtype == np.complex64:
            continue        # H(u) of a complex64 state is single precision: |u|^2 u overflows it
        lap = -60.0 * U
        mag = 60.0 * np.abs(U)
        for k, wt in ((1, 16.0), (2, -1.0)):
            for ax in (0, 1):
                for s in (-k, k):
                    v = np.zeros_like(U)
                    a = [slice(None)] * 2
                    b = [slice(None)] * 2
                    a[ax], b[ax] = (slice(s, None), slice(None, -s)) if s > 0 else (slice(None, s), slice(-s, None))
                    v[tuple(a)] = U[tuple(b)]
                    lap, mag = lap + wt * v, mag + abs(wt) * np.abs(v)
        lap, mag = lap / (12 * dx * dx), mag / (12 * dx * dx)
        a, b = c[2] * res - c[3], c[4] * d + c[5] * res
        h = (a - 1j * b) * U + 1j * lap
        M = math.fsum(d.ravel())
        S = complex(math.fsum((U.conj() * h).real.ravel()), math.fsum((U.conj() * h).imag.ravel()))
        size = math.fsum((np.abs(U) * ((np.abs(a) + np.abs(b) + c[3]) * np.abs(U) + mag)).ravel()) / M
        mu = device.chemical_potential(tu, tP, dx=dx, coeffs=c)
        assert abs(mu - 1j * S / M) <= (20 * 2.0 ** -24 if dtype == np.complex64 else 1e-13) * size


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("n", [100, 70000])
def test_non_finite_values_are_counted(dtype, n):
    import torch
    from nls_gb300 import _lib, device
    u = torch.full((n,), 0.5, dtype=torch.complex64 if dtype == np.complex64 else torch.complex128, device="cuda")
    assert abs(device.norm(u) - 0.25 * n) <= 1e-13 * n
    u[n // 2] = complex(0.0, float("inf"))
    u[n // 3] = complex(float("nan"), 1.0)
    with pytest.raises(_lib.NativeError) as err:
        device.norm(u)
    assert err.value.status == _lib.NLS_ERR_NONFINITE
