"""GPU: the FP64 diagnostics where their terms nearly cancel or nearly agree, against 40-digit sums.

Rounding errors of a node are at most 2^-53 of the size that is rounded and independent from node to
node, so a sum of many is off by their root sum of squares: ten times that is the bound, with the
additions' own 2^-53 of the sum of the terms' sizes for each level of the reduction (20 at most)."""

import math
from decimal import Decimal, getcontext

import numpy as np
import pytest

from test_gpu_parity import gpu  # noqa: F401

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


def _dec(a):
    return [Decimal(float(v)) for v in np.ravel(a)]


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("n", [97, 300])
def test_damping_integral_near_balance(gpu, n, dtype):  # noqa: F811
    """n_res within 1e-3 of 1 at every node: three roundings of n_res a node (its denominator, c12 P and
    the quotient), whatever is left of n_res - 1."""
    torch = gpu
    from nls_gb300 import device, workloads as w
    getcontext().prec = 40
    c, dx = w.coeffs(), 0.15625
    rng = np.random.default_rng(n)
    u = (0.9 + 1e-3 * rng.random((n, n))) * np.exp(2j * np.pi * rng.random((n, n)))
    u = u.astype(dtype)
    d = np.abs(u.astype(np.complex128)) ** 2
    P = ((c[12] + c[13] * d) / c[11] * (1 + 1e-3 * rng.uniform(-1, 1, (n, n)))).astype(u.real.dtype)
    got = device.damping_integral(torch.tensor(u, device="cuda"), torch.tensor(P, device="cuda"), dx=dx, coeffs=c)
    c12, c13, c14 = (Decimal(float(c[k])) for k in (11, 12, 13))
    terms = []
    for x, y, p in zip(_dec(u.real), _dec(u.imag), _dec(P)):
        s = x * x + y * y
        terms.append((c12 * p / (c13 + c14 * s) - 1) * s)
    want = sum(terms) * Decimal(dx) ** 2
    size = math.fsum(float(abs(t)) for t in terms)
    bound = (10 * math.sqrt(3) * EPS * math.sqrt(math.fsum((d ** 2).ravel())) + 20 * EPS * size) * dx * dx
    assert abs(float(Decimal(got) - want)) <= bound


@pytest.mark.parametrize("case", ["no pump", "denormal", "infinite", "nan", "large", "no saturation"])
def test_damping_integral_values_at_the_ends(gpu, case):  # noqa: F811
    torch = gpu
    from nls_gb300 import device, workloads as w
    c, dx, n = w.coeffs(), 0.15625, 40
    rng = np.random.default_rng(1)
    u = (rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))).astype(np.complex64)
    P = rng.uniform(0, 6, (n, n)).astype(np.float32)
    if case == "no pump":
        P[:] = 0.0
    if case == "denormal":
        u[::3] = 1e-40 + 1e-42j
        P[::2] = 1e-41
    if case == "infinite":
        u[3, 4] = complex(np.inf, 0.0)
    if case == "nan":
        P[3, 4] = np.nan
    if case == "large":
        u = u * np.float32(1e18)
    if case == "no saturation":
        c = c.copy()
        c[13] = 0.0
    got = device.damping_integral(torch.tensor(u, device="cuda"), torch.tensor(P, device="cuda"), dx=dx, coeffs=c)
    U, Q = u.astype(np.complex128), P.astype(np.float64)
    d = U.real ** 2 + U.imag ** 2
    with np.errstate(all="ignore"):
        res = c[11] * Q / (c[12] + c[13] * d)
        term = (res - 1.0) * d * dx ** 2
        size = math.fsum(((res + 1.0) * d * dx ** 2).ravel())
    if case in ("infinite", "nan"):
        assert not math.isfinite(got) and math.isnan(got) == math.isnan(float(term.sum()))
    else:
        assert abs(got - math.fsum(term.ravel())) <= 24 * EPS * size
