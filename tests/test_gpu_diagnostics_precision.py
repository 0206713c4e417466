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


@pytest.mark.parametrize("power", [0.0, 2.0])
def test_complex128_chemical_potential_of_a_uniform_density(gpu, power):  # noqa: F811
    """|u|^2 and the pump the same at every node, so that a node's error does not average out.  About
    ten roundings a node and twenty levels of sums, each 2^-53 / sqrt(3) of the terms' sizes rms, so
    3.2 times 2^-53 over many amplitudes: at most 8."""
    torch = gpu
    from nls_gb300 import device, workloads as w
    getcontext().prec = 40
    c, dx, n = w.coeffs(), 1.0, 24
    cf = [Decimal(float(v)) for v in c]
    # the order-5 Laplacian of a constant, mean over the grid: the neighbours outside it are missing
    wt = {1: Decimal(16) / 12, 2: Decimal(-1) / 12}
    lost = sum(wt[d] for i in range(n) for d in (1, 2) for j in (i - d, i + d) if not 0 <= j < n)
    lap = -2 * n * lost / (n * n)
    errors = []
    for amp in np.random.default_rng(1).uniform(3, 30, 80):
        u = np.full((n, n), amp * np.exp(0.7j))
        mu = device.chemical_potential(torch.tensor(u, device="cuda"), torch.full((n, n), power, dtype=torch.float64,
                                                                                 device="cuda"), dx=dx, coeffs=c)
        x, y, p = Decimal(float(u[0, 0].real)), Decimal(float(u[0, 0].imag)), Decimal(power)
        s = x * x + y * y
        r = cf[11] * p / (cf[12] + cf[13] * s)
        a, b = cf[2] * r - cf[3], cf[4] * s + cf[5] * r
        # <u, H u> / <u, u> = a - i b + i lap, and mu is i times that
        size = float(abs(cf[2] * r) + cf[3] + b) + 5.0 + 68 / 12
        errors += [float(Decimal(mu.real) - (b - lap)) / size, float(Decimal(mu.imag) - a) / size]
    assert math.sqrt(np.mean(np.square(errors))) <= 8 * EPS


@pytest.mark.parametrize("n", [255, 256, 700])
def test_norm_of_a_nearly_uniform_state(gpu, n):  # noqa: F811
    """Nodes within 1e-3 of one amplitude, so that errors of equal sign add up: the last levels of the
    sums, a dozen, round to a double's last place, 2^-53 / sqrt(3) rms each: at most four of it over
    many amplitudes, and 8 of it is the bound."""
    torch = gpu
    from nls_gb300 import device
    rng = np.random.default_rng(n)
    errors = []
    for amp in rng.uniform(0.5, 3, 24):
        u = (amp * (1 + 1e-3 * rng.random((n, n))) * np.exp(0.3j)).astype(np.complex64)
        want = math.fsum(np.float64(u.real).ravel() ** 2) + math.fsum(np.float64(u.imag).ravel() ** 2)
        errors.append(device.norm(torch.tensor(u, device="cuda")) / want - 1)
    assert math.sqrt(np.mean(np.square(errors))) <= 8 * EPS
