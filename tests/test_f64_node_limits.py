"""The complex128 coefficients (csrc/f64_node.cuh, host form) where terms cancel, where there is no pump
and over steps of all lengths, against exact rationals.

The pairs hold each of a coefficient's two terms to 2^-45 of it; they may be used while dt/2 times a term
is below 2^-8, so while the error moves the state by less than a double's last place beside 1 (2^-53) per
term; else FP64, with at most four roundings of the terms' sizes."""

import os
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "nls_gb300", "csrc")

SOURCE = r"""
#include "f64_node.cuh"
#include <cstdio>
using namespace nlsg;
int main() {
  double v[11];
  for (;;) {
    for (int i = 0; i < 11; ++i) if (scanf("%la", &v[i]) != 1) return 0;
    // c3 c4 c5 c6 c12 c13 c14, ux uy P, dt
    PhysD ph{v[0], v[1], v[2], v[3], v[4], v[5], v[6]};
    const F64Consts c = make_f64(ph, v[10]);
    double A, B;
    const F2 p = f2_split(v[9]);
    const bool ok = f64_in_range(v[9]);
    const bool pairs = f64_coeffs_pairs(v[7], v[8], p, ok, c, A, B);
    if (!pairs) f64_coeffs_plain(v[7], v[8], v[9], c, A, B);
    const F2 x = f2_split(v[7]);
    printf("%d %a %a %a\n", (int)pairs, A, B, (double)x.h + (double)x.l);
  }
}
"""


@pytest.fixture(scope="module")
def node(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("f64limits")
    (d / "main.cpp").write_text(SOURCE)
    subprocess.run([cxx, "-O1", "-std=c++17", "-ffp-contract=off", "-I", CSRC, "-o", str(d / "main"), str(d / "main.cpp")],
                   check=True)

    def call(rows):
        text = "\n".join(" ".join(float(x).hex() for x in v) for v in rows)
        out = subprocess.run([str(d / "main")], input=text, capture_output=True, text=True, check=True).stdout
        for v, ln in zip(rows, out.splitlines()):
            t = ln.split()
            c3, c4, c5, c6, c12, c13, c14, x, y, P, _ = (Fraction(float(k)) for k in v)
            s = x * x + y * y
            r = c12 * P / (c13 + c14 * s)
            got = [Fraction(float.fromhex(k)) for k in t[1:]]
            yield dict(pairs=t[0] == "1", err=[got[0] - (c3 * r - c4), got[1] - (c5 * s + c6 * r)],
                       size=[abs(c3 * r) + abs(c4), abs(c5 * s) + abs(c6 * r)], split=(got[2] - x) / x if x else 0)
    return call


def _coeffs(rng):
    gamma, R, g_R = rng.uniform(0.3, 0.8), rng.uniform(0.5, 2.0), rng.uniform(1.0, 3.0)
    return [R / 2, gamma / 2, 1.0, 2 * g_R, 1.0, 1.0, R]


@pytest.mark.parametrize("dt", [1e-4, 1e-2, 0.1, 0.5, 4.0])
@pytest.mark.parametrize("what", ["A", "B"])
def test_cancelling_terms_at_steps_of_all_lengths(node, what, dt):
    rng = np.random.default_rng(7)
    rows = []
    for _ in range(200):
        c = _coeffs(rng)
        x, y = rng.normal(size=2)
        den = c[5] + c[6] * (x * x + y * y)
        if what == "A":       # gain meets loss
            P = c[1] / c[0] * den / c[4]
        else:                 # an attractive c5 |u|^2 against the reservoir's shift
            c[2] = -1.0
            P = (x * x + y * y) / c[3] * den / c[4]
        rows.append(c + [x, y, P, dt])
    half, eps = Fraction(dt) / 2, Fraction(1, 2 ** 53)
    for v in node(rows):
        for e, size in zip(v["err"], v["size"]):
            assert abs(e) <= (2 * eps / half if v["pairs"] else 4 * eps * size)


@pytest.mark.parametrize("power", [0.0, 0.1, 8.0])
def test_errors_over_the_benchmark_ranges(node, power):
    """With and without a pump: a value is split to 2^-49 of it, A and B hold their terms to 2^-45."""
    rng = np.random.default_rng(9)
    rows = [_coeffs(rng) + list(rng.uniform(-1, 1, 2)) + [power * rng.random(), 1e-4] for _ in range(4000)]
    for v in node(rows):
        assert v["pairs"] and abs(v["split"]) <= Fraction(1, 2 ** 49)
        assert all(abs(a) <= s * Fraction(1, 2 ** 45) for a, s in zip(v["err"], v["size"]))
