"""The complex128 node arithmetic (csrc/f64_node.cuh) in its host form, against exact rationals.

Bounds, derived from the representation: the reservoir and the coefficients A and B are pairs of
floats, every operation on them rounded at 2^-47 or better, about eight on the longest chain:
2^-44 of the sum of the terms' sizes.  The stencil's neighbour part is a fixed-point sum with at
least 3 bits below a double's last place, multiplied and rounded once: 2^-52 of the sum of the
terms' sizes, 2^-51.5 for the plain additions it falls back to.  Values outside the pairs' range
take FP64 with a quotient good to 2^-42.
"""

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
  char what;
  while (scanf(" %c", &what) == 1) {
    double v[12];
    const int count = what == 'c' ? 10 : what == '1' ? 5 : 9;
    for (int i = 0; i < count; ++i) if (scanf("%la", &v[i]) != 1) return 1;
    if (what == 'c') {  // c3 c4 c5 c6 c12 c13 c14, ux uy P
      PhysD ph{v[0], v[1], v[2], v[3], v[4], v[5], v[6]};
      const F64Consts c = make_f64(ph, 1e-4);
      double A, B;
      if (!f64_coeffs_pairs(v[7], v[8], f2_split(v[9]), f64_in_range(v[9]), c, A, B))
        f64_coeffs_plain(v[7], v[8], v[9], c, A, B);
      printf("%a %a\n", A, B);
    } else {
      const F64Consts c = make_f64(PhysD{}, 1e-4, 0.0, v[0]);
      double w[8];
      bool ok;
      if (what == '1') {
        double a[4];
        for (int i = 0; i < 4; ++i) a[i] = v[1 + i];
        w[0] = cross_sum_fixed<1>(a, c, ok);
        if (!ok) w[0] = cross_sum_plain<1>(a, c);
      } else {
        double a[8];
        for (int i = 0; i < 8; ++i) a[i] = v[1 + i];
        w[0] = cross_sum_fixed<2>(a, c, ok);
        if (!ok) w[0] = cross_sum_plain<2>(a, c);
      }
      printf("%a\n", w[0]);
    }
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def node(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("f64node")
    (d / "main.cpp").write_text(SOURCE)
    subprocess.run([cxx, "-O1", "-std=c++17", "-ffp-contract=off", "-I", CSRC, "-o", str(d / "main"), str(d / "main.cpp")],
                   check=True)

    def call(lines):
        text = "\n".join(w + " " + " ".join(float(x).hex() if np.isfinite(x) else str(float(x)) for x in v)
                         for w, v in lines)
        out = subprocess.run([str(d / "main")], input=text, capture_output=True, text=True, check=True).stdout
        return [[float.fromhex(t) for t in ln.split()] for ln in out.splitlines()]
    return call


@pytest.mark.parametrize("amp,power", [(1e-3, 8.0), (1.0, 8.0), (3.0, 1e-9), (1e-25, 1.0), (0.0, 1.0), (1.0, 0.0),
                                       (1.0, -2.0)])
def test_coefficients_in_float_pairs(node, amp, power):
    rng = np.random.default_rng(3)
    rows = []
    for _ in range(300):
        c = [rng.uniform(.25, 1), rng.uniform(.1, .5), rng.uniform(.1, 2), rng.uniform(2, 6), rng.uniform(.1, 2),
             rng.uniform(2.5, 4), rng.uniform(.3, 1)]
        rows.append(c + [amp * rng.normal(), amp * rng.normal(), power * rng.uniform(0.1, 1)])
    for v, (A, B) in zip(rows, node([("c", v) for v in rows])):
        c3, c4, c5, c6, c12, c13, c14, x, y, P = (Fraction(t) for t in v)
        s = x * x + y * y
        r = c12 * P / (c13 + c14 * s)
        assert abs(Fraction(A) - (c3 * r - c4)) <= (abs(c3 * r) + c4) * Fraction(1, 2 ** 44)
        # coefficients below 2^-70 keep single precision only: nothing beside the stencil's centre
        assert abs(Fraction(B) - (c5 * s + c6 * r)) <= (c5 * s + abs(c6 * r)) * Fraction(1, 2 ** 44) + Fraction(1, 2 ** 90)


def test_coefficients_outside_the_pairs_range(node):
    base = [0.5, 0.2, 1.0, 4.0, 1.0, 1.0, 1.0]
    rows = [base + [1e9, 0.0, 2.0], base + [1.0, 1.0, 1e30], [0.5, 0.2, 1e9, 4.0, 1.0, 1.0, 1.0, 0.3, 0.4, 2.0],
            [0.5, 0.2, 1.0, 4.0, 1.0, 0.0, 1.0, 1e-20, 0.0, 1e-42], base + [2000.0, 0.0, 2.0]]
    for v, (A, B) in zip(rows, node([("c", v) for v in rows])):
        c3, c4, c5, c6, c12, c13, c14, x, y, P = (Fraction(t) for t in v)
        s = x * x + y * y
        r = c12 * P / (c13 + c14 * s)
        assert abs(Fraction(A) - (c3 * r - c4)) <= (abs(c3 * r) + c4) * Fraction(1, 2 ** 41)
        assert abs(Fraction(B) - (c5 * s + c6 * r)) <= (c5 * s + abs(c6 * r)) * Fraction(1, 2 ** 41)
    for bad in (float("nan"), float("inf")):
        for k in (7, 8, 9):
            v = base + [0.3, 0.4, 2.0]
            v[k] = bad
            (A, B), = node([("c", v)])
            assert not (np.isfinite(A) and np.isfinite(B)) or (k < 9 and np.isinf(bad) and not np.isfinite(B)), (k, bad)


@pytest.mark.parametrize("K", [1, 2])
@pytest.mark.parametrize("kind", ["near", "signs", "spread", "zeros", "tiny", "huge"])
def test_neighbour_part(node, K, kind):
    rng = np.random.default_rng(5)
    rows = []
    for _ in range(400):
        v = rng.uniform(-1, 1, 4 * K)
        if kind == "near":
            v = 1 + 0.01 * v
        if kind == "spread":
            v = np.ldexp(v, rng.integers(-80, 80, 4 * K))
        if kind == "zeros":
            v = np.where(rng.random(4 * K) < 0.5, 0.0, v)
        if kind == "tiny":
            v = np.ldexp(v, -1000)
        if kind == "huge":
            v = np.ldexp(v, 1000)
        rows.append([rng.uniform(20, 50)] + list(v))
    for v, (got,) in zip(rows, node([(str(K), v) for v in rows])):
        f = [Fraction(t) for t in v]
        near, far = f[1:5], f[5:]
        want = f[0] * ((16 if K == 2 else 1) * sum(near) - sum(far))
        size = abs(f[0]) * ((16 if K == 2 else 1) * sum(map(abs, near)) + sum(map(abs, far)))
        bound = Fraction(2) ** -52 if kind not in ("tiny", "huge") else Fraction(2) ** -51 * Fraction(8, 10)
        assert abs(Fraction(got) - want) <= size * bound, (got, float(want))


def test_neighbour_part_special_values(node):
    u = 41.0
    rows = [[u, 0.0, 0.0, 0.0, 0.0], [u, 1.5, -1.5, 0.0, 0.0], [u, 1.0, float("nan"), 2.0, 3.0],
            [u, 1.0, float("inf"), 2.0, 3.0], [u, float("inf"), -float("inf"), 2.0, 3.0], [u, 5e-324, 0.0, 0.0, 0.0]]
    got = [g[0] for g in node([("1", v) for v in rows])]
    assert got[0] == 0.0 and got[1] == 0.0 and got[5] == 41 * 5e-324
    assert np.isnan(got[2]) and got[3] == float("inf") and np.isnan(got[4])
