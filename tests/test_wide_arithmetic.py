"""The arithmetic of the reference tables (a number as a sum of two doubles), against exact rationals."""
import os
import random
import subprocess
from fractions import Fraction
from math import isqrt

from conftest import ROOT

CSRC = os.path.join(ROOT, "hdiscontinuousgalerkin.jl_gb300", "csrc")

_PROGRAM = r"""
#include "tables.cpp"
#include <cstdio>
thread_local cudaStream_t g_alloc_stream = nullptr, g_use_stream = nullptr;
void order_streams(cudaStream_t, cudaStream_t) {}
int main() {
  double a, b, c, d;
  while (std::scanf("%la %la %la %la", &a, &b, &c, &d) == 4) {
    const Wide x(a, b), y(c, d);
    for (const Wide& r : {x, y, x + y, x - y, x * y, x / y, root(mag(x))}) std::printf("%a %a ", r.hi, r.lo);
    std::printf("%d %d %d\n", x < y, x >= y, x == y);
  }
}
"""


def test_operations_to_a_hundred_bits(tmp_path):
    (tmp_path / "t.cpp").write_text(_PROGRAM)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", CSRC, "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(cuda, "include"), "-o", str(tmp_path / "t"), str(tmp_path / "t.cpp"), "-L",
                    os.path.join(cuda, "lib64"), "-lcudart"], check=True)
    rng = random.Random(4)
    lines = []
    for _ in range(4000):
        v = [rng.choice([1, -1]) * rng.uniform(0.5, 1) * 2.0 ** rng.randint(-30, 30) for _ in range(2)]
        if rng.random() < 0.3:  # sums that cancel
            v[1] = -v[0] * (1 + rng.choice([0, 2.0 ** -rng.randint(20, 52)]))
        lines.append(" ".join(x.hex() for h in v for x in (h, h * 2.0 ** -53 * rng.uniform(-1, 1))))
    out = subprocess.run([str(tmp_path / "t")], input="\n".join(lines), capture_output=True, text=True, timeout=60).stdout
    rows = out.strip().split("\n")
    assert len(rows) == len(lines)
    for row in rows:
        w = row.split()
        x, y, s, d, p, q, r = [Fraction(float.fromhex(w[2 * k])) + Fraction(float.fromhex(w[2 * k + 1])) for k in range(7)]
        assert [int(v) for v in w[14:]] == [x < y, x >= y, x == y]
        # each operation rounds a handful of times at 2^-106
        for got, want in ((s, x + y), (d, x - y), (p, x * y), (q, x / y)):
            assert abs(got - want) <= Fraction(1, 2 ** 100) * abs(want)
        m = abs(x)
        want = Fraction(isqrt(m.numerator * m.denominator << 400), m.denominator << 200)
        assert abs(r - want) <= Fraction(1, 2 ** 98) * want
