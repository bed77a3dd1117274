"""The device's own reciprocals, cosine and exponential against the same in extended precision, at the error bounds that
their comments claim: a program of its own around the headers."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu
CSRC = os.path.join(ROOT, "hdiscontinuousgalerkin.jl_gb300", "csrc")

_PROGRAM = r"""
#include <cstdio>
#include <cstdint>
#include <vector>
#include "cg_sync.cuh"
thread_local cudaStream_t g_alloc_stream = nullptr, g_use_stream = nullptr;
void order_streams(cudaStream_t, cudaStream_t) {}
__global__ void k(int n, const uint64_t* in, uint64_t* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint64_t b = in[i];
  const double d = __longlong_as_double((long long)b);
  out[i] = (uint64_t)__double_as_longlong(recip(d));
  out[n + i] = (uint64_t)__double_as_longlong(recip_cubic(d));
  out[2 * n + i] = (uint64_t)cos_turns(b);
  out[3 * n + i] = (uint64_t)__double_as_longlong(exp2_minus(b));
}
int main(int argc, char** argv) {
  FILE* f = std::fopen(argv[1], "rb");
  std::fseek(f, 0, SEEK_END);
  const int n = (int)(std::ftell(f) / 8);
  std::rewind(f);
  std::vector<uint64_t> in(n), out(4 * (size_t)n);
  if ((int)std::fread(in.data(), 8, n, f) != n) return 2;
  uint64_t *a, *o;
  if (cudaMalloc(&a, 8 * (size_t)n) || cudaMalloc(&o, 32 * (size_t)n)) return 3;
  cudaMemcpy(a, in.data(), 8 * (size_t)n, cudaMemcpyHostToDevice);
  k<<<(n + 255) / 256, 256>>>(n, a, o);
  if (cudaMemcpy(out.data(), o, 32 * (size_t)n, cudaMemcpyDeviceToHost)) return 4;
  f = std::fopen(argv[2], "wb");
  std::fwrite(out.data(), 8, out.size(), f);
  std::fclose(f);
}
"""


@pytest.fixture(scope="module")
def evaluate(tmp_path_factory):
    import __graft_entry__ as g
    build = g._build_module()
    d = tmp_path_factory.mktemp("arith")
    (d / "t.cu").write_text(_PROGRAM)
    subprocess.run([build._nvcc(), *build.ARCH, "-O3", "-std=c++17", "-I", CSRC, "-I", os.path.join(ROOT, "include"), "-o",
                    str(d / "t"), str(d / "t.cu")], check=True, capture_output=True)

    def run(bits):
        np.asarray(bits, np.uint64).tofile(d / "in")
        subprocess.run([str(d / "t"), str(d / "in"), str(d / "out")], check=True, timeout=120)
        return np.fromfile(d / "out", np.uint64).reshape(4, -1)

    return run


LD = np.longdouble
PI = LD("3.14159265358979323846264338327950288419716939937510582")


def test_reciprocals(evaluate):
    rng = np.random.default_rng(1)
    d = np.concatenate([rng.uniform(1, 2, 60000) * 2.0 ** rng.integers(-1000, 1000, 60000), rng.uniform(1, 2, 60000),
                        [1.0, 2.0, np.nextafter(2, 1), 1e300, 1e-300, 1e-290, 1e290, 5e307, 1e-307, 3.0, 2.0 ** -1000]])
    d[::3] *= -1
    got = evaluate(d.view(np.uint64))[:2].view(np.float64)
    exact = LD(1) / LD(d)
    ulp = np.spacing(np.abs(np.float64(exact)))
    for r in got:
        assert (np.abs(LD(r) - exact) <= LD(ulp)).all()
    # beyond the range of the estimate: the division itself
    d = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1e-310, -2e-308, 1.7e308])
    with np.errstate(divide="ignore", over="ignore"):
        want = 1.0 / d
    for r in evaluate(d.view(np.uint64))[:2].view(np.float64):
        assert np.array_equal(r, want, equal_nan=True)


def test_cosine_of_a_phase(evaluate):
    rng = np.random.default_rng(2)
    q = 1 << 62
    edge = [(k * q + s) % (1 << 64) for k in range(5) for s in (-3, -2, -1, 0, 1, 2, 3)] + [1 << k for k in range(64)]
    t = np.concatenate([rng.integers(0, 1 << 64, 40000, np.uint64), np.array(edge, np.uint64)])
    got = evaluate(t)[2].view(np.int64)
    want = np.cos(2 * PI * (t.astype(LD) / LD(2) ** 64))
    # the square of the folded phase is cut at 2^-62, times the slope 1.24; Horner's last products at 2^-62 each; the
    # polynomial's 2^-67; a quarter turn taken as one unit less, 2^-61
    assert np.abs(got.astype(LD) / LD(2) ** 62 - want).max() <= LD(2) ** -59


def test_two_to_a_negative_power(evaluate):
    rng = np.random.default_rng(3)
    e = np.concatenate([rng.integers(0, 1021 << 54, 40000, np.uint64), rng.integers(0, 4 << 54, 40000, np.uint64),
                        np.array([n * (1 << 54) + s for n in (0, 1, 2, 31, 500, 1020) for s in (0, 1, (1 << 54) - 1)], np.uint64)])
    got = evaluate(e)[3].view(np.float64)
    want = LD(2) ** (-(e.astype(LD) / LD(2) ** 54))
    # rounded to 53 bits; the polynomial's 2^-58.6 and Horner's cuts below 2^-60
    assert np.abs(LD(got) / want - 1).max() <= LD(2) ** -53 + LD(2) ** -58
    assert (evaluate(np.array([1021 << 54, 1023 << 54, (1 << 64) - 1], np.uint64))[3] == 0).all()
