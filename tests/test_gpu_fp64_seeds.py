"""The quotients and square roots of nuvort_b200/csrc/fp64.cuh against the IEEE operations, operand by
operand, in a kernel built from that header: equal on random operands of the range the terms may
use; within a unit of the last place where numerator and divisor both lie a few units from powers
of two (their quotient can be the middle of two doubles but for 2^-52 of a unit); and, for
numerators so small that the residual n - q x is subnormal (below 2^-969; it is rounded to a
multiple of 2^-1074, at most a unit of the quotient's last place), within two."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#include "fp64.cuh"
__device__ unsigned long long mix(unsigned long long z) {
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
__device__ double power(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }
__device__ double random_in(unsigned long long z, int lo, int hi) {  // 2^lo <= x < 2^hi
  const int e = lo + (int)((z >> 52) % (unsigned)(hi - lo));
  return __longlong_as_double((long long)(e + 1023) << 52 | (long long)(z & 0xfffffffffffffull));
}
__device__ double near_power(unsigned long long z, int lo, int hi) {  // up to 8 units off a power of two
  const double p = power(lo + (int)((z >> 40) % (unsigned)(hi - lo)));
  return __longlong_as_double(__double_as_longlong(p) + (long long)(z % 17u) - 8);
}
// out: per kind {quotients off, their largest distance in units, roots off, their largest distance}
__global__ void check(int kind, unsigned long long seed, int per, unsigned long long *out) {
  unsigned long long off[2] = {0, 0}, far[2] = {0, 0};
  const unsigned long long first = (unsigned long long)(blockIdx.x * blockDim.x + threadIdx.x) * per;
  for (int k = 0; k < per; ++k) {
    const unsigned long long a = mix(seed + 2 * (first + k)), b = mix(seed + 2 * (first + k) + 1);
    const double x = kind == 1 ? near_power(a, -400, 400) : kind == 2 ? random_in(a, 0, 1) : random_in(a, -400, 400);
    const double n = kind == 1 ? near_power(b, -400, 400) : kind == 2 ? random_in(b, -1020, -969) : random_in(b, -400, 400);
    double ys;
    const double q[2] = {quot(n, x, near_rcp(x)), near_sqrt(x, ys)}, w[2] = {__ddiv_rn(n, x), __dsqrt_rn(x)};
    for (int c = 0; c < 2; ++c) {
      const long long d = llabs(__double_as_longlong(q[c]) - __double_as_longlong(w[c]));
      off[c] += d != 0;
      if ((unsigned long long)d > far[c]) far[c] = d;
    }
    // the quotients by a root, from the root's own reciprocal
    const long long d = llabs(__double_as_longlong(quot(n, q[1], ys)) - __double_as_longlong(__ddiv_rn(n, q[1])));
    off[0] += d != 0;
    if ((unsigned long long)d > far[0]) far[0] = d;
  }
  for (int c = 0; c < 2; ++c) {
    if (off[c]) atomicAdd(&out[2 * c], off[c]);
    atomicMax(&out[2 * c + 1], far[c]);
  }
}
extern "C" int run(int kind, unsigned long long seed, unsigned long long *host) {
  unsigned long long *d = nullptr;
  if (cudaMalloc(&d, 32) != cudaSuccess || cudaMemset(d, 0, 32) != cudaSuccess) return 1;
  check<<<1024, 256>>>(kind, seed, 256, d);
  if (cudaDeviceSynchronize() != cudaSuccess) return 2;
  const int bad = cudaMemcpy(host, d, 32, cudaMemcpyDeviceToHost) != cudaSuccess;
  cudaFree(d);
  return bad ? 3 : 0;
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    from nuvort_b200 import build
    d = tmp_path_factory.mktemp("fp64_seeds")
    (d / "check.cu").write_text(SOURCE)
    subprocess.run([build.NVCC, *build.ARCH, *build.FLAGS, "-I", build.CSRC, "-shared", str(d / "check.cu"), "-o", str(d / "check.so")],
                   check=True)
    lib = ctypes.CDLL(str(d / "check.so"))

    def call(kind, seed):
        out = np.zeros(4, np.uint64)
        assert lib.run(kind, ctypes.c_ulonglong(seed), out.ctypes.data_as(ctypes.c_void_p)) == 0
        return [int(v) for v in out]
    return call


@pytest.mark.parametrize("seed", [1, 2])
def test_random_operands_are_rounded_as_ieee(run, seed):
    assert run(0, seed) == [0, 0, 0, 0]  # 2^26 quotients by x, as many by a root, 2^26 roots


def test_operands_next_to_powers_of_two(run):
    _, quotient_units, roots_off, _ = run(1, 3)
    assert quotient_units <= 1 and roots_off == 0


def test_numerators_whose_residual_is_subnormal(run):
    assert run(2, 4)[1] <= 2
