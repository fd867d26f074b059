"""The quotients without range handling (mam4b_physics.cuh) against the
division: quot_in_range and Divisor on pairs of the exponents they are used
for, half of them with mantissas at the ends of the binade, and with_quotients
on any bit patterns (zeros, subnormals, infinities, NaN). They are equal bit for
bit but for a power of two over a number one bit below a power of two, where
Markstein's correction lands on the middle of two doubles and rounds to the
lower one, and for the sign of a zero quotient."""

import ctypes
import os
import shutil
import subprocess

import pytest

from mam4xx_b200 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "mam4b_physics.cuh"
using namespace mam4b;

__device__ unsigned long long draw(unsigned long long &s) {  // splitmix64
  unsigned long long z = (s += 0x9e3779b97f4a7c15ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
// exponent within +-e, mantissa of any value or close to an end of the binade
__device__ double number(unsigned long long &s, int e) {
  unsigned long long m = draw(s) & 0xfffffffffffffull;
  const unsigned long long k = draw(s);
  if (k & 1)
    m = (k & 2) ? m & 63 : 0xfffffffffffffull - (m & 63);
  const unsigned long long x = 1023 - e + draw(s) % (2 * e);
  return __longlong_as_double((draw(s) << 63) | (x << 52) | m);
}
// Whether q is not what a / b may come out as.
__device__ bool wrong_quotient(double q, double a, double b) {
  const unsigned long long m = 0xfffffffffffffull;
  const unsigned long long x = __double_as_longlong(q), y = __double_as_longlong(a / b);
  if (x == y || q == a / b || (isnan(q) && isnan(a / b)))
    return false;
  const bool exception = (__double_as_longlong(a) & m) == 0 && (__double_as_longlong(b) & m) == m;
  return !(exception && x + 1 == y);
}

__global__ void compare(int what, unsigned long long seed, int rounds, unsigned *wrong) {
  unsigned long long s = seed + (blockIdx.x * blockDim.x + threadIdx.x) * 0x1000003ull;
  unsigned bad = 0;
  for (int i = 0; i < rounds; ++i) {
    if (what == 0) {
      const double a = number(s, 450), b = number(s, 450);
      bad += wrong_quotient(quot_in_range(a, b), a, b);
    } else if (what == 1) {
      const double b = number(s, 150);
      const Divisor d(b);
      for (int k = 0; k < 4; ++k) {
        const double a = number(s, 600);
        bad += wrong_quotient(d.under(a), a, b);
      }
    } else {
      // any bits; one operand in four zero, infinite, NaN or subnormal
      double v[4];
      for (int k = 0; k < 4; ++k) {
        v[k] = __longlong_as_double(draw(s));
        const unsigned long long kind = draw(s) % 32;
        if (kind < 4)
          v[k] = kind == 0 ? 0.0 : kind == 1 ? __longlong_as_double(0x7ffull << 52)
                 : kind == 2 ? nan("") : __longlong_as_double(draw(s) >> 12);
        else if (kind < 24)
          v[k] = number(s, 450);
      }
      double q0, q1, q2;
      with_quotients([&](auto &q) {
        const Divisor d = q.divisor(v[3]);
        q0 = q.quot(v[0], v[1]);
        q1 = q.under(d, v[0]);
        q2 = q.under(d, v[2]);
      });
      bad += wrong_quotient(q0, v[0], v[1]) + wrong_quotient(q1, v[0], v[3]) +
             wrong_quotient(q2, v[2], v[3]);
    }
  }
  if (bad)
    atomicAdd(wrong, bad);
}

extern "C" int run(int what, unsigned long long seed, int rounds, unsigned *count) {
  unsigned *d = nullptr;
  cudaError_t e = cudaMalloc(&d, sizeof(unsigned));
  if (e == cudaSuccess)
    e = cudaMemset(d, 0, sizeof(unsigned));
  if (e == cudaSuccess) {
    compare<<<1024, 256>>>(what, seed, rounds, d);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess)
    e = cudaMemcpy(count, d, sizeof(unsigned), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}
"""


@pytest.fixture(scope="module")
def quotients(tmp_path_factory):
    nvcc = os.environ.get("NVCC", "nvcc")
    if not shutil.which(nvcc):
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("quotients")
    src, lib = d / "quotients.cu", d / "quotients.so"
    src.write_text(SOURCE)
    subprocess.run([nvcc] + build.NVCC_FLAGS + ["-I", build.CSRC, str(src), "-o", str(lib)],
                   check=True)
    return ctypes.CDLL(str(lib))


@pytest.mark.parametrize("what", ["quot_in_range", "Divisor", "with_quotients"])
def test_quotients_are_the_divisions(cuda_device, quotients, what):
    wrong = ctypes.c_uint(~0 & 0xffffffff)
    k = ["quot_in_range", "Divisor", "with_quotients"].index(what)
    assert quotients.run(k, ctypes.c_ulonglong(7 + k), 1024, ctypes.byref(wrong)) == 0
    assert wrong.value == 0  # of 268 million, four and three times as many
