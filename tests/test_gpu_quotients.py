"""The paired FP32 quotient of the WENO weight sums (vnquot in weno.cuh) against IEEE division. Its reciprocal is compared
for every denominator's significand; the quotient wherever it could be rounded the other way. With a reciprocal right
to half an ulp the first quotient is within 1.5 ulp and its correction errs by less than 2^-22 ulp, so only exact
quotients that close to the middle between two FP32 numbers are in question: for numerator n and denominator d as
24-bit integers, 2^(k+1) n = (2 j + 1) d + c with |c| <= 8. The kernel solves that for every d and every |c| <= 16."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

CSRC = Path(__file__).resolve().parent.parent / "multigpu_advectiondiffusion_gb300" / "csrc"
SOURCE = r"""
#include "weno.cuh"
using namespace adv;
typedef unsigned long long u64;

__device__ u64 counts[3];  // quotients compared, quotients that differ, reciprocals that differ

__device__ void compare(unsigned n, unsigned d) {
  const float x = (float)n, y = (float)d;
  const float2 q = vnquot<float>(make_float2(x, -x * 0x1p-40f), make_float2(y, y * 0x1p-30f));
  atomicAdd(&counts[0], 1ull);
  if (q.x != -__fdiv_rn(x, y) || q.y != __fdiv_rn(x * 0x1p-40f, y * 0x1p-30f)) atomicAdd(&counts[1], 1ull);
}

__global__ void check() {
  const unsigned d = (1u << 23) + blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= 1u << 24) return;
  const float y = (float)d, r0 = rcp_approx(-y);
  if (fmaf(fmaf(y, r0, 1.f), r0, r0) != -__frcp_rn(y)) atomicAdd(&counts[2], 1ull);
  const int s = __ffs(d) - 1;  // d = 2^s m, m odd; c is an odd multiple of 2^s
  const u64 m = d >> s;
  for (int k = 23; k <= 24; ++k) {
    u64 inv = 1;  // 2^-(k - s) modulo m
    for (int i = s; i < k; ++i) inv = inv * ((m + 1) / 2) % m;
    for (int c = -(16 >> s); c <= 16 >> s; ++c) {
      if (c % 2 == 0) continue;
      const long long h = ((long long)m + c) / 2;  // 2^(k - s) n = h modulo m
      const u64 n0 = (u64)((h % (long long)m + (long long)m) % (long long)m) * inv % m;
      for (u64 n = n0; n < 1u << 24; n += m)
        if (n >= 1u << 23 && (n >= d) == (k == 23)) compare((unsigned)n, d);
    }
  }
}

extern "C" int run(u64* out) {
  check<<<1 << 15, 256>>>();
  if (cudaDeviceSynchronize() != cudaSuccess) return 1;
  return cudaMemcpyFromSymbol(out, counts, sizeof(counts)) != cudaSuccess;
}
"""


def test_quotients_are_correctly_rounded(cuda, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    (tmp_path / "q.cu").write_text(SOURCE)
    lib = tmp_path / "libq.so"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O2", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "-I", str(CSRC), str(tmp_path / "q.cu"), "-o", str(lib)], check=True)
    out = (C.c_ulonglong * 3)()
    assert C.CDLL(str(lib)).run(out) == 0
    compared, differ, reciprocals = out
    assert compared > 50_000_000
    assert reciprocals == 0 and differ == 0, (compared, differ, reciprocals)
