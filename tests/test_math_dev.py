"""The branch-free functions of csrc/cbc_math_dev.cuh: reciprocal and quotient
correctly rounded, sincos and pow_pos bit for bit those of cbc_math.h.

On the host the steps after the hardware's seed are driven with every sign and
size of the seed's error; on the GPU the functions are compared with 1.0 / x,
a / b and cbc_math.h: random arguments, both ends of every stated range, the
significands next to the reciprocal's exception, quotients next to a rounding
boundary.  No tolerance: every result has to have the same bits."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "coupled-bubble-control_b200", "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

pytestmark = pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")

COMMON = r"""
#include <stdio.h>
#include "cbc_math_dev.cuh"
typedef unsigned long long u64;
__host__ __device__ inline u64 mix(u64 z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
// 1.f 2^e with significand bits f
__host__ __device__ inline double make(u64 f, int e) {
  return cbcm::bits_to_double(((u64)(e + 1023) << 52) | (f & 0xfffffffffffffull));
}
// random significand, often close to 1 or to 2
__host__ __device__ inline u64 frac(u64 u) {
  const u64 m = u & 0xfffffffffffffull;
  const int s = 20 + (int)((u >> 54) & 31);
  return u >> 62 == 0 ? 0xfffffffffffffull - (m >> s) : u >> 62 == 1 ? m >> s : m;
}
"""

HOST = COMMON + r"""
int main() {
  // seeds with relative error up to 2^-19, both signs, among them the ones next
  // to 1/x itself
  long bad = 0, n = 0;
  for (int i = 0; i < 400000; ++i) {
    u64 f = frac(mix(3 * i));
    if (i < 4000) f = 0xfffffffffffffull - (u64)(i % 8);
    const double x = make(f, (int)(mix(3 * i + 1) % 2000) - 1000), r = 1.0 / x;
    for (int k = 0; k < 12; ++k) {
      const double rel = ldexp((k & 1) ? -1.0 : 1.0, -19 - 3 * k);
      double xa[1] = {x}, y[1] = {fma(r, k < 11 ? rel : 0.0, r)};
      cbcd::rcp_refine(xa, y);
      bad += y[0] != r;
      ++n;
    }
  }
  printf("%ld of %ld\n", bad, n);
  return bad != 0;
}
"""

GPU = COMMON + r"""
__device__ u64 bad[8];
__device__ double worst_seed;
__device__ bool same(double a, double b) { return cbcm::double_to_bits(a) == cbcm::double_to_bits(b); }
__device__ void check_rcp(double x) {
  double a[3] = {x, -x, 1.0}, y[3];
  cbcd::rcp(a, y);
  if (!same(y[0], 1.0 / x) || !same(y[1], 1.0 / -x) || y[2] != 1.0) atomicAdd(bad + 0, 1ull);
}
__device__ void check_quot(double a, double b) {
  double n[2] = {a, -a}, d[2] = {b, b}, q[2];
  cbcd::quot(n, d, q);
  if (!same(q[0], a / b) || !same(q[1], -a / b)) atomicAdd(bad + 1, 1ull);
}
__device__ void check_sincos(double x, double z) {
  double a[2] = {x, z}, s[2], c[2], s0, c0;
  cbcd::sincos(a, s, c);
  for (int i = 0; i < 2; ++i) {
    cbcm::sincos(a[i], &s0, &c0);
    if (!same(s[i], s0) || !same(c[i], c0)) atomicAdd(bad + 2, 1ull);
  }
}
__device__ void check_pow(double x, double p) {
  double a[1] = {x}, e[1] = {p}, y[1];
  cbcd::pow_pos(a, e, y);
  if (!same(y[0], cbcm::pow_pos(x, p))) atomicAdd(bad + 3, 1ull);
}
// every high word of the significand: the seed depends on no more
__global__ void seeds() {
  const u64 id = blockIdx.x * (u64)blockDim.x + threadIdx.x;
  if (id >= 1u << 20) return;
  for (int k = 0; k < 2; ++k) {
    const double x = make(id << 32 | (k ? 0xffffffffull : 0ull), 0);
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fabs(fma(-x, y, 1.0));
    atomicMax((u64*)&worst_seed, (u64)__double_as_longlong(e));
  }
}
__global__ void random_args(int n) {
  for (int i = 0; i < n; ++i) {
    const u64 u = mix(((u64)i * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x), v = mix(u), w = mix(v), z = mix(w);
    check_rcp(make(frac(u), (int)(v % 2001) - 1000 - (v % 2001 == 2000)));
    // controller ratios: 2^-400 <= a < 2^400, 2^-60 <= b < 2^400
    const double b = make(frac(w), (int)((v >> 20) % 460) - 60);
    check_quot(make(frac(z), (int)((v >> 40) % 800) - 400), b);
    // next to a rounding boundary: a = b (q + half a unit of q), rounded
    const double q = make(frac(u), (int)((v >> 30) % 200) - 100), b1 = make(frac(w), (int)((v >> 20) % 100) - 50);
    check_quot(fma(b1, q, b1 * make(0, (int)((v >> 30) % 200) - 100 - 53)), b1);
    // the quotient of a logarithm
    const double m = make(u, u >> 63 ? -1 : 0);
    if (m > 0.7 && m < 1.4143) check_quot(m - 1.0, m + 1.0);
    const double x = make(u, (int)(v % 110) - 60), x1 = (double)(long long)(w % 4000000) * 1.5707963267948966;
    check_sincos(u >> 63 ? -x : x, z >> 63 ? -x1 : x1);
    check_pow(make(frac(u), (int)(v % 128) - 64), (double)(w >> 11) * 0x1p-53 * 15.0);
    check_pow(make(frac(u), (int)(v % 800) - 400), w & 1 ? 0.2 : 0.25);
  }
}
__global__ void edges() {
  const int e = (int)blockIdx.x - 1000, k = threadIdx.x;     // 2000 exponents, 128 significands
  const u64 f = k < 64 ? k : 0xfffffffffffffull - (u64)(k - 64);
  check_rcp(make(f, e));
  if (e >= -400 && e < 400)
    for (int j = 0; j < 128; ++j) {
      const u64 g = j < 64 ? j : 0xfffffffffffffull - (u64)(j - 64);
      for (int be = -60; be < 400; be += 51) check_quot(make(f, e), make(g, be));
    }
  if (e >= -64 && e < 64) {
    check_pow(make(f, e), 15.0);
    check_pow(make(f, e), 0.0);
    check_pow(make(f, e), -15.0);
    check_pow(make(0x6a09e667f3bcdull - 64 + k, e), 4.2);    // around sqrt(2) 2^e
  }
  if (e >= -400 && e < 400) check_pow(make(f, e), 0.25);
  if (e < 50) check_sincos(make(f, e), -make(f, e));
  check_sincos(0.0, -0.0);
}
int main() {
  seeds<<<4096, 256>>>();
  random_args<<<592, 256>>>(100);
  edges<<<2000, 128>>>();
  u64 b[8];
  double w;
  if (cudaMemcpyFromSymbol(b, bad, sizeof b) != cudaSuccess || cudaMemcpyFromSymbol(&w, worst_seed, 8) != cudaSuccess) {
    printf("CUDA: %s\n", cudaGetErrorString(cudaGetLastError()));
    return 2;
  }
  printf("rcp %llu quot %llu sincos %llu pow %llu seed 2^%.3f\n", b[0], b[1], b[2], b[3], log2(w));
  // the refinement needs the cube of the seed's error far below half a unit
  return (b[0] | b[1] | b[2] | b[3]) != 0 || !(w < 0x1p-19);
}
"""


def build_and_run(tmp_path, source, *flags):
    src, exe = tmp_path / "m.cu", tmp_path / "m"
    src.write_text(source)
    subprocess.run([NVCC, "-std=c++17", "-O2", "-fmad=false", "-I", CSRC, *flags, str(src), "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)


def test_reciprocal_for_every_error_of_the_seed(tmp_path):
    r = build_and_run(tmp_path, HOST, "-gencode", "arch=compute_100a,code=sm_100a")
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
def test_device_functions(cuda, tmp_path):
    r = build_and_run(tmp_path, GPU, "-gencode", "arch=compute_100a,code=sm_100a")
    print(r.stdout)
    assert r.returncode == 0, r.stdout + r.stderr
