// sin and cos of FP64 arguments by table lookup and a short polynomial, for kernels bound by the FP64
// pipe (a GB300 SM sub-partition issues one FP64 instruction every 64 cycles).
//
// The table-driven scheme of Tang (ACM Trans. Math. Softw. 15 (1989) 144): x = n h + r with h = 2 pi / 1024
// and |r| <= h / 2 = 0.0031; sin and cos of n h come from a table of 1024 pairs, and
//   sin r = r - r^3/6 + r^5/120,  cos r - 1 = -r^2/2 + r^4/24
// leave Taylor remainders below 6e-22 and 2e-18. r is formed with two fused multiply-adds against h in two
// parts: n h_1 is subtracted without rounding error (the difference is a multiple of h_1's last place below
// h), so r is good to its own last place. The result is within 0.7 units in the last place of max(|sin|, |cos|) of what
// the table's values give, which carry the error of sincospi (CUDA states at most two such units for it).
// 16 FP64 operations and one 16-byte table read; sincos() takes about 44 of them.
#pragma once

#include <cuda_runtime.h>

namespace sg {

static constexpr int kScTable = 1024;
static constexpr double kScInv = 162.97466172610083;            // 1024 / (2 pi)
static constexpr double kScH1 = 0.006135923151542565;           // 2 pi / 1024, rounded
static constexpr double kScH2 = 2.391888279584674e-19;          // the rest of it
static constexpr double kScMagic = 6755399441055744.0;          // 1.5 2^52: n in the low mantissa bits
static constexpr unsigned kScMaxHigh = 0x41D00000u;             // high word of 2^30: beyond it sincos() itself

// (sin, cos) of 2 pi j / 1024, once per call: every block of a kernel forming it for itself took as long as three
// particles or nodes, more than the whole sum of a small system
static __global__ void __launch_bounds__(128) sc_table_kernel(double2 *table) {
  const int j = blockIdx.x * 128 + threadIdx.x;
  double s, c;
  sincospi((double)j / (kScTable / 2), &s, &c);
  table[j] = make_double2(s, c);
}
static inline void sc_table(double2 *table, cudaStream_t st) { sc_table_kernel<<<kScTable / 128, 128, 0, st>>>(table); }

// the table into shared memory; the caller synchronises
__device__ __forceinline__ void sc_load(const double2 *from, double2 *table) {
  for (int j = threadIdx.x; j < kScTable; j += blockDim.x) table[j] = __ldg(from + j);
}

__device__ __forceinline__ void sc_sincos(double x, const double2 *table, double *s, double *c) {
  if ((unsigned)(__double2hiint(x) & 0x7FFFFFFF) >= kScMaxHigh) {  // also Inf and NaN; not a comparison in FP64
    sincos(x, s, c);
    return;
  }
  const double t = fma(x, kScInv, kScMagic);
  const double n = t - kScMagic;
  const double2 T = table[__double2loint(t) & (kScTable - 1)];
  double r = fma(n, -kScH1, x);
  r = fma(n, -kScH2, r);
  const double z = r * r;
  const double sr = fma(r * z, fma(z, 1.0 / 120.0, -1.0 / 6.0), r);
  const double cm = z * fma(z, 1.0 / 24.0, -0.5);
  *s = T.x + fma(T.x, cm, T.y * sr);
  *c = T.y + fma(T.y, cm, -T.x * sr);
}

}  // namespace sg
