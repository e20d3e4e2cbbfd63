// Interval-batched FP64 coupling operator on the tensor cores.
//
// The lookup block of a pair depends on its distance only through the interval k and the fraction t,
// W_ij = D(phi)^H (sum_c t^c C_{k,c}) D(phi), D = diag(e^{i m phi}). Sorting the ordered pairs by
// interval turns the operator into one small GEMM per interval, whose matrices C_{k,c} all pairs of
// the interval share:
//
//   y_i += D^H [ (C_0 u + C_2 t^2 u) + t (C_1 u + C_3 t^2 u) ],   u = D x_j,
//
// so the work per pair that is not on the tensor cores falls from O(B^2) to O(B): rotate x_j, form
// t^2 u, and combine and rotate back the two half sums. The per-receiver kernel (sg_coupling.cu)
// interpolates B^2 coefficients in FP64 for every ordered pair, on a pipe that runs two FP64
// multiply-adds per clock and SM.
//
// FP64 accuracy on FP16 tensor cores (error-free slicing, the scheme of Ozaki, Ogita, Oishi and Rump,
// Numer. Algorithms 59 (2012)): every operand is a 60-bit fixed-point number under a power-of-two
// scale (per column of C, then per row of C; per pair and right-hand side for u) cut into six signed
// 10-bit digits, which FP16 holds exactly. A product of two digits is at most 2^18 and at most 64 of
// them are summed (K = 32 or 64), so every FP32 accumulator stays an exact integer of at most 2^24
// whatever the order of the sums. The digit products of equal weight share one accumulator (six of
// them; products below 2^-60 of the scales are dropped), and the epilogue combines the accumulators
// in 64-bit integers. The result is bitwise independent of how the pairs are grouped.
//
// One CTA per SM (216 KB of shared memory) walks a contiguous range of tiles; a tile is up to 64
// complex columns (pairs x right-hand sides) of one interval:
//   * rotate: 512 threads form u and t^2 u in FP64, cut them into digits and store them as the A
//     operand (128 rows: Re and Im of 64 columns; K = 32 per power of t^2);
//   * one thread issues the digit products against the interval's B operand (resident while the
//     interval lasts), N = 32 columns at a time: 8 rows n1 x (Re, Im) x (even, odd powers), into
//     two tensor-memory buffers of six accumulators;
//   * all warps read a buffer back, combine digits, real and imaginary parts (neighbouring lanes) and
//     the powers of t, rotate back and store the pair's contribution V while the next buffer fills.
// A second kernel sums V over the emitters of every receiver in index order (deterministic) and forms
// W x or x - T W x. V is a bounded workspace: larger problems run in chunks of tiles.
//
// Bound: the FP64 pipe, about 11 operations per real output and input of a pair (two at the digits'
// conversion, the rotations, the scaling) against 20 B per output of the per-receiver kernel.
#include <cub/cub.cuh>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <vector>

#include "sg_epilogue.h"
#include "sg_internal.h"
#include "sg_tcgen05.h"

namespace sg {

static constexpr int kIbThreads = 512;
static constexpr int kIbCols = 64;    // complex columns per tile
static constexpr int kIbDig = 6;      // digits per operand
static constexpr int kIbBP = 32;      // padded blocksize
static constexpr int kIbMaxM = 7;     // largest |m| of the phase table
static constexpr int kIbGroupN = 32;  // MMA N: 8 rows n1 x (Re, Im) x (even, odd powers)
static constexpr unsigned long long kIbBias =
    512ull * (1ull + (1ull << 10) + (1ull << 20) + (1ull << 30) + (1ull << 40) + (1ull << 50));

template <int NC>
struct IbShape {
  static constexpr int K = kIbBP * (NC / 2), KC = K / 8;  // K elements, core columns of 16 bytes
  static constexpr int ASLICE = kIbCols * 2 * K * 2;      // bytes of one digit of the A operand
  static constexpr int BSLICE = kIbGroupN * K * 2;        // bytes of one digit of one B group
  static constexpr int BBYTES = 4 * kIbDig * BSLICE;      // one interval's B operand
  static constexpr int PHS = kIbMaxM + 2;                 // phase-table row stride (double2)
  static constexpr size_t META = 2 * kIbCols * (PHS * sizeof(double2) + sizeof(double) + sizeof(long long)) +
                                 kIbCols * sizeof(int) + 2 * 64 * sizeof(int) + kIbBP * sizeof(int) + 128;
  static constexpr size_t SMEM = (size_t)kIbDig * ASLICE + BBYTES + META;
  static_assert(SMEM <= kTcSmemBudget, "shared memory");
};

struct IbArgs {
  const IbRec *rec;       // ordered pairs sorted by interval
  const int *boff;        // [nb + 1] first pair of every non-empty interval
  const int *toff;        // [nb + 1] first tile
  const unsigned char *B; // [nb] B operands
  const int *exps;        // [nb][64]: column exponents eb[32], row exponents ea[32]
  const double2 *x;       // [N][bs][R]
  const int *mofn;
  double2 *V;             // [pair - s0][rt][bs]
  long long s0;           // first pair of this chunk
  int nb, bs, mmax, R, r0, rt, per, t0, t1;  // rt right-hand sides from r0; per = pairs per tile; tiles [t0, t1)
  int *err;
};

// 60-bit digits of |v| 2^(59 - scale) as sum of six 10-bit fields, each offset by 512; `below` = how far the
// exponent of v lies below the scale's
__device__ __forceinline__ unsigned long long ib_fixed(double v, int below) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const unsigned mh = (hi & 0xFFFFFu) | 0x100000u;
  unsigned long long m = ((unsigned long long)__funnelshift_l(lo, mh, 6) << 32) | (lo << 6);
  m = (hi & 0x7FF00000u) == 0u || below > 63 ? 0ull : m >> (below & 63);
  return (int)hi < 0 ? kIbBias - m : kIbBias + m;
}

// the digits of two fixed-point numbers as packed FP16 integers in [-512, 512]
__device__ __forceinline__ void ib_digits(unsigned long long f0, unsigned long long f1, uint32_t (&d)[kIbDig]) {
#pragma unroll
  for (int s = 0; s < kIbDig; ++s) {
    const int sh = 10 * (kIbDig - 1 - s);
    uint32_t a = (uint32_t)(f0 >> sh), b = (uint32_t)(f1 >> sh);
    if (s > 0) {
      a &= 1023u;
      b &= 1023u;
    }
    // FP16 1024 + digit is 0x6400 + digit; the top digit may be 1024, where the sum is still exact (2048)
    const uint32_t p = (a | (b << 16)) + 0x64006400u;
    const __half2 h = __hadd2(*reinterpret_cast<const __half2 *>(&p), __floats2half2_rn(-1536.f, -1536.f));
    d[s] = *reinterpret_cast<const uint32_t *>(&h);
  }
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
               : "r"(taddr));
}

// v as double, exact to rounding: high and low words placed in the mantissas of 2^84 and 2^52
__device__ __forceinline__ double ib_ll2d(long long v) {
  const unsigned lo = (unsigned)v, hi = (unsigned)((unsigned long long)v >> 32) ^ 0x80000000u;
  const double h = __hiloint2double(0x45300000, (int)hi) - (19342813113834066795298816.0 +  // 2^84
                                                            9223372036854775808.0 +         // 2^63
                                                            4503599627370496.0);            // 2^52
  return h + __hiloint2double(0x43300000, (int)lo);
}

// x 2^e for a finite x
__device__ __forceinline__ double ib_scale(double x, int e) {
  const int hi = __double2hiint(x);
  const int ex = (hi >> 20) & 0x7FF;
  if (ex != 0 && ex + e > 0 && ex + e < 0x7FF) return __hiloint2double(hi + (e << 20), __double2loint(x));
  return scalbn(x, e);
}

template <int NC>
__global__ void __launch_bounds__(kIbThreads, 1) ib_kernel(const IbArgs a) {
  using Sh = IbShape<NC>;
  constexpr int KC = Sh::KC, PHS = Sh::PHS, DBUF = kIbDig * kIbGroupN;
  extern __shared__ __align__(1024) unsigned char ib_smem[];
  unsigned char *As = ib_smem, *Bs = ib_smem + (size_t)kIbDig * Sh::ASLICE;
  double2 *ph = reinterpret_cast<double2 *>(Bs + Sh::BBYTES);                  // [2][64][PHS]
  double *tf = reinterpret_cast<double *>(ph + 2 * kIbCols * PHS);             // [2][64]
  long long *xoff = reinterpret_cast<long long *>(tf + 2 * kIbCols);           // [2][64]
  uint64_t *bars = reinterpret_cast<uint64_t *>(xoff + 2 * kIbCols);           // dfull[2], bfull, fin
  int *cexp = reinterpret_cast<int *>(bars + 4);                               // [64] column scale
  int *ex = cexp + kIbCols;                                                    // [2][64]
  int *mofn_s = ex + 2 * 64;                                                   // [32]
  int *tinfo = mofn_s + kIbBP;                                                 // [2][4]: bucket, columns, first pair
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tinfo + 8);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int bs = a.bs;

  const int ntiles = a.t1 - a.t0;
  const int T0 = a.t0 + (int)((long long)ntiles * blockIdx.x / gridDim.x);
  const int T1 = a.t0 + (int)((long long)ntiles * (blockIdx.x + 1) / gridDim.x);

  if (tid < kIbBP) mofn_s[tid] = tid < bs ? a.mofn[tid] : 0;
  if (tid == 0) {
    for (int b = 0; b < 4; ++b)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bars[b])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }

  // the two last warps look one tile ahead: column c = lane of their 64 threads
  const int mc = tid - (kIbThreads - kIbCols);
  int mb = 0;
  if (mc >= 0 && T0 < T1) {  // bucket of the first tile
    int lo = 0, hi = a.nb - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (a.toff[mid] <= T0) lo = mid;
      else hi = mid - 1;
    }
    mb = lo;
  }
  auto look_ahead = [&](int T, int buf) {
    if (mc < 0 || T >= T1) return;
    while (T >= a.toff[mb + 1]) ++mb;
    const int p0 = a.boff[mb] + (T - a.toff[mb]) * a.per, p1 = min(a.boff[mb + 1], p0 + a.per);
    const int ncol = (p1 - p0) * a.rt;
    if (mc == 0) {
      tinfo[buf * 4] = mb;
      tinfo[buf * 4 + 1] = ncol;
      tinfo[buf * 4 + 2] = p0;
    }
    ex[buf * 64 + mc] = a.exps[(size_t)mb * 64 + mc];
    if (mc < ncol) {
      const int p = p0 + mc / a.rt, r = mc % a.rt;
      const IbRec rc = a.rec[p];
      tf[buf * kIbCols + mc] = rc.t;
      xoff[buf * kIbCols + mc] = (long long)rc.j * bs * a.R + a.r0 + r;
      double2 *o = ph + (size_t)(buf * kIbCols + mc) * PHS;
      double pr = 1.0, pi = 0.0;
      o[0] = make_double2(1.0, 0.0);
      for (int m = 1; m <= a.mmax; ++m) {
        const double nr = pr * rc.c - pi * rc.s;
        pi = pr * rc.s + pi * rc.c;
        pr = nr;
        o[m] = make_double2(pr, pi);
      }
    }
  };
  look_ahead(T0, 0);

  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const uint32_t idesc = (1u << 4) | ((uint32_t)(kIbGroupN >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);  // F16 in, F32 out
  const int nq = (bs + 7) / 8;  // groups of 8 rows n1
  const uint32_t a_base = smem_u32(As), b_base = smem_u32(Bs);

  // digit products of row group q into buffer q & 1 (one thread)
  auto issue = [&](int q) {
    const uint32_t d0 = tmem + (uint32_t)((q & 1) * DBUF);
#pragma unroll 1
    for (int d = 0; d < kIbDig; ++d) {
#pragma unroll 1
      for (int i = 0; i <= d; ++i) {
        const uint32_t aa = a_base + (uint32_t)(i * Sh::ASLICE);
        const uint32_t bb = b_base + (uint32_t)((q * kIbDig + d - i) * Sh::BSLICE);
#pragma unroll
        for (int ks = 0; ks < Sh::K / 16; ++ks) {
          const uint32_t acc = (i == 0 && ks == 0) ? 0u : 1u;
          asm volatile(
              "{\n\t.reg .pred p;\n\t"
              "setp.ne.b32 p, %4, 0;\n\t"
              "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d0 + (uint32_t)(d * kIbGroupN)),
              "l"(tc_desc<KC>(aa + ks * 256)), "l"(tc_desc<KC>(bb + ks * 256)), "r"(idesc), "r"(acc)
              : "memory");
        }
      }
    }
    tc_commit(smem_u32(&bars[q & 1]));
  };

  int cur_b = -1, bloads = 0, uses0 = 0, uses1 = 0;
  bool good = true, issued = false;
  for (int T = T0; T < T1 && good; ++T) {
    const int buf = (T - T0) & 1;
    const int b = tinfo[buf * 4], ncol = tinfo[buf * 4 + 1];
    const long long pair0 = (long long)tinfo[buf * 4 + 2] - a.s0;
    if (b != cur_b) {  // every MMA that read the old operand has completed (its accumulators were drained)
      cur_b = b;
      if (tid == 0) {
        const uint32_t bar = smem_u32(&bars[2]);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((uint32_t)Sh::BBYTES)
                     : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(b_base),
            "l"(a.B + (size_t)b * Sh::BBYTES), "r"((uint32_t)Sh::BBYTES), "r"(bar)
            : "memory");
      }
      ++bloads;
    }
    // ---------------------------------------------------------------- rotate and cut into digits
    {
      const int rl = lane & 7, chunk = lane >> 3, row = warp * 8 + rl, col = row >> 1, part = row & 1;
      const int *eb = ex + buf * 64;
      const bool have = col < ncol;
      double v[8];
      int e[8], emax = 0;
      const double2 *xp = a.x + (have ? xoff[buf * kIbCols + col] : 0);
      double2 xv[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int n2 = chunk * 8 + q;
        xv[q] = have && n2 < bs ? __ldg(xp + (size_t)n2 * a.R) : make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int n2 = chunk * 8 + q;
        const int m = mofn_s[n2];
        double2 p = ph[(size_t)(buf * kIbCols + (have ? col : 0)) * PHS + (m < 0 ? -m : m)];
        if (m < 0) p.y = -p.y;
        v[q] = part ? fma(p.x, xv[q].y, p.y * xv[q].x) : fma(p.x, xv[q].x, -p.y * xv[q].y);
        if (!have) v[q] = 0.0;
        const int f = (__double2hiint(v[q]) >> 20) & 0x7FF;
        e[q] = f + eb[n2];
        if (f == 0x7FF) emax = 1 << 20;  // Inf or NaN: the column's result is NaN
        else if (f != 0) emax = max(emax, e[q] + 4096);
      }
      emax = max(emax, __shfl_xor_sync(kTcFull, emax, 1));
      emax = max(emax, __shfl_xor_sync(kTcFull, emax, 8));
      emax = max(emax, __shfl_xor_sync(kTcFull, emax, 16));
      if (part == 0 && chunk == 0) cexp[col] = emax;
      const int es = emax - 4096;  // |u| < 2^(es - 1022)
      const double t = have ? tf[buf * kIbCols + col] : 0.0;
      const double t2 = t * t;
      unsigned char *dst = As + (size_t)(row >> 3) * (KC * 128) + (row & 7) * 16;
#pragma unroll
      for (int h = 0; h < NC / 2; ++h) {
        uint32_t o[kIbDig][4];
#pragma unroll
        for (int q = 0; q < 8; q += 2) {
          unsigned long long f[2];
#pragma unroll
          for (int w = 0; w < 2; ++w) {
            const double val = h == 0 ? v[q + w] : t2 * v[q + w];
            const int fe = (__double2hiint(val) >> 20) & 0x7FF;
            f[w] = ib_fixed(val, es - (fe + (e[q + w] - ((__double2hiint(v[q + w]) >> 20) & 0x7FF))));
          }
          uint32_t dg[kIbDig];
          ib_digits(f[0], f[1], dg);
#pragma unroll
          for (int s = 0; s < kIbDig; ++s) o[s][q >> 1] = dg[s];
        }
#pragma unroll
        for (int s = 0; s < kIbDig; ++s)
          *reinterpret_cast<uint4 *>(dst + (size_t)s * Sh::ASLICE + (h * 4 + chunk) * 128) =
              make_uint4(o[s][0], o[s][1], o[s][2], o[s][3]);
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      good = tc_wait1(smem_u32(&bars[2]), (uint32_t)((bloads - 1) & 1));
      if (good) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        issue(0);
        if (nq > 1) issue(1);
        issued = true;
      }
    }
    good = __shfl_sync(kTcFull, (int)good, 0) != 0;  // one decision per warp
    look_ahead(T + 1, buf ^ 1);
    // ---------------------------------------------------------------- read back, combine, rotate back
    const int sp = warp & 3, grp = warp >> 2;
    const int col = sp * 16 + (lane >> 1), part = lane & 1;
    const bool have = col < ncol;
    const double t = have ? tf[buf * kIbCols + col] : 0.0;
    const int ce = have ? cexp[col] : 0;
    const int cs = ce - 4096 - 1022;
    const double2 *pc = ph + (size_t)(buf * kIbCols + (have ? col : 0)) * PHS;
    double *vo = reinterpret_cast<double *>(a.V + (pair0 * a.rt + (have ? col : 0)) * bs) + part;
    for (int q = 0; q < nq; ++q) {
      bool ok = good;
      if (ok) {
        const int u = (q & 1) ? uses1 : uses0;
        ok = tc_waitw(smem_u32(&bars[q & 1]), (uint32_t)(u & 1));
      }
      if (q & 1) ++uses1;
      else ++uses0;
      const int n1 = q * 8 + grp * 2;
      if (ok && sp * 16 < ncol && n1 < bs) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        float f[kIbDig][8];
        const uint32_t base = tmem + ((uint32_t)(sp * 32) << 16) + (uint32_t)((q & 1) * DBUF + grp * 8);
#pragma unroll
        for (int d = 0; d < kIbDig; ++d) tmem_ld8(base + d * kIbGroupN, f[d]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        long long w[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const long long hi = ((long long)__float2int_rn(f[0][c]) << 20) + ((long long)__float2int_rn(f[1][c]) << 10) +
                               __float2int_rn(f[2][c]);
          const long long lo = ((long long)__float2int_rn(f[3][c]) << 20) + ((long long)__float2int_rn(f[4][c]) << 10) +
                               __float2int_rn(f[5][c]);
          w[c] = (hi << 18) + ((lo + 2048) >> 12);  // in units of 2^-56 of the scales
        }
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          // lane pair (Re u, Im u): Re y = C_re u_re - C_im u_im, Im y = C_re u_im + C_im u_re
          const long long oe = __shfl_xor_sync(kTcFull, w[s * 4 + 1], 1), oo = __shfl_xor_sync(kTcFull, w[s * 4 + 3], 1);
          const double E = ib_ll2d(part ? w[s * 4] + oe : w[s * 4] - oe);
          const double O = ib_ll2d(part ? w[s * 4 + 2] + oo : w[s * 4 + 2] - oo);
          const int n = n1 + s;
          double val = ib_scale(fma(t, O, E), cs + ex[buf * 64 + 32 + (n & 31)] - 56);
          if (ce >= (1 << 20)) val = __longlong_as_double(0x7FF8000000000000ll);
          const double other = __shfl_xor_sync(kTcFull, val, 1);
          const int m = mofn_s[n & 31];
          const double2 p = pc[m < 0 ? -m : m];
          // times e^{-i m phi}
          const double sg = (m < 0) != (part != 0) ? -p.y : p.y;
          const double out = fma(p.x, val, sg * other);
          if (have && n < bs) vo[2 * n] = out;
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      good = __syncthreads_and(ok);
      if (!good) break;
      if (tid == 0 && q + 2 < nq) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        issue(q + 2);
      }
    }
  }
  if (tid == 0) {
    if (!good) atomicExch(a.err, 1);
    if (bloads > 0) tc_wait1(smem_u32(&bars[2]), (uint32_t)((bloads - 1) & 1));
    if (issued) {
      tc_commit(smem_u32(&bars[3]));
      if (!tc_wait1(smem_u32(&bars[3]), 0u)) atomicExch(a.err, 1);
    }
  }
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

// ------------------------------------------------------------------ sum over the emitters
struct IbSum {
  const double2 *V;       // [pair - s0][rt][bs]
  const unsigned *slot;   // [N][N] sorted position of the ordered pair (i, j)
  double2 *acc;           // [N][bs][R] sums over the chunks
  long long s0, s1;       // pairs of this chunk
  int rt, r0, first, last, groups, width;  // width = threads per group
  const int *err;
};

// One block per receiver: `groups` thread groups take contiguous emitter ranges, each thread owns one
// (right-hand side, n1) and adds the emitters in index order; the groups' sums are added in order.
__global__ void __launch_bounds__(512) ib_sum_kernel(const CouplingLaunch L, const IbSum s) {
  extern __shared__ __align__(16) unsigned char ib_sum_smem[];
  double2 *part = reinterpret_cast<double2 *>(ib_sum_smem);  // [groups][bs * rt]
  const int i = blockIdx.x, N = L.n, bs = L.bs, E = bs * s.rt;
  const int g = threadIdx.x / s.width, e = threadIdx.x - g * s.width;
  double2 *red = part + (size_t)s.groups * E;
  if (g < s.groups && e < E) {
    const int j0 = (int)((long long)N * g / s.groups), j1 = (int)((long long)N * (g + 1) / s.groups);
    const unsigned *sl = s.slot + (size_t)i * N;
    double2 a = make_double2(0.0, 0.0);
    int j = j0;
    for (; j + 8 <= j1; j += 8) {
      double2 v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const long long p = (long long)__ldg(sl + j + q);
        v[q] = p >= s.s0 && p < s.s1 ? s.V[(size_t)(p - s.s0) * E + e] : make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        a.x += v[q].x;
        a.y += v[q].y;
      }
    }
    for (; j < j1; ++j) {
      const long long p = (long long)__ldg(sl + j);
      if (p >= s.s0 && p < s.s1) {
        const double2 v = s.V[(size_t)(p - s.s0) * E + e];
        a.x += v.x;
        a.y += v.y;
      }
    }
    part[(size_t)g * E + e] = a;
  }
  __syncthreads();
  for (int q = threadIdx.x; q < E; q += blockDim.x) {
    double2 a = part[q];
    for (int h = 1; h < s.groups; ++h) {
      a.x += part[(size_t)h * E + q].x;
      a.y += part[(size_t)h * E + q].y;
    }
    if (*s.err) a = make_double2(__longlong_as_double(0x7FF8000000000000ll), 0.0);  // a bounded wait ran out
    const int r = q / bs, n1 = q - r * bs;
    double2 *o = s.acc + ((size_t)i * bs + n1) * L.nrhs + s.r0 + r;
    if (!s.first) {
      a.x += o->x;
      a.y += o->y;
    }
    if (s.last) red[n1 * s.rt + r] = a;
    else *o = a;
  }
  if (!s.last) return;
  __syncthreads();
  coupling_epilogue(L, i, s.r0, s.rt, red);
}

// ------------------------------------------------------------------ plan
__device__ __forceinline__ int ib_interval(const double2 *pos, int i, int j, double rho_min, double res, int n_int,
                                           double *t, double *c, double *s) {
  const double dx = pos[i].x - pos[j].x, dy = pos[i].y - pos[j].y;
  const double rho = sqrt(dx * dx + dy * dy);
  const double sidx = (rho - rho_min) / res;
  const double fl = floor(sidx);
  *t = sidx - fl;
  *c = rho > 0.0 ? dx / rho : 1.0;
  *s = rho > 0.0 ? dy / rho : 0.0;
  const int k = (int)fl;
  return k < 0 ? 0 : (k > n_int - 1 ? n_int - 1 : k);
}

__global__ void ib_keys_kernel(const double2 *pos, int n, double rho_min, double res, int n_int, unsigned *keys,
                               unsigned *vals, int *counts) {
  const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= (size_t)n * n) return;
  double t, c, s;
  const int k = ib_interval(pos, (int)(p / n), (int)(p % n), rho_min, res, n_int, &t, &c, &s);
  keys[p] = (unsigned)k;
  vals[p] = (unsigned)p;
  atomicAdd(&counts[k], 1);
}

__global__ void ib_records_kernel(const double2 *pos, int n, double rho_min, double res, int n_int, const unsigned *vals,
                                  IbRec *rec, unsigned *slot) {
  const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= (size_t)n * n) return;
  const unsigned p = vals[q];
  IbRec r;
  r.i = (int)(p / (unsigned)n);
  r.j = (int)(p % (unsigned)n);
  ib_interval(pos, r.i, r.j, rho_min, res, n_int, &r.t, &r.c, &r.s);
  rec[q] = r;
  slot[p] = (unsigned)q;
}

// B operand and exponents of one non-empty interval per block
template <int NC>
__global__ void __launch_bounds__(256) ib_operand_kernel(const double2 *coef, const int *bk, int bs, unsigned char *B,
                                                         int *exps) {
  using Sh = IbShape<NC>;
  __shared__ int eb[kIbBP], ea[kIbBP];
  const int tid = threadIdx.x, b = blockIdx.x, bs2 = bs * bs;
  const double2 *C = coef + (size_t)bk[b] * NC * bs2;
  if (tid < kIbBP) eb[tid] = ea[tid] = -(1 << 20);
  __syncthreads();
  auto field = [](double v) { return (__double2hiint(v) >> 20) & 0x7FF; };
  for (int e = tid; e < NC * bs2; e += blockDim.x) {
    const int f = max(field(C[e].x), field(C[e].y));
    if (f) atomicMax(&eb[(e % bs2) / bs], f - 1022);
  }
  __syncthreads();
  for (int e = tid; e < NC * bs2; e += blockDim.x) {
    const int f = max(field(C[e].x), field(C[e].y)), n2 = (e % bs2) / bs;
    if (f) atomicMax(&ea[e % bs], f - 1022 - eb[n2]);
  }
  __syncthreads();
  if (tid < kIbBP) {
    if (eb[tid] == -(1 << 20)) eb[tid] = 0;
    if (ea[tid] == -(1 << 20)) ea[tid] = 0;
    exps[(size_t)b * 64 + tid] = eb[tid];
    exps[(size_t)b * 64 + 32 + tid] = ea[tid];
  }
  __syncthreads();
  unsigned char *out = B + (size_t)b * Sh::BBYTES;
  // one thread per (n1, part, parity of c, pair of k): k = (c / 2) * 32 + n2
  for (int e = tid; e < 128 * Sh::K / 2; e += blockDim.x) {
    const int row = e / (Sh::K / 2), k = 2 * (e - row * (Sh::K / 2));
    const int n1 = row >> 2, im = row & 1, odd = (row >> 1) & 1;  // row of the operand: n1, then Re/Im, even/odd
    unsigned long long f[2];
    for (int w = 0; w < 2; ++w) {
      const int n2 = (k + w) % kIbBP, c = 2 * ((k + w) / kIbBP) + odd;
      double v = 0.0;
      if (n1 < bs && n2 < bs) {
        const double2 cv = C[(size_t)c * bs2 + n2 * bs + n1];
        v = im ? cv.y : cv.x;
      }
      f[w] = ib_fixed(v, n1 < bs && n2 < bs ? ea[n1] + eb[n2] + 1022 - field(v) : 0);
    }
    uint32_t dg[kIbDig];
    ib_digits(f[0], f[1], dg);
    const int q = n1 >> 3, rq = row & 31;
    for (int s = 0; s < kIbDig; ++s)
      *reinterpret_cast<uint32_t *>(out + (size_t)(q * kIbDig + s) * Sh::BSLICE +
                                    ((size_t)(rq >> 3) * Sh::KC + (k >> 3)) * 128 + (rq & 7) * 16 + (k & 7) * 2) = dg[s];
  }
}

static constexpr int kIbMinParticles = 32;
static constexpr long long kIbMaxPairs = 1ll << 27;      // 4 GB of pair records
static constexpr size_t kIbWorkspace = (size_t)1 << 30;  // bytes of V per chunk

bool ib_supported(const sg_context *c) {
  if (c->vol || c->kind < 0 || c->bs > kIbBP) return false;
  if ((long long)c->n * c->n > kIbMaxPairs || c->n < kIbMinParticles) return false;
  for (int m : c->h_mofn)
    if (m > kIbMaxM || m < -kIbMaxM) return false;
  return true;
}

static void ib_build_plan(sg_context *c, cudaStream_t st) {
  auto &P = c->ib;
  const int n = c->n, n_int = c->n_int;
  const size_t np = (size_t)n * n;
  DevBuf<unsigned> keys, keys2, vals, vals2;
  DevBuf<int> counts;
  DevBuf<unsigned char> tmp;
  keys.reserve(np);
  keys2.reserve(np);
  vals.reserve(np);
  vals2.reserve(np);
  counts.reserve(n_int);
  SG_CUDA(cudaMemsetAsync(counts.ptr, 0, n_int * sizeof(int), st));
  const unsigned grid = (unsigned)((np + 255) / 256);
  ib_keys_kernel<<<grid, 256, 0, st>>>(c->pos.ptr, n, c->rho_min, c->res, n_int, keys.ptr, vals.ptr, counts.ptr);
  SG_CUDA(cudaGetLastError());
  int bits = 1;
  while ((1 << bits) < n_int) ++bits;
  size_t bytes = 0;
  SG_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, bytes, keys.ptr, keys2.ptr, vals.ptr, vals2.ptr, np, 0, bits, st));
  tmp.reserve(bytes);
  SG_CUDA(cub::DeviceRadixSort::SortPairs(tmp.ptr, bytes, keys.ptr, keys2.ptr, vals.ptr, vals2.ptr, np, 0, bits, st));
  P.rec.reserve(np);
  P.slot.reserve(np);
  ib_records_kernel<<<grid, 256, 0, st>>>(c->pos.ptr, n, c->rho_min, c->res, n_int, vals2.ptr, P.rec.ptr, P.slot.ptr);
  SG_CUDA(cudaGetLastError());
  std::vector<int> cnt(n_int);
  SG_CUDA(cudaMemcpyAsync(cnt.data(), counts.ptr, n_int * sizeof(int), cudaMemcpyDeviceToHost, st));
  SG_CUDA(cudaStreamSynchronize(st));
  std::vector<int> bk;
  P.h_boff.assign(1, 0);
  for (int k = 0; k < n_int; ++k)
    if (cnt[k] > 0) {
      bk.push_back(k);
      P.h_boff.push_back(P.h_boff.back() + cnt[k]);
    }
  P.nb = (int)bk.size();
  DevBuf<int> dbk;
  dbk.reserve(P.nb);
  P.boff.reserve(P.nb + 1);
  P.exps.reserve((size_t)P.nb * 64);
  P.B.reserve((size_t)P.nb * (c->ncoef == 2 ? IbShape<2>::BBYTES : IbShape<4>::BBYTES));
  SG_CUDA(cudaMemcpyAsync(dbk.ptr, bk.data(), P.nb * sizeof(int), cudaMemcpyHostToDevice, st));
  SG_CUDA(cudaMemcpyAsync(P.boff.ptr, P.h_boff.data(), (P.nb + 1) * sizeof(int), cudaMemcpyHostToDevice, st));
  if (c->ncoef == 2) ib_operand_kernel<2><<<P.nb, 256, 0, st>>>(c->coef64.ptr, dbk.ptr, c->bs, P.B.ptr, P.exps.ptr);
  else ib_operand_kernel<4><<<P.nb, 256, 0, st>>>(c->coef64.ptr, dbk.ptr, c->bs, P.B.ptr, P.exps.ptr);
  SG_CUDA(cudaGetLastError());
  P.err.reserve(1);
  SG_CUDA(cudaMemsetAsync(P.err.ptr, 0, sizeof(int), st));
  SG_CUDA(cudaStreamSynchronize(st));  // the temporaries are released on return
  P.tiles.clear();
  c->launches += 3;
  P.ready = true;
}

// tiles of `per` pairs: first tile of every interval
static sg_context::IbTiles &ib_tiles(sg_context *c, int per, cudaStream_t st) {
  auto &P = c->ib;
  for (auto &t : P.tiles)
    if (t->per == per) return *t;
  auto t = std::make_unique<sg_context::IbTiles>();
  t->per = per;
  t->h_toff.assign(1, 0);
  for (int b = 0; b < P.nb; ++b)
    t->h_toff.push_back(t->h_toff.back() + (P.h_boff[b + 1] - P.h_boff[b] + per - 1) / per);
  t->toff.reserve(t->h_toff.size());
  SG_CUDA(cudaMemcpyAsync(t->toff.ptr, t->h_toff.data(), t->h_toff.size() * sizeof(int), cudaMemcpyHostToDevice, st));
  SG_CUDA(cudaStreamSynchronize(st));
  P.tiles.push_back(std::move(t));
  return *P.tiles.back();
}

template <int NC>
static void ib_launch(const IbArgs &a, cudaStream_t st) {
  static bool attr_done[64] = {};
  if (first_on_device(attr_done))
    SG_CUDA(cudaFuncSetAttribute(ib_kernel<NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)IbShape<NC>::SMEM));
  ib_kernel<NC><<<std::min(sm_count(), a.t1 - a.t0), kIbThreads, IbShape<NC>::SMEM, st>>>(a);
  SG_CUDA(cudaGetLastError());
}

// y = M x or W x in FP64; returns the number of kernels launched
int launch_ibatch(sg_context *c, const double2 *x, double2 *y, int R, bool master, cudaStream_t st) {
  auto &P = c->ib;
  if (!P.ready) ib_build_plan(c, st);
  // the workspace is shared by all calls on this context: order them across streams
  if (!P.done) SG_CUDA(cudaEventCreateWithFlags(&P.done, cudaEventDisableTiming));
  else SG_CUDA(cudaStreamWaitEvent(st, P.done, 0));
  const int bs = c->bs;
  CouplingLaunch L{};
  L.n = c->n;
  L.bs = bs;
  L.x = x;
  L.y = y;
  L.nrhs = R;
  L.master = master ? 1 : 0;
  L.t = c->tmat.ptr;
  L.ptype = c->ptype.ptr;
  L.t_diag = c->t_diag;
  int mmax = 0, launched = 0;
  for (int m : c->h_mofn) mmax = std::max(mmax, std::abs(m));
  for (int r0 = 0; r0 < R; r0 += 16) {
    const int rt = std::min(16, R - r0), per = kIbCols / rt;
    auto &tl = ib_tiles(c, per, st);
    const size_t pair_bytes = (size_t)rt * bs * sizeof(double2);
    const int ntiles = tl.h_toff.back();
    const int chunk = (int)std::min<size_t>(ntiles, std::max<size_t>(1, kIbWorkspace / (pair_bytes * per)));
    P.V.reserve((size_t)std::min<long long>((long long)chunk * per, (long long)c->n * c->n) * rt * bs);
    if (chunk < ntiles) P.acc.reserve((size_t)c->n * bs * R);
    auto first_pair = [&](int t) -> long long {  // first pair of tile t
      const int b = (int)(std::upper_bound(tl.h_toff.begin(), tl.h_toff.end(), t) - tl.h_toff.begin()) - 1;
      if (b >= P.nb) return (long long)c->n * c->n;
      return P.h_boff[b] + (long long)(t - tl.h_toff[b]) * per;
    };
    IbArgs a{};
    a.rec = P.rec.ptr;
    a.boff = P.boff.ptr;
    a.toff = tl.toff.ptr;
    a.B = P.B.ptr;
    a.exps = P.exps.ptr;
    a.x = x;
    a.mofn = c->mofn.ptr;
    a.V = P.V.ptr;
    a.nb = P.nb;
    a.bs = bs;
    a.mmax = mmax;
    a.R = R;
    a.r0 = r0;
    a.rt = rt;
    a.per = per;
    a.err = P.err.ptr;
    IbSum s{};
    s.V = P.V.ptr;
    s.slot = P.slot.ptr;
    s.acc = P.acc.ptr;
    s.err = P.err.ptr;
    s.rt = rt;
    s.r0 = r0;
    s.width = (bs * rt + 31) / 32 * 32;
    s.groups = std::max(1, 512 / s.width);
    const size_t smem = (size_t)(s.groups + 1) * bs * rt * sizeof(double2);
    for (int t0 = 0; t0 < ntiles; t0 += chunk) {
      a.t0 = t0;
      a.t1 = std::min(ntiles, t0 + chunk);
      a.s0 = s.s0 = first_pair(t0);
      s.s1 = first_pair(a.t1);
      s.first = t0 == 0;
      s.last = a.t1 == ntiles;
      if (c->ncoef == 2) ib_launch<2>(a, st);
      else ib_launch<4>(a, st);
      ib_sum_kernel<<<c->n, 512, smem, st>>>(L, s);
      SG_CUDA(cudaGetLastError());
      launched += 2;
    }
  }
  SG_CUDA(cudaEventRecord(P.done, st));
  return launched;
}

bool ib_check_error(sg_context *c, cudaStream_t st) {
  if (!c->ib.ready) return false;
  int e = 0;
  SG_CUDA(cudaMemcpyAsync(&e, c->ib.err.ptr, sizeof(int), cudaMemcpyDeviceToHost, st));
  SG_CUDA(cudaStreamSynchronize(st));
  if (e) SG_CUDA(cudaMemsetAsync(c->ib.err.ptr, 0, sizeof(int), st));
  return e != 0;
}

}  // namespace sg
