// Interval-batched FP64 coupling operator on the tensor cores.
//
// The lookup block of a pair depends on its distance only through the interval k and the fraction t,
// W_ij = D(phi)^H (sum_c t^c C_{k,c}) D(phi), D = diag(e^{i m phi}). Sorting the ordered pairs by
// interval turns the operator into one small GEMM per interval, whose matrices C_{k,c} all pairs of
// the interval share:
//
//   y_i += D^H [ ((C_3 u t + C_2 u) t + C_1 u) t + C_0 u ],   u = D x_j,
//
// so the work per pair that is not on the tensor cores falls from O(B^2) to O(B): rotate x_j, combine
// the powers of t and rotate back. The per-receiver kernel (sg_coupling.cu) interpolates B^2
// coefficients in FP64 for every ordered pair, on a pipe that runs two FP64 multiply-adds per clock
// and SM.
//
// FP64 accuracy on FP16 tensor cores (error-free slicing, the scheme of Ozaki, Ogita, Oishi and Rump,
// Numer. Algorithms 59 (2012)): every operand is a 63-bit fixed-point number under a power-of-two
// scale (per column of C, then per row of C; per pair and right-hand side for u) cut into seven signed
// 9-bit digits, which FP16 holds exactly. The digit products of equal weight 2^(-9 d), d = 0..6, share
// one FP32 accumulator; smaller products (below 2^-60 of the scales) are dropped. A digit product is at
// most 2^16 and K = 32 of them (at most 30 nonzero for blocksize <= 30) times d + 1 <= 7 pairs of digits
// are summed, at most 7 * 30 * 2^16 = 13,762,560 < 2^24: every accumulator stays an exact integer
// whatever the order of the sums. Blocksizes 31 to 48 (K = 48) take 8-bit digits of 56-bit numbers and the
// weights d = 0..7, at most 7 * 48 * 2^14 = 5,505,024 per accumulator. (Ten-bit digits would need fewer products, but the sums of the
// middle weights could pass 2^24.) The digits are combined in 64-bit integers, in which the powers of
// t and the rotations follow; the result is independent of how the pairs are grouped.
//
// One CTA per SM walks a contiguous range of tiles; a tile is up to 64 complex columns (pairs x
// right-hand sides) of one interval:
//   * the warps rotate x_j, cut u into digits and store them as the A operand (128 rows: Re and Im of 64
//     columns, K = 32);
//   * one thread issues the digit products against the interval's B operand (resident while the
//     interval lasts; with K = 48 one pass at a time, copied while the last pass is combined): passes of
//     128 rows (n1, power of t, Re / Im), one job per weight d = 0..6 in a ring of four tensor-memory
//     accumulators of 128 columns;
//   * the warps read the jobs back (32 columns per warp), combine digits, real and imaginary parts
//     (neighbouring lanes) and powers of t, rotate back and store the pair's contribution V.
// A second kernel sums V over the emitters of every receiver in index order (deterministic) and forms
// W x or x - T W x. V is a bounded workspace: larger problems run in chunks of tiles.
//
// Integer arithmetic instead of FP64 for everything but the last conversion: a GB300 SM sub-partition
// issues an FP64 instruction every 64 cycles, a 32-bit integer one every two.
#include <cub/cub.cuh>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "sg_epilogue.h"
#include "sg_internal.h"
#include "sg_tcgen05.h"

namespace sg {

static constexpr int kIbWarps = 16;
static constexpr int kIbThreads = 32 * kIbWarps;
static constexpr int kIbCols = 64;   // complex columns per tile
static constexpr int kIbDig = 7;     // digits per operand
static constexpr int kIbN = 128;     // B operand rows per pass: n1 x powers of t x (Re, Im)
// 1.5 2^23: added to an integer below 2^22 it leaves that in the mantissa
static constexpr float kIbMagic = 12582912.f;
static constexpr unsigned long long kIbMagicBits = 0x4B400000ull;
// largest t in units of 2^-62 whose high word fits (t < 1 up to its last places)
static constexpr long long kIbBelowOne = (1ll << 62) - (1ll << 30) - 1;

// KP: padded blocksize, 32 or 48
template <int KP>
struct IbNumbers {
  static constexpr int BITS = KP == 32 ? 9 : 8;        // bits per digit
  static constexpr int MAXB = KP == 32 ? 30 : 48;      // largest blocksize
  static constexpr int MAXM = KP == 32 ? 3 : 4;        // largest |m| of the phase table
  static constexpr int UP = KP == 32 ? 9 : 2;          // operands are 53 + UP bits below their scale
  static constexpr int UNIT = KP == 32 ? 55 : 54;      // combinations are in units of 2^-UNIT of the scales
  static constexpr int JOBS = KP == 32 ? 7 : 8;        // weights kept: what is dropped is below 2^-60 of the scales
  static constexpr unsigned long long bias() {
    unsigned long long b = 0;
    for (int i = 0; i < kIbDig; ++i) b |= 1ull << (BITS * i + BITS - 1);
    return b;
  }
  static constexpr unsigned long long BIAS = bias();
  // what the bits of 1.5 2^23 add to a combination of digits: the weights that take them
  static constexpr unsigned long long OFFSET =
      kIbMagicBits * (KP == 32 ? (1ull << 39) + (1ull << 30) + 1 + 1
                               : (1ull << 40) + (1ull << 32) + (1ull << 24) + (1ull << 16) + (1ull << 8) + 1 + 1);
  static_assert(kIbDig * MAXB * (1 << (2 * BITS - 2)) <= (1 << 24), "exact FP32 accumulators");
  static_assert((KP == 32 ? 2 : 5) * MAXB * (1 << (2 * BITS - 2)) < (1 << 22), "weights that become integers by addition");
};

template <int NC, int KP>
struct IbShape {
  static constexpr int KC = KP / 8;               // core columns of 16 bytes
  static constexpr int SLICE = 128 * KP * 2;      // bytes of one digit of an operand
  static constexpr int OPERAND = kIbDig * SLICE;  // bytes of an A operand or one pass of B
  static constexpr int RN = 2 * NC;               // B rows per n1
  static constexpr int PN = kIbN / RN;            // n1 per pass
  static constexpr int PASSES = (KP + PN - 1) / PN;  // at most
  static constexpr int BBYTES = PASSES * OPERAND;
  static constexpr bool STREAM = KP > 32;         // B in shared memory: one pass, or all
  static constexpr int BSMEM = STREAM ? OPERAND : BBYTES;
};

// per-tile data, four tiles deep: written two tiles ahead, read until the tile is stored
template <int KP>
struct IbTile {
  int4 ph[kIbCols][IbNumbers<KP>::MAXM + 1];  // cos, sin of m phi in words of 2^-61
  int2 t[kIbCols];                // t in words of 2^-62
  long long xoff[kIbCols];        // x_j of the column
  int eb[KP], ea[KP];             // column and row exponents of the interval
  int cexp[kIbCols];              // scale of x_j (written with the A operand)
  int ncol, bucket;
  long long pair0;                // first pair, from the start of V
};

static constexpr int kIbXPitch = 31;  // x_j of a column: element n2 at (n2 mod 8) 4 + n2 / 8

template <int KP>
struct IbSmem {
  IbTile<KP> tile[4];
  IbRec rec[2][kIbCols];              // records, exponents and (columns, bucket, first pair) of the next tiles
  int exps[2][2 * KP];
  int next[2][3];
  double2 x[KP == 32 ? kIbCols * kIbXPitch : 1];  // x_j of the next tile's columns (K = 48 leaves no room for it)
  uint64_t dfull[4], dempty[4], afull, meta[4], bfull, done;
  int mofn[KP];
  uint32_t tmem;
  int lb[2];  // bucket of the two look-ahead warps
};
template <int NC, int KP>
constexpr size_t ib_smem() {
  return (size_t)IbShape<NC, KP>::OPERAND + IbShape<NC, KP>::BSMEM + (sizeof(IbSmem<KP>) + 127) / 128 * 128;
}
static_assert(ib_smem<4, 32>() <= kTcSmemBudget && ib_smem<4, 48>() <= kTcSmemBudget, "shared memory");

struct IbArgs {
  const IbRec *rec;       // ordered pairs sorted by interval
  const int *boff;        // [nb + 1] first pair of every non-empty interval
  const int *toff;        // [nb + 1] first tile
  const unsigned char *B; // [nb] B operands
  const int *exps;        // [nb][2 KP]: column exponents eb[KP], row exponents ea[KP]
  const double *x;        // [N][bs][R] complex
  const int *mofn;
  double *V;              // [pair - s0][rt][bs] complex
  long long s0;           // first pair of this chunk
  int nb, bs, mmax, R, r0, rt, per, t0, t1;  // rt right-hand sides from r0; per = pairs per tile; tiles [t0, t1)
  int *err;
};

__device__ __forceinline__ int ib_field(double v) { return (__double2hiint(v) >> 20) & 0x7FF; }

// v 2^(53 + UP - scale) truncated, for an exponent of v that lies `below` under the scale's
template <int UP>
__device__ __forceinline__ long long ib_fixed(double v, int below) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const unsigned mh = (hi & 0xFFFFFu) | 0x100000u;
  unsigned long long m = ((unsigned long long)__funnelshift_l(lo, mh, UP) << 32) | (lo << UP);
  m = (hi & 0x7FF00000u) == 0u || below > 63 ? 0ull : m >> (below & 63);
  return (int)hi < 0 ? -(long long)m : (long long)m;
}

// the digits of two fixed-point numbers as packed FP16 integers in [-2^(BITS - 1), 2^(BITS - 1)]
template <int KP>
__device__ __forceinline__ void ib_digits(long long v0, long long v1, uint32_t (&d)[kIbDig]) {
  constexpr int BITS = IbNumbers<KP>::BITS;
  const unsigned long long f0 = (unsigned long long)v0 + IbNumbers<KP>::BIAS, f1 = (unsigned long long)v1 + IbNumbers<KP>::BIAS;
#pragma unroll
  for (int s = 0; s < kIbDig; ++s) {
    const int sh = BITS * (kIbDig - 1 - s);
    const uint32_t mask = s > 0 ? (1u << BITS) - 1 : (2u << BITS) - 1;  // the top digit may be 2^BITS
    const uint32_t a = (uint32_t)(f0 >> sh);
    const uint32_t b = sh >= 16 ? (uint32_t)(f1 >> (sh - 16)) : (uint32_t)f1 << (16 - sh);
    const uint32_t p = (a & mask) | (b & (mask << 16)) | 0x64006400u;  // FP16 1024 + digit + 2^(BITS - 1)
    const float off = -1024.f - (1 << (BITS - 1));
    const __half2 h = __hadd2(*reinterpret_cast<const __half2 *>(&p), __floats2half2_rn(off, off));
    d[s] = *reinterpret_cast<const uint32_t *>(&h);
  }
}

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// Products of 62-bit fixed-point numbers from 31-bit words: three 32 x 32 -> 64 bit multiply-adds, low
// word by low word (below the last place kept) is dropped. The factors that stay the same for a pair
// (t, the phases) carry a signed low word in [-2^30, 2^30), so that what is dropped has no bias that
// would add up over the pairs.
struct IbWords {
  int h, l;
};
__device__ __forceinline__ IbWords ib_split(long long v) {
  return {(int)(v >> 31), (int)((unsigned)v & 0x7FFFFFFFu)};
}
__device__ __forceinline__ IbWords ib_split_signed(long long v) {
  return {(int)((v + 0x40000000ll) >> 31), (int)((unsigned)v << 1) >> 1};
}
__device__ __forceinline__ long long ib_mad(int a, int b, long long c) { return (long long)a * b + c; }
// a b / 2^62 + c
__device__ __forceinline__ long long ib_mul(IbWords a, int bh, int bl, long long c) {
  const long long mid = ib_mad(a.h, bl, ib_mad(a.l, bh, 0x40000000ll));
  return ib_mad(a.h, bh, c + (mid >> 31));
}

// v 2^e rounded to double: the words placed in the mantissas of 2^84 and 2^52, two FP64 additions
__device__ __forceinline__ double ib_to_double(long long v, int e) {
  const unsigned lo = (unsigned)v, hi = (unsigned)((unsigned long long)v >> 32) ^ 0x80000000u;
  const double h = __hiloint2double(0x45300000, (int)hi) - (19342813113834066795298816.0 +  // 2^84
                                                            9223372036854775808.0 +         // 2^63
                                                            4503599627370496.0);            // 2^52
  const double d = h + __hiloint2double(0x43300000, (int)lo);
  const int f = ib_field(d);
  if (f != 0 && f + e > 0 && f + e < 0x7FF) return __hiloint2double(__double2hiint(d) + (e << 20), __double2loint(d));
  return scalbn(d, e);  // zero, or outside the normal range
}

// One product of a digit of A and a digit of B (K = 16) into dst; the descriptors differ from those of the
// operands' first bytes by a constant in their low word.
template <bool ACC>
__device__ __forceinline__ void ib_mma(uint32_t dst, uint32_t a, uint32_t b, uint32_t hi, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %3};\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}" ::"r"(dst),
      "r"(a), "r"(b), "r"(hi), "r"(idesc), "n"(ACC ? 1 : 0)
      : "memory");
}

// all digit products of weight D; unrolled, because one thread issues them and every instruction between two
// MMAs costs it several cycles
template <int D, int KP>
__device__ __forceinline__ void ib_issue(uint32_t dst, uint32_t a, uint32_t b, uint32_t hi, uint32_t idesc) {
#pragma unroll
  for (int i = D < kIbDig ? 0 : D - kIbDig + 1; i <= (D < kIbDig ? D : kIbDig - 1); ++i)
#pragma unroll
    for (int ks = 0; ks < KP / 16; ++ks) {
      constexpr int SLICE = 128 * KP * 2;
      const uint32_t ao = a + (uint32_t)((i * SLICE + ks * 256) >> 4), bo = b + (uint32_t)(((D - i) * SLICE + ks * 256) >> 4);
      if (i == (D < kIbDig ? 0 : D - kIbDig + 1) && ks == 0) ib_mma<false>(dst, ao, bo, hi, idesc);
      else ib_mma<true>(dst, ao, bo, hi, idesc);
    }
}

template <int NC, int KP>
__global__ void __launch_bounds__(kIbThreads, 1) ib_kernel(const IbArgs a) {
  using Sh = IbShape<NC, KP>;
  using Num = IbNumbers<KP>;
  constexpr int RN = Sh::RN, PN = Sh::PN, WN = PN / 4;  // WN rows n1 per warp and pass
  extern __shared__ __align__(1024) unsigned char ib_raw[];
  unsigned char *As = ib_raw, *Bs = ib_raw + Sh::OPERAND;
  IbSmem<KP> &S = *reinterpret_cast<IbSmem<KP> *>(Bs + Sh::BSMEM);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int bs = a.bs;
  const int ntiles = a.t1 - a.t0;
  const int T0 = a.t0 + (int)((long long)ntiles * blockIdx.x / gridDim.x);
  const int NT = a.t0 + (int)((long long)ntiles * (blockIdx.x + 1) / gridDim.x) - T0;  // this CTA's tiles
  const int passes = (bs + PN - 1) / PN;

  if (tid < KP) S.mofn[tid] = tid < bs ? a.mofn[tid] : 0;
  if (tid == 0) {
    auto init = [](uint64_t *b, int n) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(n) : "memory");
    };
    for (int b = 0; b < 4; ++b) {
      init(&S.dfull[b], 1);
      init(&S.dempty[b], kIbWarps);
      init(&S.meta[b], 2);
    }
    init(&S.afull, kIbWarps);
    init(&S.bfull, 1);
    init(&S.done, kIbWarps);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tmem)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = S.tmem;
  bool good = true;

  // ------------------------------------------------------------------ look ahead (two warps, 32 columns each)
  const int look_half = warp == 5 ? 0 : (warp == 10 ? 1 : -1);
  if (look_half >= 0) {  // bucket of the first tile
    int lb = 0, hi = a.nb - 1;
    while (lb < hi) {
      const int mid = (lb + hi + 1) >> 1;
      if (a.toff[mid] <= T0) lb = mid;
      else hi = mid - 1;
    }
    S.lb[look_half] = lb;
    __syncwarp();
  }
  // records of tile ti on their way to shared memory
  auto look_fetch = [&](int ti) {
    if (look_half < 0 || ti >= NT) return;
    const int T = T0 + ti;
    int lb = S.lb[look_half];
    while (T >= a.toff[lb + 1]) ++lb;
    const int p0 = a.boff[lb] + (T - a.toff[lb]) * a.per, p1 = min(a.boff[lb + 1], p0 + a.per);
    __syncwarp();
    S.lb[look_half] = lb;
    if (look_half == 0 && lane == 0) {
      S.next[ti & 1][0] = (p1 - p0) * a.rt;
      S.next[ti & 1][1] = lb;
      S.next[ti & 1][2] = p0;
    }
    if (lane < KP / 4)
      cp_async16(&S.exps[ti & 1][KP * look_half + 4 * lane], a.exps + (size_t)lb * 2 * KP + KP * look_half + 4 * lane);
    const int c = look_half * 32 + lane;
    if (c < (p1 - p0) * a.rt) {
      const IbRec *r = a.rec + p0 + c / a.rt;
      cp_async16(&S.rec[ti & 1][c], r);
      cp_async16(reinterpret_cast<char *>(&S.rec[ti & 1][c]) + 16, reinterpret_cast<const char *>(r) + 16);
    }
  };
  // the words of its t and phases
  auto look_form = [&](int ti) {
    if (look_half < 0 || ti >= NT) return;
    IbTile<KP> &t = S.tile[ti & 3];
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    const int c = look_half * 32 + lane;
    const IbRec rc = S.rec[ti & 1][c];  // unused columns hold an old record
    if (look_half == 0) {
      for (int e = lane; e < KP; e += 32) t.eb[e] = S.exps[ti & 1][e];
      if (lane == 0) {
        t.ncol = S.next[ti & 1][0];
        t.bucket = S.next[ti & 1][1];
        t.pair0 = S.next[ti & 1][2] - a.s0;
      }
    } else {
      for (int e = lane; e < KP; e += 32) t.ea[e] = S.exps[ti & 1][KP + e];
    }
    auto words = [](double v, int up) {  // v in units of 2^-up, |v| <= 1
      return ib_split_signed(min(ib_fixed<10>(v, 1023 + 62 - up - ib_field(v)), kIbBelowOne));
    };
    const IbWords tw = words(rc.t, 62);
    t.t[c] = make_int2(tw.h, tw.l);
    t.xoff[c] = 2 * ((long long)rc.j * bs * a.R + a.r0 + c % a.rt);
    t.ph[c][0] = make_int4(1 << 30, 0, 0, 0);
    double pr = rc.c, pi = rc.s;
    for (int m = 1; m <= a.mmax; ++m) {
      const IbWords cw = words(pr, 61), sw = words(pi, 61);
      t.ph[c][m] = make_int4(cw.h, cw.l, sw.h, sw.l);
      const double nr = pr * rc.c - pi * rc.s;
      pi = pr * rc.s + pi * rc.c;
      pr = nr;
    }
    __syncwarp();
    if (lane == 0) tc_arrive(smem_u32(&S.meta[ti & 3]));
  };
  // ------------------------------------------------------------------ issue
  // Job number g (counted over the CTA's tiles) is issued by warp g mod 16, so that the time a thread is held while
  // the tensor core takes its MMAs (73 cycles each) is spread over the warps. Its accumulator is free once every warp
  // has read job g - 4.
  const uint32_t idesc = (1u << 4) | ((uint32_t)(kIbN >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);  // F16 in, F32 out
  const uint64_t da = tc_desc<Sh::KC>(smem_u32(As)), db = tc_desc<Sh::KC>(smem_u32(Bs));
  const uint32_t dal = (uint32_t)da, dbl = (uint32_t)db, dhi = (uint32_t)(da >> 32);
  auto issue = [&](uint32_t g, int pass, auto weight) {
    int ok = 1;
    if (lane == 0) {
      if (g >= 4) ok = tc_wait1(smem_u32(&S.dempty[g & 3]), ((g >> 2) - 1) & 1);
      if (ok) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        ib_issue<decltype(weight)::value, KP>(tmem + (g & 3) * kIbN, dal, dbl + (Sh::STREAM ? 0u : (uint32_t)(pass * (Sh::OPERAND >> 4))),
                                              dhi, idesc);
        tc_commit(smem_u32(&S.dfull[g & 3]));
      }
    }
    return __shfl_sync(kTcFull, ok, 0) != 0;
  };
    // x_j of this warp's four columns of tile ti on their way to shared memory
    auto fetch = [&](int ti) {
      const IbTile<KP> &t = S.tile[ti & 3];
      const int chunk = lane >> 3, q = lane & 7, n2 = chunk * 8 + q;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int col = warp * 4 + c;
        if (col < t.ncol && n2 < bs)
          cp_async16(&S.x[col * kIbXPitch + q * 4 + chunk], a.x + t.xoff[col] + 2 * (size_t)n2 * a.R);
      }
    };
    // rotate the columns of tile ti and cut them into digits; a lane owns a row (column and part) and every fourth
    // core column of eight n2
    auto form = [&](int ti) {
      IbTile<KP> &t = S.tile[ti & 3];
      const int rl = lane & 7, chunk = lane >> 3, row = warp * 8 + rl, col = row >> 1, part = row & 1;
      const bool have = col < t.ncol;
      if (warp * 4 < t.ncol) {
        constexpr int CH = (Sh::KC + 3) / 4;
        double xv[CH][8];
        int emax = 0;
#pragma unroll
        for (int k = 0; k < CH; ++k) {
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int n2 = (chunk + 4 * k) * 8 + q;
            if (Sh::STREAM) xv[k][q] = have && n2 < bs ? __ldg(a.x + t.xoff[col] + part + 2 * (size_t)n2 * a.R) : 0.0;
            else xv[k][q] = have && n2 < bs ? reinterpret_cast<const double *>(S.x + col * kIbXPitch + chunk)[8 * q + part] : 0.0;
          }
        }
#pragma unroll
        for (int k = 0; k < CH; ++k)
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int f = ib_field(xv[k][q]);  // zero beyond the block; Inf, NaN: see below
            if (f != 0) emax = max(emax, f == 0x7FF ? 1 << 20 : f + t.eb[(chunk + 4 * k) * 8 + q] + 4096);
          }
        emax = max(emax, __shfl_xor_sync(kTcFull, emax, 1));
        emax = max(emax, __shfl_xor_sync(kTcFull, emax, 8));
        emax = max(emax, __shfl_xor_sync(kTcFull, emax, 16));
        if (part == 0 && chunk == 0) t.cexp[col] = emax;
        const int es = emax - 4096;  // |Re x|, |Im x| < 2^(es - 1022) under the column exponents
        const int4 *pc = t.ph[have ? col : 0];
#pragma unroll
        for (int k = 0; k < CH; ++k) {
          const int core = min(chunk + 4 * k, Sh::KC - 1);
          unsigned char *dst = As + (size_t)(row >> 3) * (Sh::KC * 128) + (row & 7) * 16 + core * 128;
          uint32_t o[kIbDig][4];
#pragma unroll
          for (int q = 0; q < 8; q += 2) {
            long long u[2];
#pragma unroll
            for (int w = 0; w < 2; ++w) {
              const int n2 = core * 8 + q + w, m = S.mofn[n2];
              const double x = xv[k][q + w];
              const IbWords f = ib_split(ib_fixed<Num::UP>(x, es - t.eb[n2] - ib_field(x)));
              const int oh = __shfl_xor_sync(kTcFull, f.h, 1), ol = __shfl_xor_sync(kTcFull, f.l, 1);
              // half of Re = c xr - s xi or Im = c xi + s xr
              int4 p = pc[m < 0 ? -m : m];
              if ((m < 0) == (part != 0)) {
                p.z = -p.z;
                p.w = -p.w;
              }
              const long long mid = ib_mad(f.h, p.y, ib_mad(f.l, p.x, ib_mad(oh, p.w, ib_mad(ol, p.z, 0x40000000ll))));
              u[w] = ib_mad(f.h, p.x, ib_mad(oh, p.z, mid >> 31));
            }
            uint32_t dg[kIbDig];
            ib_digits<KP>(u[0], u[1], dg);
#pragma unroll
            for (int s = 0; s < kIbDig; ++s) o[s][q >> 1] = dg[s];
          }
          if (chunk + 4 * k < Sh::KC)
#pragma unroll
            for (int s = 0; s < kIbDig; ++s)
              *reinterpret_cast<uint4 *>(dst + (size_t)s * Sh::SLICE) = make_uint4(o[s][0], o[s][1], o[s][2], o[s][3]);
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) tc_arrive(smem_u32(&S.afull));
    };
    const int sp = warp & 3, grp = warp >> 2;
    const int col = sp * 16 + (lane >> 1), part = lane & 1, sg = part ? -1 : 1;
    const uint32_t lanes = tmem + ((uint32_t)(sp * 32) << 16) + (uint32_t)(grp * 32);
    uint32_t g = 0;  // jobs read
    // waits for the next job (weight D of pass p); read() gets 16 of this warp's 32 columns at a time; then the
    // buffer is free for the job after next three, whose issuing warp sends it off
    auto job = [&](auto weight, int p, bool work, auto &&read) {
      constexpr int D = decltype(weight)::value, DN = D + 4 < Num::JOBS ? D + 4 : D + 4 - Num::JOBS;
      if (!tc_waitw(smem_u32(&S.dfull[g & 3]), (g >> 2) & 1)) return false;
      if (work) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int h = 0; h < 32; h += 16) {
          float f[16];
          tmem_ld16(lanes + (g & 3) * kIbN + h, f);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int c = 0; c < 16; ++c) read(h + c, f[c]);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      }
      __syncwarp();
      if (lane == 0) tc_arrive(smem_u32(&S.dempty[g & 3]));
      ++g;
      const int pn = D + 4 < Num::JOBS ? p : p + 1;
      if (Sh::STREAM && D + 4 >= Num::JOBS) return true;  // the next pass starts when its operand is there
      return ((g + 3) & (kIbWarps - 1)) != warp || pn >= passes || issue(g + 3, pn, std::integral_constant<int, DN>());
    };
    int cur_b = -1, bloads = 0;
    auto wait_meta = [&](int ti) { return tc_waitw(smem_u32(&S.meta[ti & 3]), (uint32_t)((ti >> 2) & 1)); };
    // the B operand of a bucket (STREAM: one pass of it), once every MMA that read the last one has completed
    auto load_b = [&](int bucket, int pass) {
      ++bloads;
      if (warp == 0 && lane == 0) {
        const uint32_t bar = smem_u32(&S.bfull), bytes = (uint32_t)((Sh::STREAM ? 1 : passes) * Sh::OPERAND);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(Bs)),
            "l"(a.B + (size_t)bucket * Sh::BBYTES + (size_t)pass * Sh::OPERAND), "r"(bytes), "r"(bar)
            : "memory");
      }
    };
    // the first four jobs of a pass of tile ti
    auto start = [&](int ti, int pass) {
      const int mine = (int)((uint32_t)warp - g) & (kIbWarps - 1);
      if (mine >= 4) return true;
      if (pass == 0 && !tc_waitw(smem_u32(&S.afull), (uint32_t)(ti & 1))) return false;
      if (!tc_waitw(smem_u32(&S.bfull), (uint32_t)((bloads - 1) & 1))) return false;
      if (mine == 0) return issue(g, pass, std::integral_constant<int, 0>());
      if (mine == 1) return issue(g + 1, pass, std::integral_constant<int, 1>());
      if (mine == 2) return issue(g + 2, pass, std::integral_constant<int, 2>());
      return issue(g + 3, pass, std::integral_constant<int, 3>());
    };
    look_fetch(0);
    look_form(0);
    look_fetch(1);
    look_form(1);
    look_fetch(2);
    good = NT == 0 || wait_meta(0);
    if (good && NT > 0) {
      if (!Sh::STREAM) fetch(0);
      if (Sh::STREAM) load_b(S.tile[0].bucket, 0);
    }
    for (int ti = 0; ti < NT && good; ++ti) {
      IbTile<KP> &t = S.tile[ti & 3];
      look_form(ti + 2);
      // every job of the last tile has been read: its operands are free
      if (!Sh::STREAM && t.bucket != cur_b) {
        cur_b = t.bucket;
        load_b(cur_b, 0);
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncwarp();
      form(ti);
      look_fetch(ti + 3);
      if (ti + 1 < NT) {
        good = wait_meta(ti + 1);
        if (!good) break;
        if (!Sh::STREAM) fetch(ti + 1);
      }
      good = start(ti, 0);
      for (int p = 0; p < passes && good; ++p) {
        if (Sh::STREAM && p > 0) {
          good = start(ti, p);
          if (!good) break;
        }
        const int n0 = p * PN + grp * WN;
        const bool work = sp * 16 < t.ncol && n0 < bs;
        // The digits in units of 2^-UNIT of the scales; the Im rows of C are negated in the Im u lanes. What is
        // below 2^22 becomes an integer by an FP32 addition of 1.5 2^23, whose exponent bits stay in the sum
        // and are taken off it (OFFSET) below.
        auto unit = [&](int c, int u) { return c & 1 ? sg * u : u; };
        auto bits = [](float f) { return __float_as_int(f + kIbMagic); };
        auto high = [&](int c, float f, int u) {
          return (long long)((unsigned long long)((unsigned)bits(f) * (unsigned)unit(c, u)) << 32);
        };
        long long w[32];
        std::integral_constant<int, 0> w0;
        std::integral_constant<int, 1> w1;
        std::integral_constant<int, 2> w2;
        std::integral_constant<int, 3> w3;
        std::integral_constant<int, 4> w4;
        std::integral_constant<int, 5> w5;
        std::integral_constant<int, 6> w6;
        if constexpr (KP == 32) {
          good = job(w0, p, work, [&](int c, float f) { w[c] = high(c, f, 1 << 7); });
          good = good && job(w1, p, work, [&](int c, float f) { w[c] = ib_mad(bits(f), unit(c, 1 << 30), w[c]); });
          good = good && job(w2, p, work, [&](int c, float f) { w[c] = ib_mad(__float2int_rn(f), unit(c, 1 << 21), w[c]); });
          good = good && job(w3, p, work, [&](int c, float f) { w[c] = ib_mad(__float2int_rn(f), unit(c, 1 << 12), w[c]); });
          good = good && job(w4, p, work, [&](int c, float f) { w[c] = ib_mad(__float2int_rn(f), unit(c, 8), w[c]); });
          good = good && job(w5, p, work, [&](int c, float f) { w[c] = ib_mad(bits(f * 0x1p-6f), unit(c, 1), w[c]); });
          good = good && job(w6, p, work, [&](int c, float f) { w[c] = ib_mad(bits(f * 0x1p-15f), unit(c, 1), w[c]); });
        } else {
          good = job(w0, p, work, [&](int c, float f) { w[c] = high(c, f, 1 << 8); });
          good = good && job(w1, p, work, [&](int c, float f) {
            w[c] = (long long)((unsigned long long)w[c] + (unsigned long long)high(c, f, 1));
          });
          good = good && job(w2, p, work, [&](int c, float f) { w[c] = ib_mad(bits(f), unit(c, 1 << 24), w[c]); });
          good = good && job(w3, p, work, [&](int c, float f) { w[c] = ib_mad(bits(f), unit(c, 1 << 16), w[c]); });
          good = good && job(w4, p, work, [&](int c, float f) { w[c] = ib_mad(bits(f), unit(c, 1 << 8), w[c]); });
          good = good && job(w5, p, work, [&](int c, float f) { w[c] = ib_mad(__float2int_rn(f), unit(c, 1), w[c]); });
          good = good && job(w6, p, work, [&](int c, float f) { w[c] = ib_mad(bits(f * 0x1p-8f), unit(c, 1), w[c]); });
          good = good && job(std::integral_constant<int, 7>(), p, work, [&](int c, float f) {
            w[c] = ib_mad(bits(f * 0x1p-16f), unit(c, 1), w[c]);
          });
        }
        if (Sh::STREAM && good) {  // every MMA of this pass has completed
          if (p + 1 < passes) load_b(t.bucket, p + 1);
          else if (ti + 1 < NT) load_b(S.tile[(ti + 1) & 3].bucket, 0);
        }
        if (!good || !work) continue;
        const bool have = col < t.ncol;
        const int2 tw = have ? t.t[col] : make_int2(0, 0);
        const int ce = have ? t.cexp[col] : 0;
        const int cs = ce - 4096 - 1022 + 1 - Num::UNIT;  // scale of x, half of its rotation, units
        // the Re lane receives the negated Im sum (offsets cancel), the Im lane adds two positive ones
        const unsigned long long offset = part ? 0ull - 2ull * Num::OFFSET : 0ull;
        const int4 *pc = t.ph[have ? col : 0];
        double *vo = a.V + 2 * ((t.pair0 * a.rt + (have ? col : 0)) * bs) + part;
#pragma unroll
        for (int s = 0; s < WN; ++s) {
          const int n = n0 + s;
          // lane pair (Re u, Im u): Re y = C_re u_re - C_im u_im, Im y = C_re u_im + C_im u_re
          long long acc = 0;
#pragma unroll
          for (int c = NC - 1; c >= 0; --c) {
            const long long e = (long long)((unsigned long long)w[s * RN + 2 * c] + offset +
                                            (unsigned long long)__shfl_xor_sync(kTcFull, w[s * RN + 2 * c + 1], 1));
            acc = c == NC - 1 ? e : ib_mul(ib_split(acc), tw.x, tw.y, e);
          }
          const IbWords v = ib_split(acc);
          const int oh = __shfl_xor_sync(kTcFull, v.h, 1), ol = __shfl_xor_sync(kTcFull, v.l, 1);
          const int nc = min(n, KP - 1), m = S.mofn[nc];
          int4 ph = pc[m < 0 ? -m : m];
          if ((m < 0) != (part != 0)) {
            ph.z = -ph.z;
            ph.w = -ph.w;
          }
          // e^{-i m phi} times the value: c v +- s (other part)
          const long long mid = ib_mad(v.h, ph.y, ib_mad(v.l, ph.x, ib_mad(oh, ph.w, ib_mad(ol, ph.z, 0x20000000ll))));
          const long long out = 2 * ib_mad(v.h, ph.x, (long long)oh * ph.z) + (mid >> 30);
          double res = ib_to_double(out, cs + t.ea[nc]);
          if (ce >= (1 << 20)) res = __longlong_as_double(0x7FF8000000000000ll);  // Inf or NaN in x
          if (have && n < bs) vo[2 * n] = res;
        }
      }
    }
  if (!good && lane == 0) atomicExch(a.err, 1);
  // nothing of this CTA may be in flight when its memory is given back
  if (lane == 0) {
    tc_commit(smem_u32(&S.done));
    if (!tc_wait1(smem_u32(&S.done), 0u)) atomicExch(a.err, 1);
    if (warp == 0 && bloads > 0) tc_wait1(smem_u32(&S.bfull), (uint32_t)((bloads - 1) & 1));
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
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
__global__ void __launch_bounds__(768) ib_sum_kernel(const CouplingLaunch L, const IbSum s) {
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
template <int NC, int KP>
__global__ void __launch_bounds__(256) ib_operand_kernel(const double2 *coef, const int *bk, int bs, unsigned char *B,
                                                         int *exps) {
  using Sh = IbShape<NC, KP>;
  __shared__ int eb[KP], ea[KP];
  const int tid = threadIdx.x, b = blockIdx.x, bs2 = bs * bs;
  const double2 *C = coef + (size_t)bk[b] * NC * bs2;
  if (tid < KP) {
    eb[tid] = ea[tid] = -(1 << 20);
  }
  __syncthreads();
  for (int e = tid; e < NC * bs2; e += blockDim.x) {
    const int f = max(ib_field(C[e].x), ib_field(C[e].y));
    if (f) atomicMax(&eb[(e % bs2) / bs], f - 1022);
  }
  __syncthreads();
  if (tid < KP && eb[tid] == -(1 << 20)) eb[tid] = 0;
  __syncthreads();
  for (int e = tid; e < NC * bs2; e += blockDim.x) {
    const int f = max(ib_field(C[e].x), ib_field(C[e].y));
    if (f) atomicMax(&ea[e % bs], f - 1022 - eb[(e % bs2) / bs]);
  }
  __syncthreads();
  if (tid < KP && ea[tid] == -(1 << 20)) ea[tid] = 0;
  __syncthreads();
  if (tid < KP) {
    exps[(size_t)b * 2 * KP + tid] = eb[tid];
    exps[(size_t)b * 2 * KP + KP + tid] = ea[tid];
  }
  unsigned char *out = B + (size_t)b * Sh::BBYTES;
  // one thread per row (n1, power, part) and pair of n2
  for (int e = tid; e < Sh::PASSES * kIbN * KP / 2; e += blockDim.x) {
    const int row = e / (KP / 2), k = 2 * (e - row * (KP / 2));
    const int n1 = row / Sh::RN, c = (row % Sh::RN) >> 1, im = row & 1;
    long long f[2];
    for (int w = 0; w < 2; ++w) {
      const int n2 = k + w;
      double v = 0.0;
      if (n1 < bs && n2 < bs) {
        const double2 cv = C[(size_t)c * bs2 + n2 * bs + n1];
        v = im ? cv.y : cv.x;
      }
      f[w] = ib_fixed<IbNumbers<KP>::UP>(v, n1 < bs && n2 < bs ? ea[n1] + eb[n2] + 1022 - ib_field(v) : 0);
    }
    uint32_t dg[kIbDig];
    ib_digits<KP>(f[0], f[1], dg);
    const int pass = row / kIbN, r = row % kIbN;
    for (int s = 0; s < kIbDig; ++s)
      *reinterpret_cast<uint32_t *>(out + (size_t)pass * Sh::OPERAND + (size_t)s * Sh::SLICE +
                                    ((size_t)(r >> 3) * Sh::KC + (k >> 3)) * 128 + (r & 7) * 16 + (k & 7) * 2) = dg[s];
  }
}

static constexpr int kIbMinParticles = 32;
static constexpr long long kIbMaxPairs = 1ll << 27;      // 4 GB of pair records
static constexpr size_t kIbWorkspace = (size_t)2 << 30;  // bytes of V per chunk

// padded blocksize
static int ib_kp(const sg_context *c) { return c->bs <= IbNumbers<32>::MAXB ? 32 : 48; }

bool ib_supported(const sg_context *c) {
  if (c->vol || c->kind < 0 || c->bs > IbNumbers<48>::MAXB) return false;
  if ((long long)c->n * c->n > kIbMaxPairs || c->n < kIbMinParticles) return false;
  const int mmax = ib_kp(c) == 32 ? IbNumbers<32>::MAXM : IbNumbers<48>::MAXM;
  for (int m : c->h_mofn)
    if (m > mmax || m < -mmax) return false;
  return true;
}

// f(NC, KP) as compile-time constants
template <class F>
static void ib_dispatch(const sg_context *c, F &&f) {
  std::integral_constant<int, 2> two;
  std::integral_constant<int, 4> four;
  std::integral_constant<int, 32> small;
  std::integral_constant<int, 48> large;
  if (ib_kp(c) == 32) {
    if (c->ncoef == 2) f(two, small);
    else f(four, small);
  } else {
    if (c->ncoef == 2) f(two, large);
    else f(four, large);
  }
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
  P.exps.reserve((size_t)P.nb * 2 * ib_kp(c));
  ib_dispatch(c, [&](auto nc, auto kp) { P.B.reserve((size_t)P.nb * IbShape<decltype(nc)::value, decltype(kp)::value>::BBYTES); });
  SG_CUDA(cudaMemcpyAsync(dbk.ptr, bk.data(), P.nb * sizeof(int), cudaMemcpyHostToDevice, st));
  SG_CUDA(cudaMemcpyAsync(P.boff.ptr, P.h_boff.data(), (P.nb + 1) * sizeof(int), cudaMemcpyHostToDevice, st));
  ib_dispatch(c, [&](auto nc, auto kp) {
    ib_operand_kernel<decltype(nc)::value, decltype(kp)::value>
        <<<P.nb, 256, 0, st>>>(c->coef64.ptr, dbk.ptr, c->bs, P.B.ptr, P.exps.ptr);
  });
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

template <int NC, int KP>
static void ib_launch(const IbArgs &a, cudaStream_t st) {
  static bool attr_done[64] = {};
  constexpr int smem = (int)ib_smem<NC, KP>();
  if (first_on_device(attr_done))
    SG_CUDA(cudaFuncSetAttribute(ib_kernel<NC, KP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  ib_kernel<NC, KP><<<std::min(sm_count(), a.t1 - a.t0), kIbThreads, smem, st>>>(a);
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
    a.x = reinterpret_cast<const double *>(x);
    a.mofn = c->mofn.ptr;
    a.V = reinterpret_cast<double *>(P.V.ptr);
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
      ib_dispatch(c, [&](auto nc, auto kp) { ib_launch<decltype(nc)::value, decltype(kp)::value>(a, st); });
      ib_sum_kernel<<<c->n, std::max(512, s.width), smem, st>>>(L, s);
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
