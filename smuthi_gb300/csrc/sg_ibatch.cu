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
// Numer. Algorithms 59 (2012)): every operand is a 62-bit fixed-point number under a power-of-two
// scale (per column of C, then per row of C; per pair and right-hand side for u) cut into seven signed
// 9-bit digits, which FP16 holds exactly. The digit products of equal weight 2^(-9 d), d = 0..6, share
// one FP32 accumulator; smaller products (below 2^-60 of the scales) are dropped. The complex product is
// one real one of twice the depth: a row of A holds (Im u, Re u), a column of B (-Im C, Re C) or
// (Re C, Im C), so an accumulator holds Re or Im of a result. A digit product is at most 2^16 and at most
// 60 (blocksize <= 30) times d + 1 of them are summed: the weights d <= 3 stay exact integers below 2^24
// whatever the digits and the order of the sums; d = 4..6 could pass 2^24 only if nearly all digits had
// their largest magnitude and one sign, and would then be rounded at 2^-51 of the scales, under a sum
// that is itself 60 times as large. Blocksizes 31 to 48 take 8-bit digits of 55-bit numbers and the
// weights d = 0..7, at most 7 * 96 * 2^14 < 2^24. The digits are combined in 64-bit integers, in which
// the powers of t and the rotations follow; the result is independent of how the pairs are grouped. Accuracy is by the
// scales, row of C times column of x, and not by element: an element 2^-9 and more below them (2^-2 with 8-bit digits)
// keeps fewer than 53 bits.
//
// One CTA per SM walks a contiguous range of tiles; a tile is up to 128 complex columns (pairs x
// right-hand sides) of one interval:
//   * sixteen warps rotate x_j, cut u into digits and store them as the A operand in tensor memory (a
//     lane per column), which leaves shared memory to B and its bandwidth to the tensor core;
//   * one thread issues the digit products against the interval's B operand (resident while the
//     interval lasts; with K = 48 one pass at a time): passes of 64 (n1, power of t), one job per
//     weight, the least first, in one or two accumulators of 128 columns (64 Re, 64 Im);
//   * the sixteen warps read the jobs back, combine digits and powers of t, rotate back and store the
//     pair's contribution V;
//   * three more warps fetch the next tiles' records and prepare the words of t and the phases.
// A second kernel sums V over the emitters of every receiver in index order (deterministic) and forms
// W x or x - T W x. V is a bounded workspace: larger problems run in chunks of tiles.
//
// What bounds it: instruction issue (42% of the slots with 1000 spheres, half of them two-cycle integer instructions) and
// the tensor core (34%) in turn: a tile of 2000 spheres takes 44 thousand cycles, of which 16 are MMAs, 6 forming A,
// 13 the last combination; operand memory does not allow a second tile in flight. 2000 spheres, cubic lookup, one
// right-hand side: 80.5 ms with the per-receiver kernel, 9.3 with Re and Im of u as separate rows of A in shared
// memory (twice the accumulators to read and combine), 5.2 now; 1201 spheres with l_max = 4: 82.4, 8.0, 5.05; 100
// spheres, linear: 127, 51, 46 us.
//
// Integer arithmetic instead of FP64: a GB300 SM sub-partition issues an FP64 instruction every 64 cycles, a
// 32-bit integer one every two.
#include <cub/cub.cuh>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "sg_epilogue.h"
#include "sg_ibatch.h"
#include "sg_internal.h"
#include "sg_tcgen05.h"

namespace sg {

static constexpr int kIbWarps = 16;  // warps that form, read and combine; one of four more issues
static constexpr int kIbThreads = 32 * (kIbWarps + 4);
// The block is launched with 96 registers a thread (20 warps); its 61440 are split 512 x 104 + 128 x 64.
#define IB_SETMAXNREG(dir, n) asm volatile("setmaxnreg." #dir ".sync.aligned.u32 " #n ";")
static constexpr int kIbCols = 128;  // complex columns per tile
static constexpr int kIbDig = 7;     // digits per operand
static constexpr int kIbRows = 64;   // (n1, power of t) per pass: N = 128 accumulator columns, Re and Im
// 1.5 2^23: added to an integer below 2^22 it leaves that in the mantissa
static constexpr float kIbMagic = 12582912.f;
static constexpr unsigned kIbMagicBits = 0x4B400000u;
// first t in units of 2^-62 whose high word would not fit beside a signed low one
static constexpr long long kIbNearOne = (1ll << 62) - (1ll << 30);

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
      (unsigned long long)(unsigned)(kIbMagicBits * (KP == 32 ? 9u : 2u)) +
      (unsigned long long)kIbMagicBits * (KP == 32 ? (1ull << 39) + (1ull << 30) + (1ull << 21) + (1ull << 12)
                                                   : (1ull << 40) + (1ull << 32) + (1ull << 24) + (1ull << 16) + (1ull << 8));
  // weights up to 3 (K = 64) or all (K = 96) are exact in FP32 whatever the digits
  static_assert((KP == 32 ? 4 : kIbDig) * 2 * MAXB * (1 << (2 * BITS - 2)) <= (1 << 24), "exact FP32 accumulators");
  static_assert((KP == 32 ? 1 : 2) * 2 * MAXB * (1 << (2 * BITS - 2)) < (1 << 22), "weights that need no check");
};

template <int NC, int KP>
struct IbShape {
  static constexpr int KC = KP / 8;                  // chunks of eight n2: one K = 16 step of (Im u, Re u)
  static constexpr int PLANE = 3 * kIbRows * 16;     // bytes of a chunk of B: rows of -Im C, Re C, Im C
  static constexpr int SLICE = KC * PLANE;           // bytes of one digit of a pass of B
  static constexpr int OPERAND = kIbDig * SLICE;     // bytes of one pass of B
  static constexpr int PN = kIbRows / NC;            // n1 per pass
  static constexpr int PASSES = (KP + PN - 1) / PN;  // at most
  static constexpr int BBYTES = PASSES * OPERAND;
  static constexpr bool STREAM = KP > 32;            // B in shared memory: one pass, or all
  static constexpr int BSMEM = STREAM ? OPERAND : BBYTES;
  static constexpr int BUFS = KP == 32 ? 2 : 1;      // accumulators of 128 tensor-memory columns
  static constexpr int ACOL = BUFS * 128;            // first tensor-memory column of A: KP columns per digit
  static_assert(ACOL + kIbDig * KP <= 512, "tensor memory");
};

// The n2 of a warp group (a quarter of the KP) are a chunk of eight and, with KP = 48, four more that
// share a chunk with a neighbour's: chunk and place of n2.
template <int KP>
__host__ __device__ constexpr int ib_chunk(int n2) {
  return n2 % (KP / 4) < 8 ? n2 / (KP / 4) : 4 + n2 / (KP / 4) / 2;
}
template <int KP>
__host__ __device__ constexpr int ib_place(int n2) {
  return n2 % (KP / 4) < 8 ? n2 % (KP / 4) : n2 / (KP / 4) % 2 * 4 + n2 % (KP / 4) - 8;
}

// SETS: 1: the tiles have 128 columns, all warps take part in each. 2: 64 columns; odd and even tiles belong to two
// sets of eight warps and 64 tensor-memory lanes, which run half a tile apart. (The products cover all lanes; what
// they give in those of the other set, from digits that may just be being written there, nobody reads.)
template <int NC, int KP, int SETS>
struct IbSmem {
  static constexpr int COLS = kIbCols / SETS;
  // two B operands where there is room: the next interval's is on its way while the last one is used
  static constexpr int NB = KP == 32 && NC == 2 ? 2 : 1;
  struct Tile {
    int4 ph[IbNumbers<KP>::MAXM + 1][COLS];  // cos, sin of m phi in words of 2^-61
    int2 t[COLS];                // t in words of 2^-62
    int xoff[COLS];              // x_j of the column
    int eb[KP], ea[KP];          // column and row exponents of the interval
    int ncol, bucket;
    long long pair0;             // first pair, from the start of V
  };
  struct Set {
    Tile tile[4];                // written ahead, read until the tile is stored
    uint64_t dfull[2], dempty[2], afull, meta[4], tfree[4];
  } set[SETS];
  int emax[4][kIbCols];          // exponents of the quarters of a column
  uint64_t quarters[4], bfull[2], done;
  int mofn[KP];
  uint32_t tmem;
};
template <int NC, int KP, int SETS>
constexpr size_t ib_smem() {
  using Sm = IbSmem<NC, KP, SETS>;
  return (size_t)Sm::NB * IbShape<NC, KP>::BSMEM + (sizeof(Sm) + 127) / 128 * 128;
}
template <int KP, int SETS>
constexpr bool ib_fits = ib_smem<2, KP, SETS>() <= kTcSmemBudget && ib_smem<4, KP, SETS>() <= kTcSmemBudget;
static_assert(ib_fits<32, 1> && ib_fits<32, 2> && ib_fits<48, 1> && ib_fits<48, 2>, "shared memory");

struct IbArgs {
  const IbRec *rec;       // ordered pairs sorted by interval
  const int *boff;        // [nb + 1] first pair of every non-empty interval
  const int *toff;        // [nb + 1] first tile
  const unsigned char *B; // [nb] B operands
  const int *exps;        // [nb][2 KP]: column exponents eb[KP], row exponents ea[KP]
  const int4 *x;          // [N][rt][KP] words of x (ib_words_kernel)
  const int *xe;          // their exponents
  const int *mofn;
  double2 *V;             // [pair - s0][rt][bs]
  long long s0;           // first pair of this chunk
  int nb, bs, mmax, rt, per, t0, t1;  // rt right-hand sides; per = pairs per tile; tiles [t0, t1)
  int *err;
};

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
// t, in units of 2^-62. The last 2^-32 below one keep an unsigned low word: with |h|, l < 2^31 the middle products of
// ib_mul still stay within 2^63, and the bias of what it drops, below one unit, is that of the few pairs that close to
// the end of an interval.
__device__ __forceinline__ IbWords ib_split_fraction(long long v) {
  return v >= kIbNearOne ? ib_split(v) : ib_split_signed(v);
}
__device__ __forceinline__ long long ib_mad(int a, int b, long long c) { return (long long)a * b + c; }
// a b / 2^62 + c
__device__ __forceinline__ long long ib_mul(IbWords a, int bh, int bl, long long c) {
  const long long mid = ib_mad(a.h, bl, ib_mad(a.l, bh, 0x40000000ll));
  return ib_mad(a.h, bh, c + (mid >> 31));
}

// v 2^e rounded to double (halves away from zero), in integers: an FP64 conversion or addition holds its pipe for
// 64 cycles
__device__ __forceinline__ double ib_to_double(long long v, int e) {
  const unsigned sign = (unsigned)((unsigned long long)v >> 32) & 0x80000000u;
  const unsigned long long m = (unsigned long long)(v < 0 ? -v : v);
  const unsigned hi = (unsigned)(m >> 32), lo = (unsigned)m;
  const int z = __clz((int)hi), f = 1023 + 63 - z + e;  // exponent field
  if (hi != 0 && f > 0 && f < 0x7FE) {
    const unsigned mh = __funnelshift_l(lo, hi, z), ml = lo << (z & 31);
    // the leading bit adds one to the field, a carry out of the mantissa another
    const unsigned long long b = (((unsigned long long)mh << 32 | ml) >> 11) + ((ml >> 10) & 1u);
    return __hiloint2double((int)(((unsigned)(b >> 32) + ((unsigned)(f - 1) << 20)) | sign), (int)(unsigned)b);
  }
  return scalbn((double)v, e);  // below 2^32, or outside the normal range
}

// One product of a digit of A (tensor memory, column AO of it) and a digit of B (K = 16, BO bytes into the pass) into
// dst. The offsets are added here, so that the compiler does not keep a hundred addresses.
template <bool ACC, int AO, int BO>
__device__ __forceinline__ void ib_mma(uint32_t dst, uint32_t a, uint32_t b, uint32_t hi, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t.reg .b32 ra, rb;\n\t"
      "add.u32 ra, %1, %6;\n\t"
      "add.u32 rb, %2, %7;\n\t"
      "mov.b64 db, {rb, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [ra], db, %4, p;\n\t}" ::"r"(dst),
      "r"(a), "r"(b), "r"(hi), "r"(idesc), "n"(ACC ? 1 : 0), "n"(AO), "n"(BO >> 4)
      : "memory");
}

// all digit products of weight D; unrolled, because one thread issues them and every instruction between two
// MMAs costs it several cycles
template <int D, int NC, int KP, int I = (D < kIbDig ? 0 : D - kIbDig + 1), int K = 0>
__device__ __forceinline__ void ib_issue(uint32_t dst, uint32_t a, uint32_t b, uint32_t hi, uint32_t idesc) {
  using Sh = IbShape<NC, KP>;
  constexpr int I0 = D < kIbDig ? 0 : D - kIbDig + 1, I1 = D < kIbDig ? D : kIbDig - 1;
  if constexpr (K == Sh::KC) {
    ib_issue<D, NC, KP, I + 1, 0>(dst, a, b, hi, idesc);
  } else if constexpr (I <= I1) {
    ib_mma<(I != I0 || K != 0), I * KP + K * 8, (D - I) * Sh::SLICE + K * Sh::PLANE>(dst, a, b, hi, idesc);
    ib_issue<D, NC, KP, I, K + 1>(dst, a, b, hi, idesc);
  }
}

__device__ __forceinline__ void tmem_st2(uint32_t taddr, uint32_t a, uint32_t b) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1,%2};" ::"r"(taddr), "r"(a), "r"(b) : "memory");
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
               : "r"(taddr));
}

template <int NC, int KP, int SETS>
__global__ void __launch_bounds__(kIbThreads, 1) ib_kernel(const IbArgs a) {
  using Sh = IbShape<NC, KP>;
  using Num = IbNumbers<KP>;
  using Sm = IbSmem<NC, KP, SETS>;
  constexpr int PN = Sh::PN, WN = PN / 4;  // WN rows n1 per warp and pass
  constexpr int BUFS = Sh::BUFS, NB = Sm::NB;
  extern __shared__ __align__(1024) unsigned char ib_raw[];
  unsigned char *Bs = ib_raw;
  Sm &S = *reinterpret_cast<Sm *>(Bs + NB * Sh::BSMEM);
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
    for (int h = 0; h < SETS; ++h) {
      for (int b = 0; b < 2; ++b) {
        init(&S.set[h].dfull[b], 1);
        init(&S.set[h].dempty[b], kIbWarps / SETS);
      }
      for (int b = 0; b < 4; ++b) {
        init(&S.set[h].meta[b], 4 / SETS);
        init(&S.set[h].tfree[b], kIbWarps / SETS);
      }
      init(&S.set[h].afull, kIbWarps / SETS);
    }
    for (int b = 0; b < 4; ++b) init(&S.quarters[b], 4);
    for (int b = 0; b < 2; ++b) init(&S.bfull[b], 1);
    init(&S.done, 1);
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

  if (warp >= kIbWarps) {
    IB_SETMAXNREG(dec, 64);
    // ---------------------------------------------------------------- issue
    // One thread of a warp of its own: it is held while the tensor core takes an MMA (73 cycles each).
    if (warp == kIbWarps && lane == 0) {
      const uint32_t idesc = (1u << 4) | ((uint32_t)(128 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);  // F16 in, F32 out
      // B: core matrices adjacent in rows 128 bytes apart, in K 64 rows, from -Im C | Re C to Re C | Im C
      const uint32_t blo = ((smem_u32(Bs) >> 4) & 0x3FFFu) | (uint32_t)((kIbRows * 16) >> 4) << 16;
      const uint32_t bhi = (128u >> 4) | (1u << 14);
      uint32_t buf = 0;           // accumulator of the next job
      uint32_t par = 0;           // bit 2 h + b: parity of the next job of set h in accumulator b
      uint32_t user = 0;          // bits 2 b: set of the last job in accumulator b
      uint32_t used = 0;          // bit b: accumulator b has been used
      int slot = 0, held0 = -1, held1 = -1;  // operand in use; intervals in the two places
      uint32_t bpar = 0, arrived = 0;        // parity of the next load of a place; bit: its load has been waited for
      // every MMA of the last tile issued by set h has completed
      auto finished = [&](int h, uint32_t b) {
        return tc_wait1(smem_u32(&S.set[h].dfull[b]), ((par >> (2 * h + b)) & 1) ^ 1);
      };
      auto load = [&](int place, int bucket, int p) {
        const uint32_t bar = smem_u32(&S.bfull[place]), bytes = (uint32_t)((Sh::STREAM ? 1 : passes) * Sh::OPERAND);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                smem_u32(Bs) + place * Sh::BSMEM),
            "l"(a.B + (size_t)bucket * Sh::BBYTES + (size_t)(Sh::STREAM ? p : 0) * Sh::OPERAND), "r"(bytes), "r"(bar)
            : "memory");
        if (place == 0) held0 = bucket;
        else held1 = bucket;
        arrived &= ~(1u << place);
      };
      auto landed = [&](int place) {
        if ((arrived >> place) & 1) return true;
        arrived |= 1u << place;
        const uint32_t q = (bpar >> place) & 1;
        bpar ^= 1u << place;
        return tc_wait1(smem_u32(&S.bfull[place]), q);
      };
      auto bucket_of = [&](int T, int &bucket) {  // of tile T of this CTA
        const int h = T % SETS, n = T / SETS;
        if (!tc_wait1(smem_u32(&S.set[h].meta[n & 3]), (uint32_t)((n >> 2) & 1))) return false;
        bucket = S.set[h].tile[n & 3].bucket;
        return true;
      };
      int lasth = 0;         // set and accumulator of the last job
      uint32_t lastb = 0;
      for (int T = 0; T < NT && good; ++T) {
        const int h = T % SETS, n = T / SETS;
        int bucket = 0;
        good = bucket_of(T, bucket);
        if (!good) break;
        if (NB == 2 && bucket != (slot ? held1 : held0)) slot ^= 1;
        for (int p = 0; p < passes && good; ++p) {
          if (Sh::STREAM || bucket != (slot ? held1 : held0)) {
            // the operand may be replaced once every MMA that reads it has completed
            if (used) good = finished(lasth, lastb);
            if (!good) break;
            load(slot, bucket, p);
          }
          good = landed(slot);
          if (p == 0) good = good && tc_wait1(smem_u32(&S.set[h].afull), (uint32_t)(n & 1));
          const uint32_t bp = blo + (uint32_t)((slot * Sh::BSMEM) >> 4) + (Sh::STREAM ? 0u : (uint32_t)(p * (Sh::OPERAND >> 4)));
          auto issue = [&](auto weight) {
            if (!good) return;
            if ((used >> buf) & 1) {
              const uint32_t u = (user >> (2 * buf)) & 3;  // whoever had the accumulator last has read it
              good = tc_wait1(smem_u32(&S.set[SETS == 1 ? 0 : u].dempty[buf]), ((par >> (2 * u + buf)) & 1) ^ 1);
            }
            if (!good) return;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            ib_issue<decltype(weight)::value, NC, KP>(tmem + buf * 128, tmem + Sh::ACOL, bp, bhi, idesc);
            tc_commit(smem_u32(&S.set[h].dfull[buf]));
            par ^= 1u << (2 * h + buf);
            user = (user & ~(3u << (2 * buf))) | ((uint32_t)h << (2 * buf));
            used |= 1u << buf;
            lasth = h;
            lastb = buf;
            if (BUFS == 2) buf ^= 1;
          };
          if constexpr (Num::JOBS > 7) issue(std::integral_constant<int, 7>());
          issue(std::integral_constant<int, 6>());
          issue(std::integral_constant<int, 5>());
          issue(std::integral_constant<int, 4>());
          issue(std::integral_constant<int, 3>());
          issue(std::integral_constant<int, 2>());
          issue(std::integral_constant<int, 1>());
          issue(std::integral_constant<int, 0>());
          if (NB == 2 && p == 0 && T + 1 < NT && good) {
            // the other place was last read by the tile before this one, whose jobs precede this tile's
            int next = 0;
            good = bucket_of(T + 1, next);
            if (good && next != held0 && next != held1) load(slot ^ 1, next, 0);
          }
        }
      }
      // nothing of this CTA may be in flight when its memory is given back
      tc_commit(smem_u32(&S.done));
      if (!tc_wait1(smem_u32(&S.done), 0u)) good = false;
      if (held0 >= 0) landed(0);
      if (held1 >= 0) landed(1);
    }
    // ---------------------------------------------------------------- look ahead
    // Three warps take the records of the tiles, 32 columns at a time, and leave the words of t and the phases.
    if (warp > kIbWarps) {
      int lb = 0;  // interval of the tile: the last one whose first tile is not behind it
      for (int len = a.nb; len > 1;) {
        const int step = (len + 31) / 32, q = lane * step;
        const unsigned hit = __ballot_sync(kTcFull, q < len && a.toff[lb + min(q, len - 1)] <= T0);
        const int o = (__popc(hit) - 1) * step;
        lb += o;
        len = min(step, len - o);
      }
      auto fixed = [](double v, int up) { return ib_fixed<10>(v, 1023 + 62 - up - ib_field(v)); };  // |v| <= 1 in units of 2^-up
      for (int T = 0; T < NT && good; ++T) {
        while (T0 + T >= a.toff[lb + 1]) ++lb;
        const int h = T % SETS, n = T / SETS;
        auto &t = S.set[h].tile[n & 3];
        const int p0 = a.boff[lb] + (T0 + T - a.toff[lb]) * a.per, ncol = (min(a.boff[lb + 1], p0 + a.per) - p0) * a.rt;
        for (int g = 0; g < 4 / SETS && good; ++g) {
          if ((T * (4 / SETS) + g) % 3 != warp - kIbWarps - 1) continue;
          if (n >= 4) good = tc_waitw(smem_u32(&S.set[h].tfree[n & 3]), (uint32_t)(((n >> 2) - 1) & 1));
          if (!good) break;
          if (g == 0) {
            for (int e = lane; e < 2 * KP; e += 32) (e < KP ? t.eb[e] : t.ea[e - KP]) = a.exps[(size_t)lb * 2 * KP + e];
            if (lane == 0) {
              t.ncol = ncol;
              t.bucket = lb;
              t.pair0 = p0 - a.s0;
            }
          }
          const int c = g * 32 + lane;
          const IbRec rc = a.rec[p0 + min(c, ncol - 1) / a.rt];  // columns that are not there repeat the last
          const IbWords tw = ib_split_fraction(fixed(rc.t, 62));
          t.t[c] = make_int2(tw.h, tw.l);
          t.xoff[c] = rc.j * a.rt + min(c, ncol - 1) % a.rt;
          t.ph[0][c] = make_int4(1 << 30, 0, 0, 0);
          double pr = rc.c, pi = rc.s;
          for (int m = 1; m <= a.mmax; ++m) {
            const IbWords cw = ib_split_signed(fixed(pr, 61)), sw = ib_split_signed(fixed(pi, 61));
            t.ph[m][c] = make_int4(cw.h, cw.l, sw.h, sw.l);
            const double nr = pr * rc.c - pi * rc.s;
            pi = pr * rc.s + pi * rc.c;
            pr = nr;
          }
          __syncwarp();
          if (lane == 0) tc_arrive(smem_u32(&S.set[h].meta[n & 3]));
        }
      }
    }
    __syncwarp();
    __syncthreads();  // the registers come back from the other warps: none may ask for them before
    IB_SETMAXNREG(inc, 96);
  } else {
    IB_SETMAXNREG(inc, 104);
    // A thread owns a column (tensor-memory lane) and, of the four warps of its lanes, a quarter of the n2 and n1.
    const int sp = warp & 3, grp = warp >> 2;
    const int h = sp / (4 / SETS);                   // set
    const int c0w = sp % (4 / SETS) * 32, col = c0w + lane;  // column of the tile
    const int NS = (NT - h + SETS - 1) / SETS;       // the set's tiles
    auto &Q = S.set[h];
    const uint32_t lanes = tmem + ((uint32_t)(sp * 32) << 16);
    int ce = 0;           // exponent of the column
    uint32_t formed = 0;  // tiles with columns in these lanes
    // rotate the columns of the set's tile ti and cut them into digits
    auto form = [&](int ti) {
      auto &t = Q.tile[ti & 3];
      if (c0w < t.ncol) {
        constexpr int E = KP / 4;
        const int4 *xp = a.x + (size_t)t.xoff[col] * KP + grp * E;
        int4 xv[E];
        int xe[E], emax = 0;
#pragma unroll
        for (int q = 0; q < E; q += 4)
          *reinterpret_cast<int4 *>(xe + q) = __ldg(reinterpret_cast<const int4 *>(a.xe + (size_t)t.xoff[col] * KP + grp * E + q));
#pragma unroll
        for (int q = 0; q < E; ++q) xv[q] = __ldg(xp + q);
#pragma unroll
        for (int q = 0; q < E; ++q) {
          xe[q] += t.eb[grp * E + q] + 4096;
          emax = max(emax, xe[q]);
        }
        S.emax[grp][sp * 32 + lane] = emax;
        __syncwarp();
        if (lane == 0) tc_arrive(smem_u32(&S.quarters[sp]));
        good = good && tc_waitw(smem_u32(&S.quarters[sp]), formed & 1);
        ++formed;
        // |Re x|, |Im x| < 2^(ce - 4096 - 1022) under the column exponents
        ce = max(max(S.emax[0][sp * 32 + lane], S.emax[1][sp * 32 + lane]),
                 max(S.emax[2][sp * 32 + lane], S.emax[3][sp * 32 + lane]));
#pragma unroll
        for (int q4 = 0; q4 < E; q4 += 4) {
          uint32_t o[2][kIbDig][2];
#pragma unroll
          for (int q = 0; q < 4; q += 2) {
            long long u[2][2];
#pragma unroll
            for (int w = 0; w < 2; ++w) {
              const int n2 = grp * E + q4 + q + w, m = S.mofn[n2];
              const int4 x = xv[q4 + q + w];  // Re and Im in words of 2^-62 of their scale
              const int sh = min(ce - xe[q4 + q + w] + 9 - Num::UP, 63);
              // half of Re = c xr - s xi and Im = c xi + s xr
              int4 p = t.ph[m < 0 ? -m : m][col];
              if (m < 0) {
                p.z = -p.z;
                p.w = -p.w;
              }
              const long long mr = ib_mad(x.x, p.y, ib_mad(x.y, p.x, ib_mad(x.z, -p.w, ib_mad(x.w, -p.z, 0x40000000ll))));
              const long long mi = ib_mad(x.z, p.y, ib_mad(x.w, p.x, ib_mad(x.x, p.w, ib_mad(x.y, p.z, 0x40000000ll))));
              u[0][w] = ib_mad(x.z, p.x, ib_mad(x.x, p.z, mi >> 31)) >> sh;
              u[1][w] = ib_mad(x.x, p.x, ib_mad(x.z, -p.z, mr >> 31)) >> sh;
            }
#pragma unroll
            for (int w = 0; w < 2; ++w) {
              uint32_t dg[kIbDig];
              ib_digits<KP>(u[w][0], u[w][1], dg);
#pragma unroll
              for (int s = 0; s < kIbDig; ++s) o[w][s][q >> 1] = dg[s];
            }
          }
          // two columns of the chunk's Im part, then of its Re part
          const int c0 = ib_chunk<KP>(grp * E + q4) * 8 + (ib_place<KP>(grp * E + q4) >> 1);
#pragma unroll
          for (int w = 0; w < 2; ++w)
#pragma unroll
            for (int s = 0; s < kIbDig; ++s)
              tmem_st2(lanes + Sh::ACOL + s * KP + c0 + 4 * w, o[w][s][0], o[w][s][1]);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) tc_arrive(smem_u32(&Q.afull));
    };
    uint32_t buf = 0, par = 0;  // accumulator of the next job; parities of the set's next jobs in the two
    auto wait_job = [&]() {
      if (good) good = tc_waitw(smem_u32(&Q.dfull[buf]), (par >> buf) & 1);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    };
    auto release = [&]() {
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) tc_arrive(smem_u32(&Q.dempty[buf]));
      par ^= 1u << buf;
      if (BUFS == 2) buf ^= 1;
    };
    // the next job: block() gets eight at a time of this warp's 16 Re and 16 Im columns
    auto job = [&](auto &&block) {
      wait_job();
      const uint32_t src = lanes + buf * 128 + grp * 16;
#pragma unroll
      for (int h = 0; h < 32; h += 8) {
        float f[8];
        tmem_ld8(src + (h < 16 ? h : h - 16 + kIbRows), f);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (h == 24) release();
        block(h, f);
      }
    };
    for (int ti = 0; ti < NS && good; ++ti) {
      auto &t = Q.tile[ti & 3];
      good = tc_waitw(smem_u32(&Q.meta[ti & 3]), (uint32_t)((ti >> 2) & 1));
      if (!good) break;
      if (BUFS == 2) buf = (uint32_t)((ti * SETS + h) * passes * Num::JOBS) & 1;
      form(ti);  // every job of the set's last tile has been read: its operand is free
      for (int p = 0; p < passes && good; ++p) {
        const int n0 = p * PN + grp * WN;
        if (c0w >= t.ncol || n0 >= bs) {
          for (int k = 0; k < Num::JOBS; ++k) {
            wait_job();
            release();
          }
          continue;
        }
        // The digits in units of 2^-UNIT of the scales, least weights first. What is below 2^22 becomes an integer
        // by an FP32 addition of 1.5 2^23, whose exponent bits stay in the sum and are taken off it (OFFSET) below;
        // a warp that meets a larger sum converts.
        auto bits = [](float f) { return (unsigned)__float_as_int(f + kIbMagic); };
        auto ints = [&](float (&f)[8]) {
          float m = 0.f;
#pragma unroll
          for (int c = 0; c < 8; c += 2) asm("max.abs.f32 %0, %0, %1, %2;" : "+f"(m) : "f"(f[c]), "f"(f[c + 1]));
          if (__any_sync(kTcFull, m >= 4194304.f)) {
#pragma unroll
            for (int c = 0; c < 8; ++c) f[c] = __int_as_float(__float2int_rn(f[c]) + (int)kIbMagicBits);
          } else {
#pragma unroll
            for (int c = 0; c < 8; ++c) f[c] += kIbMagic;
          }
        };
        auto wide = [](float v, unsigned u, unsigned long long c) {
          return (unsigned long long)(unsigned)__float_as_int(v) * u + c;
        };
        float low[32];
        unsigned long long w[32];
#define IB_EACH(stmt) [&](int h, float (&f)[8]) { _Pragma("unroll") for (int c = 0; c < 8; ++c) { stmt; } }
#define IB_INTS(stmt) [&](int h, float (&f)[8]) { ints(f); _Pragma("unroll") for (int c = 0; c < 8; ++c) { stmt; } }
        if constexpr (KP == 32) {
          job(IB_EACH(low[h + c] = f[c] * 0x1p-15f));
          job(IB_EACH(low[h + c] = fmaf(f[c], 0x1p-6f, low[h + c])));
          job(IB_INTS(low[h + c] = __int_as_float((int)((unsigned)__float_as_int(f[c]) * 8u + bits(low[h + c])))));
          job(IB_INTS(w[h + c] = wide(f[c], 1u << 12, (unsigned)__float_as_int(low[h + c]))));
          job(IB_INTS(w[h + c] = wide(f[c], 1u << 21, w[h + c])));
          job(IB_INTS(w[h + c] = wide(f[c], 1u << 30, w[h + c])));
          job(IB_EACH(w[h + c] += (unsigned long long)(bits(f[c]) * 128u) << 32));
        } else {
          job(IB_EACH(low[h + c] = f[c] * 0x1p-16f));
          job(IB_EACH(low[h + c] = fmaf(f[c], 0x1p-8f, low[h + c])));
          job(IB_INTS(low[h + c] = __int_as_float((int)((unsigned)__float_as_int(f[c]) + bits(low[h + c])))));
          job(IB_INTS(w[h + c] = wide(f[c], 1u << 8, (unsigned)__float_as_int(low[h + c]))));
          job(IB_INTS(w[h + c] = wide(f[c], 1u << 16, w[h + c])));
          job(IB_INTS(w[h + c] = wide(f[c], 1u << 24, w[h + c])));
          job(IB_EACH(w[h + c] += (unsigned long long)bits(f[c]) << 32));
          job(IB_EACH(w[h + c] += (unsigned long long)(bits(f[c]) * 256u) << 32));
        }
#undef IB_EACH
#undef IB_INTS
        if (!good) break;
        const bool have = col < t.ncol;
        const int2 tw = t.t[col];
        const int cs = ce - 4096 - 1022 + 1 - Num::UNIT;  // scale of x, half of its rotation, units
        double2 *vo = a.V + (t.pair0 * a.rt + col) * bs;
#pragma unroll
        for (int s = 0; s < WN; ++s) {
          const int n = n0 + s;
          if (n >= bs) break;
          long long y[2];
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int c = NC - 1; c >= 0; --c) {
              const long long e = (long long)(w[16 * h + s * NC + c] - Num::OFFSET);
              y[h] = c == NC - 1 ? e : ib_mul(ib_split(y[h]), tw.x, tw.y, e);
            }
          const IbWords r = ib_split(y[0]), i = ib_split(y[1]);
          const int m = S.mofn[n];
          int4 ph = t.ph[m < 0 ? -m : m][col];
          if (m < 0) {
            ph.z = -ph.z;
            ph.w = -ph.w;
          }
          // e^{-i m phi} times the value: Re = c r + s i, Im = c i - s r
          const long long mr = ib_mad(r.h, ph.y, ib_mad(r.l, ph.x, ib_mad(i.h, ph.w, ib_mad(i.l, ph.z, 0x20000000ll))));
          const long long mi = ib_mad(i.h, ph.y, ib_mad(i.l, ph.x, ib_mad(r.h, -ph.w, ib_mad(r.l, -ph.z, 0x20000000ll))));
          const int e = cs + t.ea[n];
          double2 res = make_double2(ib_to_double(2 * ib_mad(r.h, ph.x, (long long)i.h * ph.z) + (mr >> 30), e),
                                     ib_to_double(2 * ib_mad(i.h, ph.x, (long long)r.h * -ph.z) + (mi >> 30), e));
          if (ce >= (1 << 20)) res.x = res.y = __longlong_as_double(0x7FF8000000000000ll);  // Inf or NaN in x
          if (have) vo[n] = res;
        }
      }
      __syncwarp();
      if (lane == 0) tc_arrive(smem_u32(&Q.tfree[ti & 3]));
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    IB_SETMAXNREG(dec, 96);
    __syncthreads();
  }
  if (!good && lane == 0) atomicExch(a.err, 1);
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

// ------------------------------------------------------------------ words of x
// Re and Im of every element in words of 2^-62 of a power-of-two scale of its own, and the scale's exponent field: the
// N pairs of an emitter share them.
template <int KP>
__global__ void __launch_bounds__(256) ib_words_kernel(const double2 *x, int n, int bs, int R, int r0, int rt, int4 *xw, int *xe) {
  const size_t q = (size_t)blockIdx.x * 256 + threadIdx.x;  // (j, r, n2)
  if (q >= (size_t)n * rt * KP) return;
  const int n2 = (int)(q % KP), r = (int)(q / KP % rt);
  const size_t j = q / ((size_t)KP * rt);
  int4 w = make_int4(0, 0, 0, 0);
  int f = 0;
  if (n2 < bs) {
    double2 v = x[(j * bs + n2) * R + r0 + r];
    f = max(ib_field(v.x), ib_field(v.y));
    const bool tiny = f < 64;  // a part of it may be subnormal: lifted by 2^128, its exponent below zero
    if (tiny) {
      v = make_double2(v.x * 0x1p128, v.y * 0x1p128);
      f = max(ib_field(v.x), ib_field(v.y));
    }
    const IbWords re = ib_split(ib_fixed<9>(v.x, f - ib_field(v.x))), im = ib_split(ib_fixed<9>(v.y, f - ib_field(v.y)));
    w = make_int4(re.h, re.l, im.h, im.l);
    f = f == 0 ? -(1 << 24) : f == 0x7FF ? 1 << 21 : tiny ? f - 128 : f;  // zero; Inf or NaN
  } else {
    f = -(1 << 24);
  }
  xw[q] = w;
  xe[q] = f;
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
  if (g < s.groups) {  // a whole warp (the width is a multiple of 32)
    const int j0 = (int)((long long)N * g / s.groups), j1 = (int)((long long)N * (g + 1) / s.groups);
    const int lane = threadIdx.x & 31;
    const unsigned *sl = s.slot + (size_t)i * N;
    const double2 *V = s.V + min(e, E - 1);
    double2 a = make_double2(0.0, 0.0);
    for (int j = j0; j < j1; j += 32) {
      const long long p = j + lane < j1 ? (long long)__ldg(sl + j + lane) - s.s0 : -1;
      unsigned m = __ballot_sync(kTcFull, p >= 0 && p < s.s1 - s.s0);
      // the pairs of this chunk among 32, several loads in flight; what is not in it costs no FP64 addition (64 cycles)
      auto take = [&](auto count) {
        constexpr int C = decltype(count)::value;
        double2 v[C];
#pragma unroll
        for (int q = 0; q < C; ++q) {
          v[q] = V[(size_t)__shfl_sync(kTcFull, (unsigned)p, __ffs(m) - 1) * E];
          m &= m - 1;
        }
#pragma unroll
        for (int q = 0; q < C; ++q) {
          a.x += v[q].x;
          a.y += v[q].y;
        }
      };
      while (__popc(m) >= 8) take(std::integral_constant<int, 8>());
      if (__popc(m) >= 4) take(std::integral_constant<int, 4>());
      if (__popc(m) >= 2) take(std::integral_constant<int, 2>());
      if (m) take(std::integral_constant<int, 1>());
    }
    if (e < E) part[(size_t)g * E + e] = a;
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
  ib_exponents<NC, KP>(C, bs, eb, ea);
  if (tid < KP) {
    exps[(size_t)b * 2 * KP + tid] = eb[tid];
    exps[(size_t)b * 2 * KP + KP + tid] = ea[tid];
  }
  unsigned char *out = B + (size_t)b * Sh::BBYTES;
  // one thread per row (n1, power) and pair of n2
  for (int e = tid; e < Sh::PASSES * kIbRows * KP / 2; e += blockDim.x) {
    const int row = e / (KP / 2), k = 2 * (e - row * (KP / 2));
    const int n1 = row / NC, c = row % NC;
    long long f[2][2];
    for (int w = 0; w < 2; ++w) {
      const int n2 = k + w;
      const bool in = n1 < bs && n2 < bs;
      const double2 v = in ? C[(size_t)c * bs2 + n2 * bs + n1] : make_double2(0.0, 0.0);
      const int s = in ? ea[n1] + eb[n2] + 1022 : 0;
      f[0][w] = ib_fixed<IbNumbers<KP>::UP>(v.x, s - ib_field(v.x));
      f[1][w] = ib_fixed<IbNumbers<KP>::UP>(v.y, s - ib_field(v.y));
    }
    const int pass = row / kIbRows, r = row % kIbRows;
    unsigned char *o = out + (size_t)pass * Sh::OPERAND + ib_chunk<KP>(k) * Sh::PLANE + (r >> 3) * 128 + (r & 7) * 16 +
                       ib_place<KP>(k) * 2;
    uint32_t dg[3][kIbDig];
    ib_digits<KP>(-f[1][0], -f[1][1], dg[0]);
    ib_digits<KP>(f[0][0], f[0][1], dg[1]);
    ib_digits<KP>(f[1][0], f[1][1], dg[2]);
    for (int h = 0; h < 3; ++h)
      for (int s = 0; s < kIbDig; ++s)
        *reinterpret_cast<uint32_t *>(o + (size_t)s * Sh::SLICE + h * (kIbRows * 16)) = dg[h][s];
  }
}

static constexpr int kIbMinParticles = 32;  // down to here ib_pays has been measured
static constexpr long long kIbMaxPairs = 1ll << 27;      // 4 GB of pair records
static constexpr size_t kIbMaxOperands = (size_t)32 << 30;  // bytes of the intervals' B operands

// padded blocksize
static int ib_kp(const sg_context *c) { return c->bs <= IbNumbers<32>::MAXB ? 32 : 48; }

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

void ib_drop(sg_context *c) {
  auto &P = c->ib;
  P.ready = P.digits_ready = P.halves_ready = P.captured = false;
  P.tiles.clear();
  P.rec.release();
  P.slot.release();
  P.ints.release();
  P.tmp.release();
  P.B.release();
  P.H.release();
  P.xh.release();
  P.top.release();
  P.V.release();
  P.acc.release();
  P.xw.release();
  P.xe.release();
}

void ib_drop_halves(sg_context *c) {
  auto &P = c->ib;
  if (!P.digits_ready) return ib_drop(c);
  P.halves_ready = false;
  P.H.release();
  P.xh.release();
}

bool ib_supported(const sg_context *c) {
  if (c->vol || c->kind < 0 || c->ib.refused || c->bs > IbNumbers<48>::MAXB) return false;
  const long long pairs = (long long)c->n * c->n;
  if (pairs > kIbMaxPairs || c->n < kIbMinParticles) return false;
  size_t operand = 0;
  ib_dispatch(c, [&](auto nc, auto kp) { operand = IbShape<decltype(nc)::value, decltype(kp)::value>::BBYTES; });
  if (std::min<size_t>(c->n_int, pairs) * operand > kIbMaxOperands) return false;
  const int mmax = ib_kp(c) == 32 ? IbNumbers<32>::MAXM : IbNumbers<48>::MAXM;
  for (int m : c->h_mofn)
    if (m > mmax || m < -mmax) return false;
  return true;
}

// Beyond it the batched operator is the faster one however fine the lookup: 400 spheres on a 0.5 nm grid 0.72 ms against
// 2.36, l_max = 1 0.70 against 0.90.
static constexpr int kIbSmall = 640;

void ib_count_pairs(sg_context *c, const double2 *pos) {
  auto &P = c->ib;
  P.h_counts.clear();
  P.pays.clear();
  const int n = c->n;
  if (n < kIbMinParticles || n > kIbSmall) return;
  std::vector<int> count(c->n_int, 0);
  auto interval = [&](double rho) { return std::max(0, std::min(c->n_int - 1, (int)((rho - c->rho_min) / c->res))); };
  count[interval(0.0)] += n;
  for (int i = 0; i < n; ++i)
    for (int j = i + 1; j < n; ++j) {
      const double dx = pos[i].x - pos[j].x, dy = pos[i].y - pos[j].y;
      count[interval(std::sqrt(dx * dx + dy * dy))] += 2;
    }
  for (int k : count)
    if (k) P.h_counts.push_back(k);
}

// pairs per tile, and the sets of warps, for rt right-hand sides: tiles(per) counts them
template <class F>
static int ib_sets(int rt, F &&tiles) {
  return 3 * tiles(kIbCols / 2 / rt) <= 4 * tiles(kIbCols / rt) ? 2 : 1;
}

// The batched operator's time goes by tiles, the per-receiver kernel's by pairs: few particles on a fine grid leave most
// tiles with one pair. Both times in microseconds from 1364 products of 32 to 400 particles (l_max 1 to 4, grids of 0.5
// to 5 nm, 1 to 16 right-hand sides), which they meet within a quarter. 32 spheres, 0.5 nm, linear: 51 us batched,
// 25 per receiver; 100 spheres, 0.5 nm, cubic: 329 and 257, 1 nm: 237 and 257, 5 nm: 89 and 234.
bool ib_pays(sg_context *c, int R) {
  auto &P = c->ib;
  if (c->n > kIbSmall) return true;
  for (const auto &p : P.pays)
    if (p.first == R) return p.second;
  const int bs = c->bs, wide = (bs + 31) / 32, most = ib_group(c, R);
  const int rows = kIbRows / c->ncoef, passes = (bs + rows - 1) / rows;
  const double size = ib_kp(c) == 32 ? 1.0 : 1.65;
  double batched = 0.0;
  for (int r0 = 0, rt; r0 < R; r0 += rt) {
    rt = std::min(most, R - r0);
    auto tiles = [&](int per) {
      long long t = 0;
      for (int k : P.h_counts) t += (k + per - 1) / per;
      return t;
    };
    const int sets = ib_sets(rt, tiles);
    const double tile = size * (sets == 2 ? 3.0 + 6.5 * passes : 4.0 + 6.5 * passes + 0.2 * bs);
    batched += 16.0 + 7.0 * passes * size + tile * tiles(kIbCols / sets / rt) / sm_count();
  }
  const double pairs = 1e-3 * c->n * c->n * 152 / sm_count();
  const double receiver = wide * (0.35 * c->n + pairs * (2.3 + 0.129 * bs * (c->ncoef - 1) + 0.286 * bs * R));
  const bool pays = receiver >= 0.95 * batched;
  P.pays.push_back({R, pays});
  return pays;
}

// Few allocations and one synchronisation: a first product is most of what a small system's program may ask for. The
// sort's buffers stay for the next plan unless they are large. 100 spheres, linear: first product 0.43 ms with an
// allocation of its own for every array and four synchronisations, 0.35 now, 0.20 on new particles of the same context
// (0.24 before; the per-receiver kernel 0.19 and 0.18); 1000 spheres 2.12 and 1.70 (13.5).
static constexpr size_t kIbKeep = (size_t)64 << 20;

void ib_plan(sg_context *c, cudaStream_t st) {
  auto &P = c->ib;
  if (P.ready) return;
  const int n = c->n, n_int = c->n_int, kp = ib_kp(c);
  const size_t np = (size_t)n * n;
  int bits = 1;
  while ((1 << bits) < n_int) ++bits;
  size_t bytes = 0;
  unsigned *none = nullptr;
  SG_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, bytes, none, none, none, none, np, 0, bits, st));
  const size_t part = (np * sizeof(unsigned) + 255) / 256 * 256, rest = (n_int * sizeof(int) + 255) / 256 * 256;
  P.take(P.tmp, 4 * part + rest + bytes);
  unsigned *keys = reinterpret_cast<unsigned *>(P.tmp.ptr), *keys2 = keys + part / 4, *vals = keys2 + part / 4,
           *vals2 = vals + part / 4;
  int *counts = reinterpret_cast<int *>(vals2 + part / 4);
  SG_CUDA(cudaMemsetAsync(counts, 0, n_int * sizeof(int), st));
  const unsigned grid = (unsigned)((np + 255) / 256);
  ib_keys_kernel<<<grid, 256, 0, st>>>(c->pos.ptr, n, c->rho_min, c->res, n_int, keys, vals, counts);
  SG_CUDA(cudaGetLastError());
  SG_CUDA(cub::DeviceRadixSort::SortPairs(reinterpret_cast<unsigned char *>(counts) + rest, bytes, keys, keys2, vals, vals2, np,
                                          0, bits, st));
  P.take(P.rec, np);
  P.take(P.slot, np);
  ib_records_kernel<<<grid, 256, 0, st>>>(c->pos.ptr, n, c->rho_min, c->res, n_int, vals2, P.rec.ptr, P.slot.ptr);
  SG_CUDA(cudaGetLastError());
  std::vector<int> cnt(n_int);
  SG_CUDA(cudaMemcpyAsync(cnt.data(), counts, n_int * sizeof(int), cudaMemcpyDeviceToHost, st));
  SG_CUDA(cudaStreamSynchronize(st));
  // intervals, first pairs, error flag (zero) and, filled with the operands, exponents
  P.h_ints.clear();
  P.h_boff.assign(1, 0);
  for (int k = 0; k < n_int; ++k)
    if (cnt[k] > 0) {
      P.h_ints.push_back(k);
      P.h_boff.push_back(P.h_boff.back() + cnt[k]);
    }
  P.nb = (int)P.h_ints.size();
  P.h_ints.insert(P.h_ints.end(), P.h_boff.begin(), P.h_boff.end());
  P.h_ints.push_back(0);
  P.take(P.ints, P.h_ints.size() + (size_t)P.nb * 2 * kp);
  P.bk = P.ints.ptr;
  P.boff = P.bk + P.nb;
  P.err = P.boff + P.nb + 1;
  P.exps = P.err + 1;
  SG_CUDA(cudaMemcpyAsync(P.ints.ptr, P.h_ints.data(), P.h_ints.size() * sizeof(int), cudaMemcpyHostToDevice, st));
  if (P.tmp.n > kIbKeep) P.tmp.release();
  P.tiles.clear();
  c->launches += 2;
  P.ready = true;
  P.digits_ready = P.halves_ready = false;
}

static void ib_digit_operands(sg_context *c, cudaStream_t st) {
  auto &P = c->ib;
  if (P.digits_ready) return;
  ib_dispatch(c, [&](auto nc, auto kp) {
    constexpr int NC = decltype(nc)::value, KP = decltype(kp)::value;
    P.take(P.B, (size_t)P.nb * IbShape<NC, KP>::BBYTES);
    ib_operand_kernel<NC, KP><<<P.nb, 256, 0, st>>>(c->coef64.ptr, P.bk, c->bs, P.B.ptr, P.exps);
  });
  SG_CUDA(cudaGetLastError());
  c->launches += 1;
  P.digits_ready = true;
}

void ib_enter(sg_context *c, cudaStream_t st) {
  auto &P = c->ib;
  if (capturing(st)) {  // a wait for the event would tie the graph to this one call; the host may wait in relaxed mode
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    SG_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
    const cudaError_t e = cudaEventSynchronize(P.done);
    SG_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
    SG_CUDA(e);
    P.captured = true;
    return;
  }
  if (!P.done) SG_CUDA(cudaEventCreateWithFlags(&P.done, cudaEventDisableTiming));
  else SG_CUDA(cudaStreamWaitEvent(st, P.done, 0));
}

void ib_leave(sg_context *c, cudaStream_t st) {
  if (!capturing(st)) SG_CUDA(cudaEventRecord(c->ib.done, st));
}

// The tiles for rt right-hand sides: first tile of every interval. Where 64 columns make hardly more tiles than 128,
// most are not half full and two sets of warps that overlap their tiles are faster: 100 spheres (1.00 times the tiles)
// 51 against 63 us, 220 (1.27) 108 against 117, 200 with the cubic lookup (1.25) 144 against 141, 301 (1.54) 165
// against 161, 1000 (1.8) 1140 against 1056.
sg_context::IbTiles &ib_tiles(sg_context *c, int rt, int sets, cudaStream_t st) {
  auto &P = c->ib;
  for (auto &t : P.tiles)
    if (t->rt == rt && t->asked == sets) return *t;
  auto t = std::make_unique<sg_context::IbTiles>();
  auto count = [&](int per) {
    long long n = 0;
    for (int b = 0; b < P.nb; ++b) n += (P.h_boff[b + 1] - P.h_boff[b] + per - 1) / per;
    return n;
  };
  t->rt = rt;
  t->asked = sets;
  t->sets = sets ? sets : ib_sets(rt, count);
  const int per = t->per = kIbCols / t->sets / rt;
  t->h_toff.assign(1, 0);
  for (int b = 0; b < P.nb; ++b)
    t->h_toff.push_back(t->h_toff.back() + (P.h_boff[b + 1] - P.h_boff[b] + per - 1) / per);
  P.take(t->toff, t->h_toff.size());
  SG_CUDA(cudaMemcpyAsync(t->toff.ptr, t->h_toff.data(), t->h_toff.size() * sizeof(int), cudaMemcpyHostToDevice, st));
  P.tiles.push_back(std::move(t));
  return *P.tiles.back();
}

bool ib_has_tiles(const sg_context *c, int rt, int sets) {
  for (const auto &t : c->ib.tiles)
    if (t->rt == rt && t->asked == sets) return true;
  return false;
}

// Right-hand sides at a time: their pairs share t and the phases and fill the tiles of a sparse interval, but every
// further chunk goes through the slots again. 16 of them, one / four / sixteen at a time: 301 spheres (0.07 GB of V a
// right-hand side) 2.90 / 1.76 / 1.45 ms, 1000 (0.5 GB) 23.7 / 20.9 / 20.6, 2000 (1.9 GB) 85.8 / 82.4 / 83.0, 4000
// (7.7 GB) 334 / 334 / 374.
int ib_group(const sg_context *c, int R) {
  const size_t row = (size_t)c->n * c->n * c->bs * sizeof(double2);
  return std::min(R, (int)std::min<size_t>(16, std::max<size_t>(1, 4 * c->ib.workspace / row)));
}

bool ib_prepared(const sg_context *c, int R) {
  const int most = ib_group(c, R);
  return c->ib.ready && c->ib.digits_ready && ib_has_tiles(c, most, 0) && (R % most == 0 || ib_has_tiles(c, R % most, 0));
}

template <int NC, int KP, int SETS>
static void ib_launch(const IbArgs &a, cudaStream_t st) {
  static bool attr_done[64] = {};
  constexpr int smem = (int)ib_smem<NC, KP, SETS>();
  if (first_on_device(attr_done))
    SG_CUDA(cudaFuncSetAttribute(ib_kernel<NC, KP, SETS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  ib_kernel<NC, KP, SETS><<<std::min(sm_count(), a.t1 - a.t0), kIbThreads, smem, st>>>(a);
  SG_CUDA(cudaGetLastError());
}

// y = M x or W x in FP64; returns the number of kernels launched
int launch_ibatch(sg_context *c, const double2 *x, double2 *y, int R, bool master, cudaStream_t st) {
  auto &P = c->ib;
  CallMemory mem(st);
  ib_enter(c, st);
  if (!mem.graph) {
    ib_plan(c, st);
    ib_digit_operands(c, st);
  }
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
  const int most = ib_group(c, R);
  double2 *acc = nullptr;
  for (int r0 = 0, rt; r0 < R; r0 += rt) {
    rt = std::min(most, R - r0);
    auto &tl = ib_tiles(c, rt, 0, st);
    const int per = tl.per;
    const size_t pair_bytes = (size_t)rt * bs * sizeof(double2);
    const int ntiles = tl.h_toff.back();
    const int chunk = (int)std::min<size_t>(ntiles, std::max<size_t>(1, c->ib.workspace / (pair_bytes * per)));
    double2 *V = ib_scratch(c, mem, P.V, (size_t)std::min<long long>((long long)chunk * per, (long long)c->n * c->n) * rt * bs);
    if (chunk < ntiles && !acc) acc = ib_scratch(c, mem, P.acc, (size_t)c->n * bs * R);
    auto first_pair = [&](int t) -> long long {  // first pair of tile t
      const int b = (int)(std::upper_bound(tl.h_toff.begin(), tl.h_toff.end(), t) - tl.h_toff.begin()) - 1;
      if (b >= P.nb) return (long long)c->n * c->n;
      return P.h_boff[b] + (long long)(t - tl.h_toff[b]) * per;
    };
    IbArgs a{};
    a.rec = P.rec.ptr;
    a.boff = P.boff;
    a.toff = tl.toff.ptr;
    a.B = P.B.ptr;
    a.exps = P.exps;
    const size_t words = (size_t)c->n * rt * ib_kp(c);
    int4 *xw = ib_scratch(c, mem, P.xw, words);
    int *xe = ib_scratch(c, mem, P.xe, words);
    (ib_kp(c) == 32 ? ib_words_kernel<32> : ib_words_kernel<48>)<<<(unsigned)((words + 255) / 256), 256, 0, st>>>(
        x, c->n, bs, R, r0, rt, xw, xe);
    SG_CUDA(cudaGetLastError());
    ++launched;
    a.x = xw;
    a.xe = xe;
    a.mofn = c->mofn.ptr;
    a.V = V;
    a.nb = P.nb;
    a.bs = bs;
    a.mmax = mmax;
    a.rt = rt;
    a.per = per;
    a.err = P.err;
    IbSum s{};
    s.V = V;
    s.slot = P.slot.ptr;
    s.acc = acc;
    s.err = P.err;
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
      ib_dispatch(c, [&](auto nc, auto kp) {
        if (tl.sets == 1) ib_launch<decltype(nc)::value, decltype(kp)::value, 1>(a, st);
        else ib_launch<decltype(nc)::value, decltype(kp)::value, 2>(a, st);
      });
      ib_sum_kernel<<<c->n, std::max(512, s.width), smem, st>>>(L, s);
      SG_CUDA(cudaGetLastError());
      launched += 2;
    }
  }
  ib_leave(c, st);
  return launched;
}

bool ib_check_error(sg_context *c, cudaStream_t st) {
  if (!c->ib.ready) return false;
  int e = 0;
  SG_CUDA(cudaMemcpyAsync(&e, c->ib.err, sizeof(int), cudaMemcpyDeviceToHost, st));
  SG_CUDA(cudaStreamSynchronize(st));
  if (e) SG_CUDA(cudaMemsetAsync(c->ib.err, 0, sizeof(int), st));
  return e != 0;
}

}  // namespace sg

size_t sg_context::Ib::bytes() const {
  size_t n = rec.n * sizeof(sg::IbRec) + (slot.n + ints.n + top.n + xe.n) * 4 + tmp.n + B.n + H.n +
             xh.n * sizeof(float2) + (V.n + acc.n) * sizeof(double2) + xw.n * sizeof(int4);
  for (const auto &t : tiles) n += t->toff.n * 4;
  return n;
}
