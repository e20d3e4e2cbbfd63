// Interval-batched FP32 coupling operator on the tensor cores, for many right-hand sides.
//
// The same grouping as the FP64 form (sg_ibatch.cu): all pairs of a lookup interval share its coefficient matrices,
// W_ij = D(phi)^H (sum_c t^c C_{k,c}) D(phi), so that one small matrix product per interval replaces the interpolation
// of every pair's block, and the coefficients are read once per interval instead of once per pair. Here the operands
// are split into two FP16 parts (11 bits each) under power-of-two scales, and three of the four products are summed
// in one FP32 accumulator: hi lo, lo hi, hi hi. The scales leave 2^14 as the largest element, so that an element keeps
// both parts down to 2^-28 of it. Rotations, powers of t and the sums over the pairs are FP32.
//
// One CTA per SM walks a contiguous range of tiles of up to 128 complex columns (pairs x right-hand sides) of one
// interval. Even and odd tiles belong to two sets of eight warps that run half a tile apart: a set rotates x_j, splits
// it and writes the A operand (a lane per column, K = 2 blocksize: Im and Re) to tensor memory, waits for the products
// (one accumulator of 64 Re and 64 Im columns per set and pass), combines the powers of t, rotates back and adds the
// contribution to y_i with vector atomics (in any order: the last bits of a product differ from run to run; with many
// particles in chunks of tiles, ih_chunks). One thread issues the MMAs against the interval's B operand in shared memory
// (rows -Im C, Re C, Im C as in the FP64 form); three warps prepare the tiles' t and phases ahead.
//
// Every wait is bounded; a wait that runs out sets the error flag, and all roles leave.
//
// What bounds it: each set's own chain. 1000 spheres, 16 right-hand sides: 60% of the issue slots, 36% of the tensor core;
// the schedulers' five warps wait for x_j and for the set's products (2000 spheres: 6.8 of 7.2 ms without the atomics, 8.6
// against 9.4 without two thirds of the MMAs in a first form whose scales were two factors per element; fetching the next
// tile's x ahead costs more registers than it hides, 7.56). Four powers of t times three products make 14.5 ms of MMAs of
// 1500 spheres with l_max 4 and 64 right-hand sides. Against the pair-symmetric 3xTF32 kernel: 2000 spheres, cubic, 16:
// 13.6 -> 7.28 ms, error of x - T W x 4.5e-7 -> 1.2e-7; film of 4001, linear, 16: 45.9 -> 24.1 ms, 2.7e-7 -> 7.3e-8;
// against the one-directional one, which repeats exactly: 1500 spheres, l_max 4, 64: 33.6 -> 31.0 ms, 8.3e-7 -> 1.4e-7.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "sg_ibatch.h"
#include "sg_internal.h"
#include "sg_tcgen05.h"

namespace sg {

static constexpr int kIhWarps = 16;  // two sets of eight; one of four more issues
static constexpr int kIhThreads = 32 * (kIhWarps + 4);
static constexpr int kIhCols = 128;  // complex columns per tile
static constexpr int kIhRows = 64;   // (n1, power of t) per pass
static constexpr int kIhUp = 14;     // the largest element of an operand is in [2^13, 2^14]

// The block is launched with 96 registers a thread (20 warps); its 61440 are split 512 x 104 + 128 x 64.
#define IH_SETMAXNREG(dir, n) asm volatile("setmaxnreg." #dir ".sync.aligned.u32 " #n ";")

template <int NC, int KP>
struct IhShape {
  static constexpr int KC = KP / 8;                  // chunks of eight n2: one K = 16 step of (Im u, Re u)
  static constexpr int PLANE = 3 * kIhRows * 16;     // bytes of a chunk of B: rows of -Im C, Re C, Im C
  static constexpr int PART = KC * PLANE;            // bytes of the hi or lo part of a pass of B
  static constexpr int OPERAND = 2 * PART;
  static constexpr int PN = kIhRows / NC;            // n1 per pass
  static constexpr int PASSES = (KP + PN - 1) / PN;  // at most
  static constexpr int BBYTES = PASSES * OPERAND;
  static constexpr int NB = KP == 32 ? 2 : 1;        // B operands in shared memory
  static constexpr int MAXM = KP == 32 ? 3 : 4;
  static constexpr int ACOL = 256;                   // first tensor-memory column of A: 2 KP columns per set
  static_assert(ACOL + 4 * KP <= 512, "tensor memory");
};

template <int KP>
struct IhSmem {
  struct Tile {
    float2 ph[KP == 32 ? 7 : 9][kIhCols];  // cos, sin of m phi per pair, from m = -3 or -4
    float fe[KP], fa[KP];                  // column scales under their largest 2^E0; row scales times 2^(E0 - 14)
    float t[kIhCols];
    int j[kIhCols], i[kIhCols];
    int ncol, bucket;
  };
  struct Set {
    Tile tile[4];
    int big[2][kIhCols];  // largest |Re|, |Im| of a column's halves, as bits
    uint64_t dfull, dempty, afull, meta[4], tfree[4], halves[4];
  } set[2];
  uint64_t bfull[2], done;
  int mrow[KP];  // row of the phase table of n, times its length
  uint32_t tmem;
};
template <int NC, int KP>
constexpr size_t ih_smem() {
  return (size_t)IhShape<NC, KP>::NB * IhShape<NC, KP>::BBYTES + (sizeof(IhSmem<KP>) + 127) / 128 * 128;
}
static_assert(ih_smem<2, 32>() <= kTcSmemBudget && ih_smem<4, 32>() <= kTcSmemBudget && ih_smem<2, 48>() <= kTcSmemBudget &&
                  ih_smem<4, 48>() <= kTcSmemBudget,
              "shared memory");

struct IhArgs {
  const IbRec *rec;
  const int *boff, *toff;
  const unsigned char *B;
  const int *exps;
  const float2 *x;  // [N][KP][rt]
  const int *mofn;
  float2 *y;        // [N][bs][R]
  int nb, bs, mmax, R, r0, rt, per, t0, t1;  // tiles [t0, t1)
  int *err;
};

template <bool ACC, int AO, int BO>
__device__ __forceinline__ void ih_mma(uint32_t dst, uint32_t a, uint32_t b, uint32_t hi, uint32_t idesc) {
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

// hi lo, lo hi, hi hi: the small products first
template <int NC, int KP, int P = 0, int K = 0>
__device__ __forceinline__ void ih_issue(uint32_t dst, uint32_t a, uint32_t b, uint32_t hi, uint32_t idesc) {
  using Sh = IhShape<NC, KP>;
  if constexpr (K == Sh::KC) {
    ih_issue<NC, KP, P + 1, 0>(dst, a, b, hi, idesc);
  } else if constexpr (P < 3) {
    constexpr int PA = P == 1 ? 1 : 0, PB = P == 0 ? 1 : 0;
    ih_mma<(P != 0 || K != 0), PA * KP + K * 8, PB * Sh::PART + K * Sh::PLANE>(dst, a, b, hi, idesc);
    ih_issue<NC, KP, P, K + 1>(dst, a, b, hi, idesc);
  }
}

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]), "r"(v[1]),
               "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}

// 2^e, zero below the normal range and Inf above it
__device__ __forceinline__ float ih_pow2(int e) { return e < -126 ? 0.f : __int_as_float((min(e, 128) + 127) << 23); }

// two floats as packed FP16 parts
__device__ __forceinline__ void ih_split(float a, float b, uint32_t &hi, uint32_t &lo) {
  const __half2 h = __floats2half2_rn(a, b);
  const float2 f = __half22float2(h);
  const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
  hi = *reinterpret_cast<const uint32_t *>(&h);
  lo = *reinterpret_cast<const uint32_t *>(&l);
}

template <int NC, int KP>
__global__ void __launch_bounds__(kIhThreads, 1) ih_kernel(const IhArgs a) {
  using Sh = IhShape<NC, KP>;
  using Sm = IhSmem<KP>;
  constexpr int PN = Sh::PN, NB = Sh::NB;
  extern __shared__ __align__(1024) unsigned char ih_raw[];
  unsigned char *Bs = ih_raw;
  Sm &S = *reinterpret_cast<Sm *>(Bs + NB * Sh::BBYTES);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int bs = a.bs;
  const int ntiles = a.t1 - a.t0;
  const int T0 = a.t0 + (int)((long long)ntiles * blockIdx.x / gridDim.x);
  const int NT = a.t0 + (int)((long long)ntiles * (blockIdx.x + 1) / gridDim.x) - T0;  // this CTA's tiles
  const int passes = (bs + PN - 1) / PN;

  if (tid < KP) S.mrow[tid] = ((tid < bs ? a.mofn[tid] : 0) + Sh::MAXM) * kIhCols;
  if (tid == 0) {
    auto init = [](uint64_t *b, int n) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(n) : "memory");
    };
    for (int h = 0; h < 2; ++h) {
      init(&S.set[h].dfull, 1);
      init(&S.set[h].dempty, kIhWarps / 2);
      init(&S.set[h].afull, kIhWarps / 2);
      for (int b = 0; b < 4; ++b) {
        init(&S.set[h].meta[b], 1);
        init(&S.set[h].tfree[b], kIhWarps / 2);
        init(&S.set[h].halves[b], 2);
      }
      init(&S.bfull[h], 1);
    }
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

  if (warp >= kIhWarps) {
    IH_SETMAXNREG(dec, 64);
    // ---------------------------------------------------------------- issue
    if (warp == kIhWarps && lane == 0) {
      const uint32_t idesc = (1u << 4) | ((uint32_t)(128 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);  // F16 in, F32 out
      // B: core matrices adjacent in rows 128 bytes apart, in K 64 rows, from -Im C | Re C to Re C | Im C
      const uint32_t blo = ((smem_u32(Bs) >> 4) & 0x3FFFu) | (uint32_t)((kIhRows * 16) >> 4) << 16;
      const uint32_t bhi = (128u >> 4) | (1u << 14);
      uint32_t jobs[2] = {0, 0};       // issued per set
      int held[2] = {-1, -1};          // intervals in the places of B
      uint32_t loads[2] = {0, 0}, landed[2] = {0, 0};
      // every MMA issued so far has completed
      auto finished = [&]() {
        bool ok = true;
        for (int h = 0; h < 2; ++h)
          if (ok && jobs[h] > 0) ok = tc_wait1(smem_u32(&S.set[h].dfull), (jobs[h] - 1) & 1);
        return ok;
      };
      // the place of a bucket, loaded into `place` if it is in none
      auto fetch = [&](int bucket, int place) {
        for (int q = 0; q < NB; ++q)
          if (held[q] == bucket) return q;
        good = good && finished();
        if (!good) return place;
        const uint32_t bar = smem_u32(&S.bfull[place]), bytes = (uint32_t)(passes * Sh::OPERAND);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                smem_u32(Bs) + place * Sh::BBYTES),
            "l"(a.B + (size_t)bucket * Sh::BBYTES), "r"(bytes), "r"(bar)
            : "memory");
        held[place] = bucket;
        ++loads[place];
        return place;
      };
      auto arrived = [&](int place) {
        if (landed[place] == loads[place]) return true;
        landed[place] = loads[place];
        return tc_wait1(smem_u32(&S.bfull[place]), (loads[place] - 1) & 1);
      };
      auto job = [&](int T, int p, int place) {
        if (!good) return;
        const int h = T & 1, n = T >> 1;
        if (p == 0) good = arrived(place) && tc_wait1(smem_u32(&S.set[h].afull), (uint32_t)(n & 1));
        if (good && jobs[h] > 0) good = tc_wait1(smem_u32(&S.set[h].dempty), (jobs[h] - 1) & 1);
        if (!good) return;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        ih_issue<NC, KP>(tmem + h * 128, tmem + Sh::ACOL + h * 2 * KP,
                         blo + (uint32_t)((place * Sh::BBYTES + p * Sh::OPERAND) >> 4), bhi, idesc);
        tc_commit(smem_u32(&S.set[h].dfull));
        ++jobs[h];
      };
      int last = 0;  // place used last
      for (int T = 0; T < NT && good; T += 2) {
        int bucket[2] = {0, 0};
        const int m = min(2, NT - T);
        for (int q = 0; q < m && good; ++q) {
          good = tc_wait1(smem_u32(&S.set[q].meta[(T >> 1) & 3]), (uint32_t)((T >> 3) & 1));
          if (good) bucket[q] = S.set[q].tile[(T >> 1) & 3].bucket;
        }
        if (!good) break;
        if (m == 2 && (NB == 2 || bucket[0] == bucket[1])) {
          const int first = fetch(bucket[0], NB == 2 ? last ^ 1 : 0);
          const int second = fetch(bucket[1], NB == 2 ? first ^ 1 : 0);
          for (int p = 0; p < passes; ++p) {
            job(T, p, first);
            job(T + 1, p, second);
          }
          last = second;
        } else {
          for (int q = 0; q < m; ++q) {
            last = fetch(bucket[q], NB == 2 ? last ^ 1 : 0);
            for (int p = 0; p < passes; ++p) job(T + q, p, last);
          }
        }
      }
      // nothing of this CTA may be in flight when its memory is given back
      tc_commit(smem_u32(&S.done));
      if (!tc_wait1(smem_u32(&S.done), 0u)) good = false;
      for (int q = 0; q < NB; ++q)
        if (!arrived(q)) good = false;
    }
    __syncwarp();
    // ---------------------------------------------------------------- look ahead: every third tile
    if (warp > kIhWarps) {
      int lb = 0;  // interval of the tile: the last one whose first tile is not behind it
      for (int len = a.nb; len > 1;) {
        const int step = (len + 31) / 32, q = lane * step;
        const unsigned hit = __ballot_sync(kTcFull, q < len && a.toff[lb + min(q, len - 1)] <= T0);
        const int o = (__popc(hit) - 1) * step;
        lb += o;
        len = min(step, len - o);
      }
      for (int T = warp - kIhWarps - 1; T < NT && good; T += 3) {
        while (T0 + T >= a.toff[lb + 1]) ++lb;
        const int h = T & 1, n = T >> 1;
        auto &t = S.set[h].tile[n & 3];
        const int p0 = a.boff[lb] + (T0 + T - a.toff[lb]) * a.per, np = min(a.boff[lb + 1] - p0, a.per);
        if (n >= 4) good = tc_waitw(smem_u32(&S.set[h].tfree[n & 3]), (uint32_t)(((n >> 2) - 1) & 1));
        if (!good) break;
        const int *ex = a.exps + (size_t)lb * 2 * KP;
        int e0 = -(1 << 20);
        for (int e = lane; e < bs; e += 32) e0 = max(e0, ex[e]);
        e0 = __reduce_max_sync(kTcFull, e0);
        for (int e = lane; e < KP; e += 32) {
          t.fe[e] = ih_pow2(ex[e] - e0);
          t.fa[e] = ih_pow2(ex[KP + e] + e0 - kIhUp);
        }
        if (lane == 0) {
          t.ncol = np * a.rt;
          t.bucket = lb;
        }
        for (int c = lane; c < np; c += 32) {
          const IbRec rc = a.rec[p0 + c];
          t.t[c] = (float)rc.t;
          t.j[c] = rc.j;
          t.i[c] = rc.i;
          t.ph[Sh::MAXM][c] = make_float2(1.f, 0.f);
          double pr = rc.c, pi = rc.s;
          for (int m = 1; m <= a.mmax; ++m) {
            t.ph[Sh::MAXM + m][c] = make_float2((float)pr, (float)pi);
            t.ph[Sh::MAXM - m][c] = make_float2((float)pr, -(float)pi);
            const double nr = pr * rc.c - pi * rc.s;
            pi = pr * rc.s + pi * rc.c;
            pr = nr;
          }
        }
        __syncwarp();
        if (lane == 0) tc_arrive(smem_u32(&S.set[h].meta[n & 3]));
      }
    }
    __syncwarp();
    __syncthreads();  // the registers come back from the other warps: none may ask for them before
    IH_SETMAXNREG(inc, 96);
  } else {
    IH_SETMAXNREG(inc, 104);
    // A thread owns a column (tensor-memory lane) and half of the n2 and of a pass's n1.
    const int h = warp >> 3, sp = warp & 3, half = (warp >> 2) & 1, col = sp * 32 + lane;
    const int pair = col / a.rt, rr = col - pair * a.rt;
    const int NS = (NT - h + 1) / 2;  // the set's tiles
    auto &Q = S.set[h];
    const uint32_t lanes = tmem + ((uint32_t)(sp * 32) << 16);
    const uint32_t acc = lanes + h * 128, aop = lanes + Sh::ACOL + h * 2 * KP;
    uint32_t formed = 0, job = 0;
    for (int n = 0; n < NS && good; ++n) {
      auto &t = Q.tile[n & 3];
      good = tc_waitw(smem_u32(&Q.meta[n & 3]), (uint32_t)((n >> 2) & 1));
      if (!good) break;
      const int ncol = t.ncol;
      const bool active = sp * 32 < ncol;
      const int pc = min(pair, ncol / a.rt - 1);  // columns that are not there repeat the last pair
      const float2 *phase = &t.ph[0][pc];
      float gc = 0.f;     // scale of the column's results
      bool tiny = false;  // a column below 2^-90 is lifted by 2^64 first
      if (active) {
        constexpr int E = KP / 2;
        const float2 *xp = a.x + ((size_t)t.j[pc] * KP + half * E) * a.rt + min(rr, a.rt - 1);
        float2 xv[E];
#pragma unroll
        for (int q = 0; q < E; ++q) xv[q] = __ldg(xp + (size_t)q * a.rt);
        float big = 0.f;  // NaN if there is one
#pragma unroll
        for (int q = 0; q < E; ++q) {
          const float f = t.fe[half * E + q];
          xv[q].x *= f;
          xv[q].y *= f;
          asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(big) : "f"(xv[q].x), "f"(xv[q].y));
        }
        Q.big[half][col] = __float_as_int(big) & 0x7FFFFFFF;
        __syncwarp();
        if (lane == 0) tc_arrive(smem_u32(&Q.halves[sp]));
        good = good && tc_waitw(smem_u32(&Q.halves[sp]), formed & 1);
        ++formed;
        int top = max(Q.big[0][col], Q.big[1][col]);  // bits: NaN above Inf above the rest
        tiny = top < (37 << 23) && top != 0;
        if (__any_sync(kTcFull, tiny)) {
          const float lift = tiny ? 0x1p64f : 1.f;
          top = __float_as_int(__int_as_float(top) * lift);
#pragma unroll
          for (int q = 0; q < E; ++q) {
            xv[q].x *= lift;
            xv[q].y *= lift;
          }
        }
        const int e = max((top >> 23) - 126, -100);  // |x| < 2^e under the column scales (0: any)
        const float fc = ih_pow2(kIhUp - e);
        gc = top >= 0x7F800000 ? __int_as_float(0x7FC00000) : ih_pow2(e - kIhUp);  // Inf or NaN in x: NaN
#pragma unroll
        for (int k = 0; k < E / 8; ++k) {
          uint32_t hi[8], lo[8];  // four words of Im parts, four of Re parts
#pragma unroll
          for (int q = 0; q < 8; q += 2) {
            float u[2][2];
#pragma unroll
            for (int w = 0; w < 2; ++w) {
              const float2 x = xv[k * 8 + q + w], p = phase[S.mrow[half * E + k * 8 + q + w]];
              const float xr = x.x * fc, xi = x.y * fc;
              u[0][w] = fmaf(xr, p.y, xi * p.x);
              u[1][w] = fmaf(-xi, p.y, xr * p.x);
            }
            ih_split(u[0][0], u[0][1], hi[q >> 1], lo[q >> 1]);
            ih_split(u[1][0], u[1][1], hi[4 + (q >> 1)], lo[4 + (q >> 1)]);
          }
          const uint32_t c0 = aop + (half * (E / 8) + k) * 8;
          tmem_st8(c0, hi);
          tmem_st8(c0 + KP, lo);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) tc_arrive(smem_u32(&Q.afull));
      for (int p = 0; p < passes; ++p, ++job) {
        if (good) good = tc_waitw(smem_u32(&Q.dfull), job & 1);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int n0 = p * PN + half * (PN / 2);
        const bool work = active && n0 < bs;
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          float dr[16], di[16];
          if (work) {
            tmem_ld16(acc + half * 32 + g * 16, dr);
            tmem_ld16(acc + kIhRows + half * 32 + g * 16, di);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          }
          if (g == 1) {
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) tc_arrive(smem_u32(&Q.dempty));
          }
          if (!work) continue;
          const float tt = t.t[pc];
          float2 *yo = a.y + (size_t)t.i[pc] * bs * a.R + a.r0 + rr;
#pragma unroll
          for (int s = 0; s < 16 / NC; ++s) {
            const int n1 = n0 + g * (16 / NC) + s;
            if (n1 >= bs) break;
            float yr = dr[s * NC + NC - 1], yi = di[s * NC + NC - 1];
#pragma unroll
            for (int c = NC - 2; c >= 0; --c) {
              yr = fmaf(yr, tt, dr[s * NC + c]);
              yi = fmaf(yi, tt, di[s * NC + c]);
            }
            const float2 ph = phase[S.mrow[n1]];
            const float f = gc * t.fa[n1];
            // e^{-i m phi} times the value
            float2 v = make_float2(fmaf(yi, ph.y, yr * ph.x) * f, fmaf(-yr, ph.y, yi * ph.x) * f);
            if (tiny) v = make_float2(v.x * 0x1p-64f, v.y * 0x1p-64f);
            if (good && col < ncol) atomicAdd(yo + (size_t)n1 * a.R, v);
          }
        }
      }
      __syncwarp();
      if (lane == 0) tc_arrive(smem_u32(&Q.tfree[n & 3]));
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    IH_SETMAXNREG(dec, 96);
    __syncthreads();
  }
  if (!good && lane == 0) atomicExch(a.err, 1);
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

// largest exponent field of every right-hand side: the sums over the pairs, whose atomics flush subnormals, stay in the
// middle of the FP32 range for x of any magnitude
__global__ void __launch_bounds__(256) ih_top_kernel(const double2 *x, size_t rows, int R, int *top) {
  __shared__ int m[256];  // R <= 256
  m[threadIdx.x] = 0;
  __syncthreads();
  const size_t total = rows * R;
  for (size_t e = (size_t)blockIdx.x * 256 + threadIdx.x; e < total; e += (size_t)gridDim.x * 256) {
    const double2 d = x[e];
    const int f = max(ib_field(d.x), ib_field(d.y));
    if (f < 0x7FF) atomicMax(&m[e % R], f);
  }
  __syncthreads();
  if (threadIdx.x < R && m[threadIdx.x] > 0) atomicMax(&top[threadIdx.x], m[threadIdx.x]);
}

// FP32 copy of x under its scale, [N][KP][rt], zero beyond the block
__global__ void __launch_bounds__(256) ih_copy_kernel(const double2 *x, int n, int bs, int kp, int R, int r0, int rt,
                                                      const int *top, float2 *o) {
  const size_t q = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (q >= (size_t)n * kp * rt) return;
  const int r = (int)(q % rt), n2 = (int)(q / rt % kp);
  const size_t j = q / ((size_t)kp * rt);
  float2 v = make_float2(0.f, 0.f);
  if (n2 < bs) {
    const double2 d = x[(j * bs + n2) * R + r0 + r];
    const double s = fp32_scale(top[r0 + r]);
    v = make_float2((float)(d.x * s), (float)(d.y * s));
  }
  o[q] = v;
}

// FP32 sums of a chunk of pairs, columns r0 .. r0 + rt of R: into the FP64 totals, and zero again; the last chunk
// leaves the total in their place
__global__ void __launch_bounds__(256) ih_fold_kernel(float2 *y, double2 *total, size_t rows, int R, int r0, int rt, int first, int last) {
  const size_t q = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (q >= rows * rt) return;
  const size_t e = q / rt * R + r0 + q % rt;
  const float2 v = y[e];
  double2 s = make_double2(v.x, v.y);
  if (!first) {
    const double2 o = total[e];
    s = make_double2(s.x + o.x, s.y + o.y);
  }
  if (!last) total[e] = s;
  y[e] = last ? make_float2((float)s.x, (float)s.y) : make_float2(0.f, 0.f);
}

// B operand and exponents of one non-empty interval per block
template <int NC, int KP>
__global__ void __launch_bounds__(256) ih_operand_kernel(const double2 *coef, const int *bk, int bs, unsigned char *B, int *exps) {
  using Sh = IhShape<NC, KP>;
  __shared__ int eb[KP], ea[KP];
  const int tid = threadIdx.x, b = blockIdx.x, bs2 = bs * bs;
  const double2 *C = coef + (size_t)bk[b] * NC * bs2;
  ib_exponents<NC, KP>(C, bs, eb, ea);
  if (tid < KP) {
    exps[(size_t)b * 2 * KP + tid] = eb[tid];
    exps[(size_t)b * 2 * KP + KP + tid] = ea[tid];
  }
  unsigned char *out = B + (size_t)b * Sh::BBYTES;
  for (int e = tid; e < Sh::PASSES * kIhRows * KP; e += blockDim.x) {
    const int row = e / KP, n2 = e - row * KP, n1 = row / NC, c = row % NC;
    double2 v = make_double2(0.0, 0.0);
    if (n1 < bs && n2 < bs) {
      v = C[(size_t)c * bs2 + n2 * bs + n1];
      v.x = scalbn(v.x, kIhUp - ea[n1] - eb[n2]);
      v.y = scalbn(v.y, kIhUp - ea[n1] - eb[n2]);
    }
    const int pass = row / kIhRows, r = row % kIhRows;
    unsigned char *o = out + (size_t)pass * Sh::OPERAND + (n2 >> 3) * Sh::PLANE + (r >> 3) * 128 + (r & 7) * 16 + (n2 & 7) * 2;
    const double parts[3] = {-v.y, v.x, v.y};
    for (int h = 0; h < 3; ++h) {
      const __half hi = __double2half(parts[h]), lo = __double2half(parts[h] - (double)__half2float(hi));
      *reinterpret_cast<__half *>(o + h * (kIhRows * 16)) = hi;
      *reinterpret_cast<__half *>(o + Sh::PART + h * (kIhRows * 16)) = lo;
    }
  }
}

static constexpr size_t kIhMaxOperands = (size_t)16 << 30;

// Pairs of a receiver that are added one after the other in FP32, on average. Larger systems run in chunks of tiles whose
// sums are added in FP64, for two reasons. The error of n such roundings grows with n: films of 2000 / 4001 / 10000
// spheres 9.1e-7 / 1.3e-6 / 2.1e-6 in one chunk (the pair-symmetric tensor-core kernel: 1.7e-6), now 4.4e-7 / 4.6e-7 /
// 3.4e-7. And their order differs from product to product, so that the residual of a solve does not fall below what it
// changes, which a film multiplies by five: with 2.3e-7 (1024 terms) 10000 spheres stood at 1.2e-6 before the correction's
// 1e-6 for 302 to 362 iterations, with 1.4e-7 it takes 185. Every chunk costs a launch, a last wave and a pass over the
// sums: 7.26 ms instead of 7.17 with 2000 spheres, cubic, 24.1 instead of 23.8 with 4001, 152.1 instead of 149.0 with
// 10000. From 5000 particles on a chunk is long enough to halve the terms for 1%, which keeps what changes below 1.5e-7.
static int ih_chunks(int n) { return (n + (n > 5000 ? 255 : 511)) / (n > 5000 ? 256 : 512); }

template <class F>
static void ih_dispatch(const sg_context *c, F &&f) {
  std::integral_constant<int, 2> two;
  std::integral_constant<int, 4> four;
  std::integral_constant<int, 32> small;
  std::integral_constant<int, 48> large;
  if (c->bs <= 32) {
    if (c->ncoef == 2) f(two, small);
    else f(four, small);
  } else {
    if (c->ncoef == 2) f(two, large);
    else f(four, large);
  }
}

bool ib32_supported(const sg_context *c, int R) {
  // the FP64 form's plan (and, with its operands' padded size, its exponents) must apply
  if (R < 16 || !ib_supported(c) || (c->bs > 30 && c->bs <= 32)) return false;
  size_t operand = 0;
  ih_dispatch(c, [&](auto nc, auto kp) { operand = IhShape<decltype(nc)::value, decltype(kp)::value>::BBYTES; });
  return std::min<size_t>(c->n_int, (size_t)c->n * c->n) * operand <= kIhMaxOperands;
}

bool ib32_prepared(const sg_context *c, int R) {
  return c->ib.ready && c->ib.halves_ready && ib_has_tiles(c, 16, 1) && (R % 16 == 0 || ib_has_tiles(c, R % 16, 1));
}

// y = M x or W x in FP32; returns the number of kernels launched
int launch_ibatch32(sg_context *c, const double2 *x, double2 *y, int R, bool master, cudaStream_t st) {
  auto &P = c->ib;
  CallMemory mem(st);
  ib_enter(c, st);
  if (!mem.graph) ib_plan(c, st);
  const int bs = c->bs, kp = bs <= 32 ? 32 : 48;
  int launched = 0;
  if (!P.halves_ready) {
    ih_dispatch(c, [&](auto nc, auto kpc) {
      constexpr int NC = decltype(nc)::value, KP = decltype(kpc)::value;
      P.take(P.H, (size_t)P.nb * IhShape<NC, KP>::BBYTES);
      ih_operand_kernel<NC, KP><<<P.nb, 256, 0, st>>>(c->coef64.ptr, P.bk, bs, P.H.ptr, P.exps);
    });
    SG_CUDA(cudaGetLastError());
    ++launched;
    P.halves_ready = true;
  }
  const size_t len = (size_t)c->n * bs * R;
  float2 *yacc = mem.get(c->sym_yacc, len);
  SG_CUDA(cudaMemsetAsync(yacc, 0, len * sizeof(float2), st));
  int *top = ib_scratch(c, mem, P.top, 256);
  SG_CUDA(cudaMemsetAsync(top, 0, R * sizeof(int), st));
  const size_t rows = (size_t)c->n * bs;
  ih_top_kernel<<<(unsigned)std::min<size_t>((rows * R + 2047) / 2048, (size_t)sm_count() * 4), 256, 0, st>>>(x, rows, R, top);
  SG_CUDA(cudaGetLastError());
  ++launched;
  IhArgs a{};
  a.rec = P.rec.ptr;
  a.boff = P.boff;
  a.B = P.H.ptr;
  a.exps = P.exps;
  a.mofn = c->mofn.ptr;
  a.y = yacc;
  a.nb = P.nb;
  a.bs = bs;
  a.R = R;
  a.err = P.err;
  for (int m : c->h_mofn) a.mmax = std::max(a.mmax, std::abs(m));
  const int chunks = ih_chunks(c->n);
  double2 *total = chunks > 1 ? ib_scratch(c, mem, P.acc, len) : nullptr;
  float2 *xh = ib_scratch(c, mem, P.xh, (size_t)c->n * kp * std::min(16, R));
  for (int r0 = 0; r0 < R; r0 += 16) {
    a.r0 = r0;
    a.rt = std::min(16, R - r0);
    auto &tl = ib_tiles(c, a.rt, 1, st);
    a.toff = tl.toff.ptr;
    a.per = tl.per;
    const int ntiles = tl.h_toff.back();
    const size_t elems = (size_t)c->n * kp * a.rt;
    ih_copy_kernel<<<(unsigned)((elems + 255) / 256), 256, 0, st>>>(x, c->n, bs, kp, R, r0, a.rt, top, xh);
    SG_CUDA(cudaGetLastError());
    ++launched;
    a.x = xh;
    for (int q = 0; q < chunks; ++q) {
      a.t0 = (int)((long long)ntiles * q / chunks);
      a.t1 = (int)((long long)ntiles * (q + 1) / chunks);
      if (a.t0 < a.t1) {
        ih_dispatch(c, [&](auto nc, auto kpc) {
          constexpr int NC = decltype(nc)::value, KP = decltype(kpc)::value;
          static bool attr_done[64] = {};
          constexpr int smem = (int)ih_smem<NC, KP>();
          if (first_on_device(attr_done))
            SG_CUDA(cudaFuncSetAttribute(ih_kernel<NC, KP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
          ih_kernel<NC, KP><<<std::min(sm_count(), a.t1 - a.t0), kIhThreads, smem, st>>>(a);
        });
        SG_CUDA(cudaGetLastError());
        ++launched;
      }
      if (chunks > 1) {
        ih_fold_kernel<<<(unsigned)((rows * a.rt + 255) / 256), 256, 0, st>>>(a.y, total, rows, R, r0, a.rt, q == 0,
                                                                              q == chunks - 1);
        SG_CUDA(cudaGetLastError());
        ++launched;
      }
    }
  }
  launch_fp32_epilogue(c, x, y, R, master, st, top, P.err, yacc);
  ib_leave(c, st);
  return launched + 1;
}

}  // namespace sg
