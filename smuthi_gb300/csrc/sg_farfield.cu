// Particle sum of the scattered field's plane-wave expansion, for the cross sections.
//
// The far field of N particles at one height (smuthi/postprocessing/far_field.py:363-427, through
// smuthi/postprocessing/scattered_field.py:80-150 and smuthi/fields/transformations.py:133-233)
// needs, for every in-plane wavenumber kappa_k and azimuth alpha_a, the sum over particles
//
//   g[r][p][k][a] = sum_i exp(-i kappa_k (cos alpha_a x_i + sin alpha_a y_i))
//                         sum_n c[i][n][r] S[n][p][k] exp(i m(n) alpha_a)
//
// (S: the SVWF -> plane-wave transformation coefficient of multipole n and polarisation p at
// kappa_k, computed on the host; the k-dependent prefactor and the layer response are applied on
// the host afterwards). Particles at different heights carry a per-particle factor
// zphase[k][i] = exp(+-i k_z,k (z_ref - z_i)) inside the sum (null: all at one height, the factor is
// part of the host prefactor). On the host this is a dense N-long contraction for every (k, a, r, p):
// 72 s for 1000 particles and one RHS on the default angular grid, so hours at 10 000 particles and
// 16 RHS. Here one thread owns one azimuth a of one kappa_k and a tile of CT (r, p) columns; a block
// stages, for a chunk of CH particles, the m-resolved data D[m][i][col] = sum_{n: m(n) = m}
// c[i][n][r] S[n][p][k] in shared memory (computed once per block and chunk), and every thread then
// applies its lateral phase. All arithmetic is FP64, and the FP64 pipe bounds the kernel.
//
// Up to m_max = 4 the sums are kept apart for every m (F[m][col] += phase D[m][i][col], 4 FP64 operations
// each) and exp(i m alpha_a) is applied once at the end; with the table-driven phase that is 19 + 4 CT (2
// m_max + 1) operations per particle and direction. One right-hand side has two columns, so its tile is two
// columns wide; more right-hand sides share each phase between four. (A tile of eight columns, with phase
// times exp(i m alpha) formed per particle, spent 296 operations on one right-hand side's two columns: 1000
// particles, l_max 3, 181 x 721 directions 69.8 ms; now 19.5.) Larger m_max takes the general kernel, whose
// registers do not grow with m_max, and so do a few particles with many right-hand sides (ff_sum_per_m).
#include <cuda_runtime.h>
#include <math.h>

#include "sg_internal.h"
#include "sg_sincos.h"

namespace sg {

static constexpr int kFfThreads = 128;  // azimuths per block
static constexpr int kFfCH = 32;        // particles per staged chunk
static constexpr int kFfCT = 8;         // (r, p) columns per block
static constexpr int kFfMaxM = 16;

struct FfArgs {
  const double2 *xy;     // [N]
  const double2 *coef;   // [N][B][R]
  const double2 *S;      // [B][2][K]
  const double *kpar;    // [K]
  const double *alpha;   // [A]
  const int *moff;       // [nm + 1] CSR over m = -mmax..mmax of the n with that m
  const int *mlist;      // [B]
  const double2 *zph;    // [K][N] per-particle height factor, or null
  const double2 *sc;     // sine table
  double2 *out;          // [R][2][K][A]
  int N, B, R, K, A, mmax;
};

// D[m][i][col] of the chunk of particles at i0 for the columns from c0
template <int CT>
__device__ __forceinline__ void ff_stage(const FfArgs &f, int k, int i0, int c0, double2 *D) {
  const int nm = 2 * f.mmax + 1, ncol = 2 * f.R;
  for (int e = threadIdx.x; e < nm * kFfCH * CT; e += kFfThreads) {
    const int mi = e / (kFfCH * CT), rem = e - mi * kFfCH * CT;
    const int ii = rem / CT, c = rem - ii * CT;
    const int i = i0 + ii, col = c0 + c;
    double2 v = make_double2(0.0, 0.0);
    if (i < f.N && col < ncol) {
      const int p = col / f.R, r = col - p * f.R;
      for (int q = f.moff[mi]; q < f.moff[mi + 1]; ++q) {
        const int n = f.mlist[q];
        const double2 cv = f.coef[((size_t)i * f.B + n) * f.R + r];
        const double2 sv = f.S[((size_t)n * 2 + p) * f.K + k];
        v.x = fma(cv.x, sv.x, fma(-cv.y, sv.y, v.x));
        v.y = fma(cv.x, sv.y, fma(cv.y, sv.x, v.y));
      }
      if (f.zph) {
        const double2 zp = f.zph[(size_t)k * f.N + i];
        v = make_double2(v.x * zp.x - v.y * zp.y, v.x * zp.y + v.y * zp.x);
      }
    }
    D[e] = v;
  }
}

template <int CT>
__device__ __forceinline__ void ff_store(const FfArgs &f, int k, int a, int c0, const double2 (&acc)[CT]) {
#pragma unroll
  for (int cc = 0; cc < CT; ++cc) {
    const int col = c0 + cc;
    if (col < 2 * f.R) {
      const int p = col / f.R, r = col - p * f.R;
      f.out[(((size_t)r * 2 + p) * f.K + k) * f.A + a] = acc[cc];
    }
  }
}

// m_max = MM <= 4: one sum per m
template <int MM, int CT>
__global__ void __launch_bounds__(kFfThreads) ff_sum_m_kernel(const FfArgs f) {
  constexpr int NM = 2 * MM + 1;
  extern __shared__ double2 ff_smem[];
  double2 *T = ff_smem, *D = ff_smem + kScTable;  // D: [NM][CH][CT]
  const int k = blockIdx.x, a = blockIdx.y * kFfThreads + threadIdx.x, c0 = blockIdx.z * CT;
  const double kap = f.kpar[k];
  double ca = 1.0, sa = 0.0;
  if (a < f.A) sincos(f.alpha[a], &sa, &ca);
  sc_load(f.sc, T);
  double2 F[NM][CT];
#pragma unroll
  for (int m = 0; m < NM; ++m)
#pragma unroll
    for (int c = 0; c < CT; ++c) F[m][c] = make_double2(0.0, 0.0);
  for (int i0 = 0; i0 < f.N; i0 += kFfCH) {
    __syncthreads();
    ff_stage<CT>(f, k, i0, c0, D);
    __syncthreads();
    if (a < f.A) {
      const int nch = min(kFfCH, f.N - i0);
      for (int ii = 0; ii < nch; ++ii) {
        const double2 pos = f.xy[i0 + ii];
        double s, c;
        sc_sincos(-kap * (ca * pos.x + sa * pos.y), T, &s, &c);  // exp(-i kappa (cos a x + sin a y))
#pragma unroll
        for (int m = 0; m < NM; ++m)
#pragma unroll
          for (int cc = 0; cc < CT; ++cc) {
            const double2 d = D[(m * kFfCH + ii) * CT + cc];
            F[m][cc].x = fma(c, d.x, fma(-s, d.y, F[m][cc].x));
            F[m][cc].y = fma(c, d.y, fma(s, d.x, F[m][cc].y));
          }
      }
    }
  }
  if (a >= f.A) return;
  double2 acc[CT];
#pragma unroll
  for (int c = 0; c < CT; ++c) acc[c] = make_double2(0.0, 0.0);
#pragma unroll
  for (int m = MM; m >= 0; --m) {  // m and -m share their sine and cosine
    double s = 0.0, c = 1.0;
    if (m > 0) sincos((double)m * f.alpha[a], &s, &c);
#pragma unroll
    for (int h = 0; h < (m > 0 ? 2 : 1); ++h) {
      const double sh = h ? s : -s;
#pragma unroll
      for (int cc = 0; cc < CT; ++cc) {
        const double2 v = F[h ? MM + m : MM - m][cc];
        acc[cc].x = fma(c, v.x, fma(-sh, v.y, acc[cc].x));
        acc[cc].y = fma(c, v.y, fma(sh, v.x, acc[cc].y));
      }
    }
  }
  ff_store<CT>(f, k, a, c0, acc);
}

// any m_max
__global__ void __launch_bounds__(kFfThreads) ff_sum_kernel(const FfArgs f) {
  extern __shared__ double2 ff_smem[];
  const int nm = 2 * f.mmax + 1;
  double2 *D = ff_smem;  // [nm][CH][CT]
  const int k = blockIdx.x;
  const int a = blockIdx.y * kFfThreads + threadIdx.x;
  const int c0 = blockIdx.z * kFfCT;
  const double kap = f.kpar[k];
  double ca = 1.0, sa = 0.0;
  double2 em[2 * kFfMaxM + 1];
  if (a < f.A) {
    sincos(f.alpha[a], &sa, &ca);
    for (int mi = 0; mi < nm; ++mi) {
      double s, c;
      sincos((double)(mi - f.mmax) * f.alpha[a], &s, &c);
      em[mi] = make_double2(c, s);
    }
  }
  double2 acc[kFfCT];
#pragma unroll
  for (int c = 0; c < kFfCT; ++c) acc[c] = make_double2(0.0, 0.0);

  for (int i0 = 0; i0 < f.N; i0 += kFfCH) {
    __syncthreads();
    ff_stage<kFfCT>(f, k, i0, c0, D);
    __syncthreads();
    if (a < f.A) {
      const int nch = min(kFfCH, f.N - i0);
      for (int ii = 0; ii < nch; ++ii) {
        const double2 pos = f.xy[i0 + ii];
        double s, c;
        sincos(-kap * (ca * pos.x + sa * pos.y), &s, &c);  // lateral phase exp(-i kappa (cos a x + sin a y))
        for (int mi = 0; mi < nm; ++mi) {
          const double wr = c * em[mi].x - s * em[mi].y, wi = c * em[mi].y + s * em[mi].x;
          const double2 *d = D + ((size_t)mi * kFfCH + ii) * kFfCT;
#pragma unroll
          for (int cc = 0; cc < kFfCT; ++cc) {
            const double2 dv = d[cc];
            acc[cc].x = fma(wr, dv.x, fma(-wi, dv.y, acc[cc].x));
            acc[cc].y = fma(wr, dv.y, fma(wi, dv.x, acc[cc].y));
          }
        }
      }
    }
  }
  if (a < f.A) ff_store<kFfCT>(f, k, a, c0, acc);
}

template <int MM>
static void ff_launch(const FfArgs &f, cudaStream_t st) {
  const int ct = f.R == 1 ? 2 : 4;
  const size_t smem = (kScTable + (size_t)(2 * MM + 1) * kFfCH * ct) * sizeof(double2);
  const dim3 grid(f.K, (f.A + kFfThreads - 1) / kFfThreads, (2 * f.R + ct - 1) / ct);
  static bool attr_done[2][64] = {};
  if (f.R == 1) {
    if (first_on_device(attr_done[0]))
      SG_CUDA(cudaFuncSetAttribute(ff_sum_m_kernel<MM, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    ff_sum_m_kernel<MM, 2><<<grid, kFfThreads, smem, st>>>(f);
  } else {
    if (first_on_device(attr_done[1]))
      SG_CUDA(cudaFuncSetAttribute(ff_sum_m_kernel<MM, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    ff_sum_m_kernel<MM, 4><<<grid, kFfThreads, smem, st>>>(f);
  }
}

// The kernel with one sum per m spends more once per direction and column tile (its tiles are half as wide), the general
// one more per particle; FP64 operations of both. 16 right-hand sides, l_max 3, 181 x 721 directions: 1 particle 0.88 ms
// against 0.66 with the general kernel, 5 1.80 against 1.69, 20 5.3 against 5.5; one right-hand side 0.25 against 0.30.
static bool ff_sum_per_m(int n, int nrhs, int mmax) {
  if (mmax > 4) return false;
  const double nm = 2 * mmax + 1, ct = nrhs == 1 ? 2 : 4;
  const int wide = (2 * nrhs + kFfCT - 1) / kFfCT, narrow = (2 * nrhs + (int)ct - 1) / (int)ct;
  return narrow * (n * (19 + 4 * ct * nm) + 44 * mmax + 300) <= wide * (n * (44 + 38 * nm) + 44 * nm + 172);
}

// returns the number of kernels launched
int farfield_sum(const double2 *xy, int n, int bs, int nrhs, const double2 *coef, int mmax, const int *mofn_host,
                  int nk, const double *kpar, const double2 *S, int na, const double *alpha, const double2 *zphase,
                  double2 *out, cudaStream_t st) {
  SG_REQUIRE(n >= 1 && bs >= 1 && nrhs >= 1 && nk >= 1 && na >= 1, "empty far-field problem");
  SG_REQUIRE(mmax >= 0 && mmax <= kFfMaxM, "m_max must be in [0, 16]");
  const int nm = 2 * mmax + 1;
  std::vector<int> moff(nm + 1, 0), mlist;
  for (int mi = 0; mi < nm; ++mi) {
    for (int q = 0; q < bs; ++q) {
      SG_REQUIRE(mofn_host[q] >= -mmax && mofn_host[q] <= mmax, "m_of_n outside [-m_max, m_max]");
      if (mofn_host[q] == mi - mmax) mlist.push_back(q);
    }
    moff[mi + 1] = (int)mlist.size();
  }
  moff.insert(moff.end(), mlist.begin(), mlist.end());
  DevBuf<double2> scratch;  // sine table, then moff and mlist
  scratch.reserve(kScTable + (moff.size() * sizeof(int) + sizeof(double2) - 1) / sizeof(double2));
  int *d_moff = reinterpret_cast<int *>(scratch.ptr + kScTable);
  SG_CUDA(cudaMemcpyAsync(d_moff, moff.data(), moff.size() * sizeof(int), cudaMemcpyHostToDevice, st));
  const bool per_m = ff_sum_per_m(n, nrhs, mmax);
  if (per_m) sc_table(scratch.ptr, st);
  FfArgs f{xy, coef, S, kpar, alpha, d_moff, d_moff + nm + 1, zphase, scratch.ptr, out, n, bs, nrhs, nk, na, mmax};
  switch (per_m ? mmax : kFfMaxM) {
    case 0: ff_launch<0>(f, st); break;
    case 1: ff_launch<1>(f, st); break;
    case 2: ff_launch<2>(f, st); break;
    case 3: ff_launch<3>(f, st); break;
    case 4: ff_launch<4>(f, st); break;
    default: {
      const size_t smem = (size_t)nm * kFfCH * kFfCT * sizeof(double2);
      SG_CUDA(cudaFuncSetAttribute(ff_sum_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      dim3 grid(nk, (na + kFfThreads - 1) / kFfThreads, (2 * nrhs + kFfCT - 1) / kFfCT);
      ff_sum_kernel<<<grid, kFfThreads, smem, st>>>(f);
    }
  }
  SG_CUDA(cudaGetLastError());
  SG_CUDA(cudaStreamSynchronize(st));  // the scratch buffer above is released on return
  return per_m ? 2 : 1;
}

}  // namespace sg
