// Epilogue shared by the FP64-result coupling kernels: W x, or x - T (W x) with diagonal or full T
// blocks, from one receiver's reduced sums.
#pragma once

#include "sg_internal.h"

namespace sg {

// red: shared [bs][RT] reduced coupling sums for receiver i and RHS r0..r0+RT-1.
static __device__ void coupling_epilogue(const CouplingLaunch &L, int i, int r0, int RT, const double2 *red) {
  const int bs = L.bs, R = L.nrhs;
  for (int e = threadIdx.x; e < bs * RT; e += blockDim.x) {
    const int n1 = e / RT, r = e - n1 * RT;
    const size_t o = ((size_t)i * bs + n1) * R + r0 + r;
    double2 v = red[e];
    if (L.master) {
      const int ty = L.ptype[i];
      double2 tw;
      if (L.t_diag) {
        const double2 t = L.t[(size_t)ty * bs + n1];
        tw = make_double2(t.x * v.x - t.y * v.y, t.x * v.y + t.y * v.x);
      } else {
        const double2 *trow = L.t + ((size_t)ty * bs + n1) * bs;
        double ar = 0.0, ai = 0.0;
        for (int n2 = 0; n2 < bs; ++n2) {
          const double2 t = trow[n2];
          const double2 a = red[n2 * RT + r];
          ar = fma(t.x, a.x, fma(-t.y, a.y, ar));
          ai = fma(t.x, a.y, fma(t.y, a.x, ai));
        }
        tw = make_double2(ar, ai);
      }
      const double2 xv = L.x[o];
      v = make_double2(xv.x - tw.x, xv.y - tw.y);
    }
    L.y[o] = v;
  }
}

}  // namespace sg
