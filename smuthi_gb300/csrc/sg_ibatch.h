// Plan of the interval-batched operators (sg_ibatch.cu: FP64, sg_ibatch32.cu: FP32): the ordered pairs sorted by
// lookup interval, and the power-of-two scales of an interval's coefficients.
#pragma once

#include <cuda_runtime.h>

#include "sg_internal.h"

namespace sg {

__device__ __forceinline__ int ib_field(double v) { return (__double2hiint(v) >> 20) & 0x7FF; }

// Scales of the NC coefficient matrices C [NC][n2][n1] of an interval, by a whole block: |Re|, |Im| of an element are
// below 2^(ea[n1] + eb[n2]). Column exponents first, then row exponents of what they leave. A column of zeros keeps an
// exponent below all others: nothing that x holds for it may take part in the scale of the products.
template <int NC, int KP>
__device__ __forceinline__ void ib_exponents(const double2 *C, int bs, int *eb, int *ea) {
  const int tid = threadIdx.x, bs2 = bs * bs;
  if (tid < KP) eb[tid] = ea[tid] = -(1 << 20);
  __syncthreads();
  for (int e = tid; e < NC * bs2; e += blockDim.x) {
    const int f = max(ib_field(C[e].x), ib_field(C[e].y));
    if (f) atomicMax(&eb[(e % bs2) / bs], f - 1022);
  }
  __syncthreads();
  for (int e = tid; e < NC * bs2; e += blockDim.x) {
    const int f = max(ib_field(C[e].x), ib_field(C[e].y));
    if (f) atomicMax(&ea[e % bs], f - 1022 - eb[(e % bs2) / bs]);
  }
  __syncthreads();
  if (tid < KP && ea[tid] == -(1 << 20)) ea[tid] = 0;
  __syncthreads();
}

// the sorted pairs, made at the first use after a change of particles or lookup
void ib_plan(sg_context *c, cudaStream_t st);
// tiles for rt right-hand sides; sets = 0: chosen for the FP64 operator
sg_context::IbTiles &ib_tiles(sg_context *c, int rt, int sets, cudaStream_t st);
// scratch memory of a call, within the limit
template <typename T>
T *ib_scratch(sg_context *c, CallMemory &mem, DevBuf<T> &kept, size_t count) {
  if (!mem.graph) c->ib.take(kept, count);
  return mem.get(kept, count);
}
// the tiles exist
bool ib_has_tiles(const sg_context *c, int rt, int sets);
// right-hand sides of the FP64 operator at a time
int ib_group(const sg_context *c, int R);
// Orders the calls that use the plan and its workspaces across streams. A captured call has workspaces of its own and only
// needs the plan: what prepares it must have run.
void ib_enter(sg_context *c, cudaStream_t st);
void ib_leave(sg_context *c, cudaStream_t st);

}  // namespace sg
