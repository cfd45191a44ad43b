// FP64 recovered gradient of a listed tet vertex (a patch that grows or takes
// the FP64 fit), for the FP32 and learned kernels.
#pragma once
#include "sprg_internal.h"

namespace sprg {

// sum_i w_i grad u over patch `it` by one warp: lanes over the elements, FP64
// gradients, fixed reduction tree; every lane gets the sum.  false: the
// patch has no weights (SPRG_EPATCH).
__device__ __forceinline__ bool listed_grad_sum(const DevMesh& m, const double* __restrict__ u, const PatchWeights& pw,
                                                int it, double* acc) {
  const int lane = threadIdx.x & 31;
  const int n = pw.wn[it];
  acc[0] = acc[1] = acc[2] = 0;
  if (n < 0) {
    if (lane == 0 && atomicCAS(&pw.st->code, 0, SPRG_EPATCH) == 0) pw.st->where = pw.v[it];
    return false;
  }
  const int* el = pw.el + (size_t)it * pw.stride;
  const double* wi = pw.w + pw.woff[it];
  for (int i = lane; i < n; i += 32) {
    const int4 tv = __ldg(reinterpret_cast<const int4*>(m.ev) + el[i]);
    const int id[4] = {tv.x, tv.y, tv.z, tv.w};
    double x[4][3], e[3][3], du[3];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int k = 0; k < 3; ++k) x[a][k] = __ldg(m.xyz + 3 * (size_t)id[a] + k);
    const double u0 = __ldg(u + id[0]);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      du[a] = __ldg(u + id[a + 1]) - u0;
#pragma unroll
      for (int k = 0; k < 3; ++k) e[a][k] = x[a + 1][k] - x[0][k];
    }
    double cf[3][3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double* p = e[(a + 1) % 3];
      const double* q = e[(a + 2) % 3];
      cf[a][0] = p[1] * q[2] - p[2] * q[1];
      cf[a][1] = p[2] * q[0] - p[0] * q[2];
      cf[a][2] = p[0] * q[1] - p[1] * q[0];
    }
    const double wk = wi[i] / (e[0][0] * cf[0][0] + e[0][1] * cf[0][1] + e[0][2] * cf[0][2]);
#pragma unroll
    for (int k = 0; k < 3; ++k) acc[k] += wk * (cf[0][k] * du[0] + cf[1][k] * du[1] + cf[2][k] * du[2]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < 3; ++k) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
  return true;
}

}  // namespace sprg
