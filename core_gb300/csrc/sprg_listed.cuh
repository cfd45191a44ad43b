// FP64 recovered gradient of a listed tet vertex (a patch that grows or takes
// the FP64 fit), for the FP32 and learned kernels.
#pragma once
#include "sprg_internal.h"
#include "sprg_metric_f64.cuh"

namespace sprg {

// The gradient on a tet in the reference's operation order (apf::getGrad through
// J^-1 and the shape gradients 0, 1 and -1; elem_record_of and k_grad_ip give the
// same bits).  Rounded operations by name: this unit may be compiled with
// contraction.  A formula in differences of u would be exact on a constant
// field, where the sizes are those of the reference's rounding.
__device__ __forceinline__ void apply_gradients(const double* j, const double* g0, const double* u, double* g) {
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    double s = __dmul_rn(g0[r], u[0]);
#pragma unroll
    for (int k = 0; k < 3; ++k) s = __dadd_rn(s, __dmul_rn(j[3 * r + k], u[k + 1]));
    g[r] = s;
  }
}

// without the per-mesh records (no memory for them)
static __device__ __noinline__ void listed_grad_in_place(const DevMesh& mesh, const int* id, const double* u, double* g) {
  double x[4][3];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int k = 0; k < 3; ++k) x[a][k] = __ldg(mesh.xyz + 3 * (size_t)id[a] + k);
  double m[3][3];
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int k = 0; k < 3; ++k) m[r][k] = __dsub_rn(x[r + 1][k], x[0][k]);
  auto minor = [](double a, double b, double c, double d) { return __dsub_rn(__dmul_rn(a, b), __dmul_rn(c, d)); };
  double c[3][3];  // J^-1 det J
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int p = (i + 1) % 3, q = (i + 2) % 3;
#pragma unroll
    for (int k = 0; k < 3; ++k)
      c[i][k] = minor(m[(k + 1) % 3][p], m[(k + 2) % 3][q], m[(k + 2) % 3][p], m[(k + 1) % 3][q]);
  }
  double det = __dmul_rn(m[0][0], c[0][0]);
  det = __dadd_rn(det, __dmul_rn(m[1][0], c[0][1]));
  det = __dadd_rn(det, __dmul_rn(m[2][0], c[0][2]));
  bool safe = bexp(det) >= 623 && bexp(det) <= 1423;  // see quotient()
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    const int ex = bexp(c[i / 3][i % 3]);
    safe = safe && ex <= 1523 && (ex >= 523 || c[i / 3][i % 3] == 0.0);
  }
  if (safe) {
    const double y = __drcp_rn(det);
#pragma unroll
    for (int i = 0; i < 9; ++i) c[i / 3][i % 3] = quotient(c[i / 3][i % 3], det, y);
  } else {
#pragma unroll 1
    for (int i = 0; i < 3; ++i) {
      bool fine = true;
      for (int k = 0; k < 3; ++k) {
        c[i][k] = __ddiv_rn(c[i][k], det);
        fine = fine && bexp(c[i][k]) != 0x7ff;
      }
      if (!fine)  // its products with the shape gradients' zeros
        for (int k = 0; k < 3; ++k) c[i][k] = __longlong_as_double(0x7ff8000000000000ll);
    }
  }
  double g0[3];
#pragma unroll
  for (int r = 0; r < 3; ++r) g0[r] = __dsub_rn(__dsub_rn(-c[r][0], c[r][1]), c[r][2]);
  apply_gradients(&c[0][0], g0, u, g);
}

// sum_i w_i grad u over patch `it` by one warp: lanes over the elements, FP64
// gradients, fixed reduction tree; every lane gets the sum (the FP64 form's
// bits).  false: the patch has no weights (SPRG_EPATCH).
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
    double uv[4], g[3];
#pragma unroll
    for (int a = 0; a < 4; ++a) uv[a] = __ldg(u + id[a]);
    const double wk = wi[i];
    if (pw.g) {  // these chains are the longest of a small pass: no coordinates, no division
      const double2* r = reinterpret_cast<const double2*>(pw.g + 12 * (pw.woff[it] + i));
      double j[12];
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        const double2 t = __ldg(r + k);
        j[2 * k] = t.x;
        j[2 * k + 1] = t.y;
      }
      apply_gradients(j, j + 9, uv, g);
    } else {
      listed_grad_in_place(m, id, uv, g);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) acc[k] = __dadd_rn(acc[k], __dmul_rn(wk, g[k]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < 3; ++k) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
  return true;
}

}  // namespace sprg
