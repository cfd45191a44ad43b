// FP64 metric edge lengths (MetricSizeField::measure, ma/maSize.cc:158-214),
// shared by the FP64 translation units (-fmad=false).
#pragma once
#include "sprg_refmath.cuh"

namespace sprg {

__device__ __forceinline__ int bexp(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }

// a / b rounded to nearest, y = 1 / b rounded to nearest: two exact-residual
// corrections of a y.  The first leaves a faithful quotient, the second
// rounds it correctly (P. Markstein, "Computation of elementary functions on
// the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990), given
// that nothing under- or overflows (the callers check exponents: b in
// [2^-400, 2^400], a 0 or in [2^-500, 2^500]).  Five FP64 operations instead
// of a division each.
__device__ __forceinline__ double quotient(double a, double b, double y) {
  double q = a * y;
  q = fma(fma(-b, q, a), y, q);
  return fma(fma(-b, q, a), y, q);
}

// 2-point Gauss, the reference's own sequence
__device__ __forceinline__ double metric_length(const ref::V3& x0, const ref::V3& x1, const double* hv,
                                                const double* Rv) {
  ref::V3 x[2] = {x0, x1};
  ref::M3 J = ref::jacobian(x, 2, 1);
  const double gp[2] = {0.577350269189626, -0.577350269189626};
  double measurement = 0;
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    double N[2];
    ref::edge_shape_values(gp[p], N);
    ref::M3 Q = ref::get_transform(hv, Rv, N, 2);
    double dV2 = ref::jacobian_det(ref::mul(J, Q), 1);
    measurement += 1 * dV2;
  }
  return measurement;
}

__device__ __forceinline__ void identity9(double* R) {
  for (int k = 0; k < 9; ++k) R[k] = (k % 4 == 0) ? 1.0 : 0.0;
}

static __device__ __noinline__ double iso_length_ref(const ref::V3& x0, const ref::V3& x1, double sa, double sb) {
  double hv[6] = {sa, sa, sa, sb, sb, sb}, Rv[18];
  identity9(Rv);
  identity9(Rv + 9);
  return metric_length(x0, x1, hv, Rv);
}

// sizes at the two Gauss points of an edge with end sizes sa, sb
__device__ __forceinline__ void gauss_sizes(double sa, double sb, double* h) {
  const double gp[2] = {0.577350269189626, -0.577350269189626};
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    double N[2];
    ref::edge_shape_values(gp[p], N);
    h[p] = sa * N[0] + sb * N[1];
  }
}

// The isotropic length, bitwise the reference's: the interpolated identity
// frames are the identity again (N0 + N1 rounds to 1), so the transform is
// 1 / h on the diagonal; the edge's Jacobian is half the coordinate
// difference, and that factor (a power of two) is taken once at the end.
// About 55 FP64 operations.  Sizes or a length outside the exponents where
// that holds (0, subnormal, not finite, far from 1) take the sequence itself.
__device__ __forceinline__ double iso_length(const ref::V3& x0, const ref::V3& x1, double sa, double sb) {
  double h[2], s[2];
  gauss_sizes(sa, sb, h);
  const ref::V3 d = ref::sub(x1, x0);
#pragma unroll
  for (int p = 0; p < 2; ++p) s[p] = ref::len(ref::scale(d, __drcp_rn(h[p])));
  const double L = 0.5 * (s[0] + s[1]);
  const int e0 = bexp(h[0]), e1 = bexp(h[1]), el = bexp(L);
  if (min(min(e0, e1), el) < 623 || max(max(e0, e1), el) > 1423) return iso_length_ref(x0, x1, sa, sb);
  return L;
}

}  // namespace sprg
