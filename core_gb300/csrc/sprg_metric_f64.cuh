// The powers of an element error and FP64 metric edge lengths
// (MetricSizeField::measure, ma/maSize.cc:158-214), shared by the FP64
// translation units (-fmad=false).
#pragma once
#include "sprg_refmath.cuh"

namespace sprg {

// err to the exponents the size field needs in D dimensions (p = 1):
//   q = (sqrt err)^(-2 / (2 + D))  = err^(-1/(D+2))
//   g = (sqrt err)^(2 D / (2 + D)) = err q^2, on triangles the root itself
// Reduced to err = 2^(P k) m with m in [1, 2^P), P = D + 2: the hardware
// log2 / exp2 give m^(-1/P) to 2^-21, one step of the cubically convergent
// Householder iteration on 1 - m r^P squares that twice over, 2^-k goes into
// the exponent.  9 FP64 operations on tets, within 2 ulps (against extended
// precision, rms in units of 2^-53: q 0.44 and g 1.07, the sequence 4.0 and 8.0 in
// space; q 0.44 against 0.48 in the plane); pow(sqrt(err)) took about 110 for
// each of the two.  Zero, subnormal, negative and not finite errors
// take the sequence itself.
template <int D>
static __device__ __noinline__ void error_powers_ref(double err, double* q, double* g) {
  const double t = sqrt(err), p = 1, d = D;
  *q = pow(t, -(2 / (2 * p + d)));
  *g = pow(t, (2 * d) / (2 * p + d));
}

template <int D>
__device__ __forceinline__ void error_powers(double err, double& q, double& g) {
  constexpr int P = D + 2;
  const int hi = __double2hiint(err), lo = __double2loint(err);
  if (hi < 0x00100000 || hi >= 0x7ff00000) {
    error_powers_ref<D>(err, &q, &g);
    return;
  }
  const int e = (hi >> 20) - 1023;
  const int k = (e + 300 * P) / P - 300;  // floor(e / P)
  const int r = e - P * k, mant = hi & 0xfffff;
  const double m = __hiloint2double(mant | ((r + 1023) << 20), lo);
  float l, sf = __int_as_float((mant << 3) | (int)((unsigned)lo >> 29) | ((r + 127) << 23));
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(sf));
  l *= -1.0f / P;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(sf) : "f"(l));
  const int b = __float_as_int(sf);
  const double r0 = __hiloint2double((b >> 3) + (896 << 20), b << 29);
  const double r2 = r0 * r0, r4 = r2 * r2;
  const double h = fma(-m, P == 5 ? r4 * r0 : r4, 1.0);
  const double c = P == 5 ? fma(h, 3.0 / 25.0, 0.2) : fma(h, 5.0 / 32.0, 0.25);
  const double y = fma(r0 * h, c, r0);
  q = __hiloint2double(__double2hiint(y) - (k << 20), __double2loint(y));
  g = D == 2 ? sqrt(err) : err * (q * q);
}

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

// ---- anisotropic transforms -------------------------------------------
__device__ __forceinline__ bool all_zero(double a, double b, double c, double d) {
  return ((__double_as_longlong(a) | __double_as_longlong(b) | __double_as_longlong(c) | __double_as_longlong(d)) << 1) ==
         0;
}
// a size whose reciprocal is an ordinary number (the products with 0 that the
// transform leaves out are then 0)
__device__ __forceinline__ bool ordinary(double h) { return (unsigned)(bexp(h) - 523) <= 1000u; }

// AnisoSizeField's Q = orth(R) diag(1/h) (ma/maSize.cc:94-117, 395-412) for an
// interpolated frame R and ordinary sizes h, bitwise: the products with the
// diagonal matrix's zeros are left out
__device__ __forceinline__ ref::M3 transform_of(const double* h, const ref::M3& R) {
  ref::M3 Q = ref::orthogonalize(R);
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const double ih = 1 / h[j];
#pragma unroll
    for (int i = 0; i < 3; ++i) Q.m[i][j] *= ih;
  }
  return Q;
}

// the same where the third row and column are (0, 0, .): the 2 x 2 block q =
// {Q00, Q01, Q10, Q11}, and the third direction's z (1/h2 not applied)
__device__ __forceinline__ double planar_transform(double h0, double h1, double a, double b, double c, double d,
                                                   double* q) {
  // first column (a, c), second (b, d)
  const double n0 = sqrt(a * a + c * c);
  const double r0x = a / n0, r0y = c / n0;
  const double t = r0x * b + r0y * d;
  const double x = b - r0x * t, y = d - r0y * t;
  const double n1 = sqrt(x * x + y * y);
  const double r1x = x / n1, r1y = y / n1;
  const double i0 = 1 / h0, i1 = 1 / h1;
  q[0] = r0x * i0;
  q[1] = r1x * i1;
  q[2] = r0y * i0;
  q[3] = r1y * i1;
  return r0x * r1y - r0y * r1x;
}

static __device__ __noinline__ double aniso_length_ref(const ref::V3& x0, const ref::V3& x1, const double* hv,
                                                       const double* Rv) {
  return metric_length(x0, x1, hv, Rv);
}

// AnisoSizeField's length of an edge, bitwise metric_length: half the edge
// vector is taken once at the end (a power of two), products with the fixed
// zeros are left out, and an edge and frames in a z = const plane take the
// 2 x 2 block alone: about 250 FP64 operations, or 390 in space, against 550.
// Sizes or a length outside the ordinary range take the sequence itself.
__device__ __forceinline__ double aniso_length(const ref::V3& x0, const ref::V3& x1, const double* hv,
                                               const double* Rv) {
  const double gp[2] = {0.577350269189626, -0.577350269189626};
  const ref::V3 d = ref::sub(x1, x0);
  bool fine = true;
  double s[2];
  if (all_zero(Rv[2], Rv[5], Rv[6], Rv[7]) && all_zero(Rv[11], Rv[14], Rv[15], Rv[16]) && d.v[2] == 0.0) {
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      double N[2], q[4];
      ref::edge_shape_values(gp[p], N);
      const double h0 = hv[0] * N[0] + hv[3] * N[1], h1 = hv[1] * N[0] + hv[4] * N[1],
                   h2 = hv[2] * N[0] + hv[5] * N[1];
      fine = fine && ordinary(h0) && ordinary(h1) && ordinary(h2);
      planar_transform(h0, h1, Rv[0] * N[0] + Rv[9] * N[1], Rv[1] * N[0] + Rv[10] * N[1], Rv[3] * N[0] + Rv[12] * N[1],
                       Rv[4] * N[0] + Rv[13] * N[1], q);
      const double a = d.v[0] * q[0] + d.v[1] * q[2], b = d.v[0] * q[1] + d.v[1] * q[3];
      s[p] = sqrt(a * a + b * b);
    }
  } else {
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      double N[2], h[3];
      ref::edge_shape_values(gp[p], N);
      ref::M3 R;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        h[k] = hv[k] * N[0] + hv[3 + k] * N[1];
        fine = fine && ordinary(h[k]);
      }
#pragma unroll
      for (int k = 0; k < 9; ++k) R.m[k / 3][k % 3] = Rv[k] * N[0] + Rv[9 + k] * N[1];
      const ref::M3 Q = transform_of(h, R);
      ref::V3 e;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        double t = d.v[0] * Q.m[0][j];
        t += d.v[1] * Q.m[1][j];
        t += d.v[2] * Q.m[2][j];
        e.v[j] = t;
      }
      s[p] = ref::len(e);
    }
  }
  const double L = 0.5 * (s[0] + s[1]);
  const int el = bexp(L);
  if (!fine || el < 623 || el > 1423) return aniso_length_ref(x0, x1, hv, Rv);
  return L;
}

// The same length where both ends' frames are rotations about z and the edge
// lies in a z = const plane (what the Hessian's metric gives on a triangle
// mesh): the interpolated second column is the first's +90 degree rotation, so
// with c the first column, a = d . c, b = d x c and h0, h1 the interpolated sizes
//   |e Q| = sqrt((a / h0)^2 + (b / h1)^2) / |c|
//         = n / sqrt(n |c|^2 (h0 h1)^2),   n = (a h1)^2 + (b h0)^2:
// about 75 FP64 operations an edge against 250.  The two agree to a few ulps
// times the sizes' ratio (the cancellation in a and b, which both have), so a
// length within 2^24 ulps of a threshold is left to the sequence, as are ratios
// past 2^19, sizes, lengths or columns outside the ordinary range.  Against
// extended precision, rms in units of 2^-53 at sizes 1:2, 1:1000 and 1:500000
// apart: 0.99, 1.2 and 5.1 here, 0.99, 1.5 and 6.8 for the sequence.  False: not
// taken.
__device__ __forceinline__ bool rotated_length(const ref::V3& d, const double* hv, const double* Rv, double* L) {
  const unsigned long long sign = 0x8000000000000000ull;
  auto bits = [](double x) { return (unsigned long long)__double_as_longlong(x); };
  auto turned = [&](const double* R) {  // {c, -s, 0; s, c, 0; 0, 0, .}
    return all_zero(R[2], R[5], R[6], R[7]) && bits(R[4]) == bits(R[0]) &&
           (bits(R[1]) == (bits(R[3]) ^ sign) || ((bits(R[1]) | bits(R[3])) << 1) == 0);
  };
  auto size = [](double h) { return (unsigned)((__double2hiint(h) >> 20) - 923) <= 200u; };  // (0, 2^+-100)
  const int spread = max(max(bexp(hv[0]), bexp(hv[1])), max(bexp(hv[3]), bexp(hv[4]))) -
                     min(min(bexp(hv[0]), bexp(hv[1])), min(bexp(hv[3]), bexp(hv[4])));
  if (!(turned(Rv) && turned(Rv + 9) && (bits(d.v[2]) << 1) == 0 && spread <= 19)) return false;
  if (!(size(hv[0]) && size(hv[1]) && size(hv[2]) && size(hv[3]) && size(hv[4]) && size(hv[5]))) return false;
  const double N0 = (1.0 - 0.577350269189626) / 2.0, N1 = (1.0 + 0.577350269189626) / 2.0;
  double s[2];
  bool fine = true;
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const double w0 = p ? N1 : N0, w1 = p ? N0 : N1;
    const double h0 = fma(hv[0], w0, hv[3] * w1), h1 = fma(hv[1], w0, hv[4] * w1);
    const double cx = fma(Rv[0], w0, Rv[9] * w1), cy = fma(Rv[3], w0, Rv[12] * w1);
    const double a = fma(d.v[0], cx, d.v[1] * cy), b = fma(d.v[1], cx, -(d.v[0] * cy));
    const double ah = a * h1, bh = b * h0, hh = h0 * h1;
    const double n = fma(ah, ah, bh * bh), c2 = fma(cx, cx, cy * cy);
    fine = fine && bexp(c2) >= 1003 && bexp(c2) <= 1033 && (unsigned)(bexp(n) - 523) <= 1000u;
    s[p] = n * rsqrt(n * (c2 * (hh * hh)));
  }
  *L = 0.5 * (s[0] + s[1]);
  const long long l = (long long)bits(*L);
  auto away = [&](double t) { return llabs(l - __double_as_longlong(t)) > (1ll << 24); };
  return fine && bexp(*L) >= 923 && bexp(*L) <= 1123 && away(1.5) && away(0.5);
}

// ---- log-interpolated transforms (LogAnisoSizeField) ------------------------
// |e Q|^2 at one point, e the edge vector and Q = R diag(sqrt(exp(lambda))) of
// the interpolated log-metric A = R diag(lambda) R^T (a: rows 0 and 1 from
// the diagonal on, then A22): the squares of e in the eigenvectors' frame
// weighted with exp(lambda).  The eigenvalues come from mth::eigenQR's own
// iteration (mth/mthQR.cc:192-297: Hessenberg reduction, Wilkinson shifts,
// 1e-10 deflation from the bottom, the same failures) in its symmetric
// tridiagonal form: two rotations a step, applied to e instead of to an
// accumulated Q.  Same shifts and tests up to rounding; about 95 FP64
// operations a step against 400 for the full 3 x 3 matrices.
// Returns eigenQR's status (1 converged).
__device__ __forceinline__ int log_length2(const double* a, const ref::V3& e, double* out) {
  double d0 = a[0], d1 = a[3], d2 = a[5], e0 = a[1], e1 = a[4];
  double w0 = e.v[0], w1 = e.v[1], w2 = e.v[2];
  if (a[2] != 0.0) {
    const double n2 = fma(e0, e0, a[2] * a[2]), rn = rsqrt(n2), c = e0 * rn, s = a[2] * rn;
    const double cs = c * s, df = d2 - d1, t = 2 * cs * e1;
    e1 = fma(cs, df, (c * c - s * s) * e1);
    const double sd = s * s * df;
    d1 += sd + t;
    d2 -= sd + t;
    e0 = n2 * rn;
    const double y = fma(c, w1, s * w2);
    w2 = fma(c, w2, -s * w1);
    w1 = y;
  }
  int m = 3, status = 0;
  for (int it = 0; it < 100; ++it) {
    if (m == 3 && fabs(e1) < 1e-10) m = 2;
    if (m == 2 && fabs(e0) < 1e-10) m = 1;
    if (m == 1) {
      status = 1;
      break;
    }
    const double hi = m == 3 ? d1 : d0, lo = m == 3 ? d2 : d1, b = m == 3 ? e1 : e0;
    const double sig = (hi - lo) * 0.5, b2 = b * b;
    const double den = fabs(sig) + sqrt(fma(sig, sig, b2));
    if (!(den > 1e-10)) {
      status = -1;
      break;
    }
    const double mu = lo - copysign(b2, sig < 0 ? -1.0 : 1.0) / den;
    // two rotations; a column shorter than 1e-10 is left alone
    const double x0 = d0 - mu, x1 = d1 - mu, x2 = d2 - mu;
    double c0 = 1, s0 = 0, r0 = x0, c1 = 1, s1 = 0;
    const double n0 = fma(x0, x0, e0 * e0);
    if (!(n0 < 1e-20)) {
      const double rn = rsqrt(n0);
      c0 = x0 * rn;
      s0 = e0 * rn;
      r0 = n0 * rn;
    }
    const double r01 = fma(c0, e0, s0 * x1), q1 = fma(c0, x1, -s0 * e0), p1 = c0 * e1;
    double r1 = q1;
    const double n1 = fma(q1, q1, e1 * e1);
    if (!(n1 < 1e-20)) {
      const double rn = rsqrt(n1);
      c1 = q1 * rn;
      s1 = e1 * rn;
      r1 = n1 * rn;
    }
    const double r12 = fma(c1, p1, s1 * x2), r22 = fma(c1, x2, -s1 * p1);
    d0 = fma(r0, c0, r01 * s0) + mu;
    e0 = r1 * s0;
    d1 = fma(r1 * c0, c1, r12 * s1) + mu;
    e1 = r22 * s1;
    d2 = r22 * c1 + mu;
    const double y0 = fma(c0, w0, s0 * w1), y1 = fma(c0, w1, -s0 * w0);
    w0 = y0;
    w1 = fma(c1, y1, s1 * w2);
    w2 = fma(c1, w2, -s1 * y1);
  }
  *out = w0 * w0 * exp(d0) + w1 * w1 * exp(d1) + w2 * w2 * exp(d2);
  return status;
}

// the reference's sequence at one Gauss point
static __device__ __noinline__ double log_point_ref(const ref::V3& x0, const ref::V3& x1, const double* la,
                                                    const double* lb, double xi, bool* ok) {
  const ref::V3 x[2] = {x0, x1};
  const ref::M3 J = ref::jacobian(x, 2, 1);
  double Mv[18], N[2];
  for (int k = 0; k < 9; ++k) {
    Mv[k] = la[k];
    Mv[9 + k] = lb[k];
  }
  ref::edge_shape_values(xi, N);
  const ref::M3 Q = ref::log_transform(Mv, N, 2, ok);
  return ref::jacobian_det(ref::mul(J, Q), 1);
}

// MetricSizeField::measure under LogAnisoSizeField (ma/maSize.cc:158-216,
// 508-523): two Gauss points, the ends' log-metrics la, lb interpolated.
// Entries above 200 in magnitude (sizes beyond e^-100: the absolute deflation
// test is then near the rounding) or not finite, a first column the
// reduction would leave alone (below 1e-10, not 0), and squared lengths outside
// [2^-600, 2^600] or not finite (edges with infinite, huge or equal ends) take
// the sequence itself.
__device__ __forceinline__ double log_metric_length(const ref::V3& x0, const ref::V3& x1,
                                                    const double* __restrict__ la, const double* __restrict__ lb,
                                                    bool* ok) {
  const double gp[2] = {0.577350269189626, -0.577350269189626};
  const int at[6] = {0, 3, 6, 4, 7, 8};  // the lower triangle by columns
  const ref::V3 d = ref::sub(x1, x0);
  double L = 0;
#pragma unroll 1
  for (int p = 0; p < 2; ++p) {
    double N[2], a[6];
    ref::edge_shape_values(gp[p], N);
    double big = 0;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      a[k] = la[at[k]] * N[0] + lb[at[k]] * N[1];
      big = fmax(big, fabs(a[k]));
    }
    double s;
    const double col = fmax(fabs(a[1]), fabs(a[2]));
    const bool fast = big <= 200.0 && a[0] == a[0] && a[1] == a[1] && a[2] == a[2] && a[3] == a[3] && a[4] == a[4] &&
                      a[5] == a[5] && (a[2] == 0.0 || col >= 1e-10);
    const int status = fast ? log_length2(a, d, &s) : 0;
    if (fast && (unsigned)(bexp(s) - 423) <= 1200u) {
      if (status != 1) *ok = false;
      L += 0.5 * sqrt(s);
    } else {
      L += log_point_ref(x0, x1, la, lb, gp[p], ok);
    }
  }
  return L;
}

}  // namespace sprg
