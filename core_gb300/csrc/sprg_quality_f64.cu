// FP64 mean-ratio qualities (measureTetQuality / measureTriQuality with
// useMax = true, ma/maQuality.cc:83-167) under isotropic, anisotropic and
// log-interpolated size fields.  Compiled with -fmad=false; the calls' qualities
// are bitwise the reference's sequence, the anisotropic pass's on triangles
// (PASS) as near the exact values.
#include "sprg_internal.h"
#include "sprg_metric_f64.cuh"

namespace sprg {

using ref::M3;
using ref::V3;

namespace {

constexpr int kBlock = 256;
constexpr int kXf = 10;  // doubles of a vertex's transform record: Q row-major, then its determinant

inline int nblk(long n, int b = kBlock) { return (int)((n + b - 1) / b); }

__device__ __forceinline__ V3 load_xyz(const double* __restrict__ xyz, int v) {
  return V3{{xyz[3 * (size_t)v], xyz[3 * (size_t)v + 1], xyz[3 * (size_t)v + 2]}};
}

// the transform at a vertex: the size field interpolated with N = {1}
__device__ __noinline__ void aniso_transform_ref(const double* h, const double* R, M3* Q) {
  const double N[1] = {1.0};
  *Q = ref::get_transform(h, R, N, 1);
}

__device__ __forceinline__ M3 aniso_transform(const double* __restrict__ sizes, const double* __restrict__ frames,
                                              int v) {
  double h[3], R[9];
#pragma unroll
  for (int k = 0; k < 3; ++k) h[k] = __ldg(sizes + 3 * (size_t)v + k);
#pragma unroll
  for (int k = 0; k < 9; ++k) R[k] = __ldg(frames + 9 * (size_t)v + k);
  M3 Q;
  if (!ordinary(h[0]) || !ordinary(h[1]) || !ordinary(h[2])) {
    aniso_transform_ref(h, R, &Q);
  } else if (all_zero(R[2], R[5], R[6], R[7])) {
    double q[4];
    const double z = planar_transform(h[0], h[1], R[0], R[1], R[3], R[4], q);
    Q = M3{{{q[0], q[1], 0.0}, {q[2], q[3], 0.0}, {0.0, 0.0, z * (1 / h[2])}}};
  } else {
    M3 f;
#pragma unroll
    for (int k = 0; k < 9; ++k) f.m[k / 3][k % 3] = R[k];
    Q = transform_of(h, f);
  }
  return Q;
}

__device__ __noinline__ M3 log_transform_at(const double* logm, bool* ok) {
  const double N[1] = {1.0};
  return ref::log_transform(logm, N, 1, ok);
}

template <bool LOG>
__device__ __forceinline__ M3 vertex_transform(const double* __restrict__ sizes, const double* __restrict__ frames,
                                               const double* __restrict__ logm, int v, bool* ok) {
  if (LOG) return log_transform_at(logm + 9 * (size_t)v, ok);
  return aniso_transform(sizes, frames, v);
}

// Every vertex's transform once, instead of once per element around it (six
// triangles, 24 tets).  bad: the log-metric's eigen iteration failed.
template <int D, bool LOG>
__global__ void __launch_bounds__(kBlock) k_vertex_transforms(int V, const double* __restrict__ sizes,
                                                              const double* __restrict__ frames,
                                                              const double* __restrict__ logm,
                                                              double* __restrict__ xf,
                                                              unsigned char* __restrict__ bad) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= V) return;
  bool ok = true;
  const M3 Q = vertex_transform<LOG>(sizes, frames, logm, v, &ok);
  double* o = xf + kXf * (size_t)v;
#pragma unroll
  for (int k = 0; k < 9; ++k) o[k] = Q.m[k / 3][k % 3];
  o[9] = ref::jacobian_det(Q, D);
  if (LOG) bad[v] = !ok;
}

// the reference's sequence for one element under the transform Q
__device__ __forceinline__ double q_measure(const V3* x, int nn, int edim, const M3& Q) {
  M3 J = ref::jacobian(x, nn, edim);
  double w = edim == 3 ? 1.0 / 6.0 : (edim == 2 ? 1.0 / 2.0 : 2.0);
  double dV2 = ref::jacobian_det(ref::mul(J, Q), edim);
  double measurement = 0;
  measurement += w * dV2;
  return measurement;
}

__constant__ int c_edges[6][2] = {{0, 1}, {1, 2}, {2, 0}, {0, 3}, {1, 3}, {2, 3}};  // triangles: the first three

template <int D>
__device__ __forceinline__ double ratio_of(double Vm, double s) {
  if (D == 2) return 48 * (Vm * Vm) / (s * s);
  if (Vm < 0) return -15552 * (Vm * Vm) / (s * s * s);
  return 15552 * (Vm * Vm) / (s * s * s);
}

template <int D>
__device__ __noinline__ double quality_ref(const V3* x, const M3* Q) {
  double s = 0;
  for (int i = 0; i < (D == 3 ? 6 : 3); ++i) {
    const V3 xe[2] = {x[c_edges[i][0]], x[c_edges[i][1]]};
    const double l = q_measure(xe, 2, 1, *Q);
    s += l * l;
  }
  return ratio_of<D>(q_measure(x, D + 1, D, *Q), s);
}

// the edge vector d in metric space
__device__ __forceinline__ V3 to_metric(const V3& d, const M3& Q) {
  V3 e;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    double t = d.v[0] * Q.m[0][j];
    t += d.v[1] * Q.m[1][j];
    t += d.v[2] * Q.m[2][j];
    e.v[j] = t;
  }
  return e;
}

// Quality from the metric edge vectors of vertex 0 (e[0..D-1], the rows of
// the element's J Q) and of the others (o: 1-2, then 1-3 and 2-3): each edge
// length is the vector's own (the reference halves the vector and doubles the
// length, exactly).  *s returns the sum of squared lengths for the range check.
template <int D>
__device__ __forceinline__ double quality_of(const V3* e, const V3* o, double* s) {
  auto add = [&](double acc, const V3& v) {
    const double l = ref::len(v);
    return acc + l * l;
  };
  double acc = add(0.0, e[0]);
  acc = add(acc, o[0]);
  acc = add(acc, e[1]);
  if (D == 3) {
    acc = add(acc, e[2]);
    acc = add(acc, o[1]);
    acc = add(acc, o[2]);
  }
  *s = acc;
  double dV;
  if (D == 3) {
    const M3 a{{{e[0].v[0], e[0].v[1], e[0].v[2]}, {e[1].v[0], e[1].v[1], e[1].v[2]}, {e[2].v[0], e[2].v[1], e[2].v[2]}}};
    dV = ref::det3(a);
  } else {
    dV = ref::len(ref::cross(e[0], e[1]));
  }
  return ratio_of<D>((D == 3 ? 1.0 / 6.0 : 1.0 / 2.0) * dV, acc);
}

// PASS: the anisotropic passes' qualities: the squared lengths as they are,
// without the reference's root and square of each, the third edge as a sum,
// fused products (about 40 FP64 operations a triangle of 115).  Against extended
// precision 2.2 to 2.5 units of 2^-53 off (rms; sizes 1:2 to 1:500000 apart), the
// sequence 2.7 to 3.0.
template <int D, bool PASS>
__device__ __forceinline__ double element_quality(const V3* x, const M3& Q) {
  double s, r;
  auto same = [](double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); };
  if (D == 2 && all_zero(Q.m[0][2], Q.m[1][2], Q.m[2][0], Q.m[2][1]) && same(x[1].v[2], x[0].v[2]) &&
      same(x[2].v[2], x[0].v[2])) {
    // an element and frames in a z = const plane: the 2 x 2 block alone
    if constexpr (PASS) {
      const double ax = x[1].v[0] - x[0].v[0], ay = x[1].v[1] - x[0].v[1], bx = x[2].v[0] - x[1].v[0],
                   by = x[2].v[1] - x[1].v[1];
      const double ux = fma(ax, Q.m[0][0], ay * Q.m[1][0]), uy = fma(ax, Q.m[0][1], ay * Q.m[1][1]);
      const double vx = fma(bx, Q.m[0][0], by * Q.m[1][0]), vy = fma(bx, Q.m[0][1], by * Q.m[1][1]);
      const double wx = ux + vx, wy = uy + vy;  // edge 0-2
      s = fma(ux, ux, fma(uy, uy, fma(vx, vx, fma(vy, vy, fma(wx, wx, wy * wy)))));
      const double z = fma(ux, vy, -(uy * vx));  // twice the metric area
      r = 12 * (z * z) / (s * s);
    } else {
      double acc = 0, ex[3], ey[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {  // edges 0-1, 1-2, 0-2
        const int p = i == 1 ? 1 : 0, q = i == 0 ? 1 : 2;
        const double dx = x[q].v[0] - x[p].v[0], dy = x[q].v[1] - x[p].v[1];
        ex[i] = dx * Q.m[0][0] + dy * Q.m[1][0];
        ey[i] = dx * Q.m[0][1] + dy * Q.m[1][1];
        const double l = sqrt(ex[i] * ex[i] + ey[i] * ey[i]);
        acc += l * l;
      }
      s = acc;
      const double z = ex[0] * ey[2] - ey[0] * ex[2];
      // |z| = sqrt(z^2) while the square neither under- nor overflows
      const double dV = (unsigned)(bexp(z) - 623) <= 800u ? fabs(z) : sqrt(z * z);
      r = ratio_of<2>(0.5 * dV, acc);
    }
  } else {
    V3 e[3], o[3];
#pragma unroll
    for (int k = 0; k < D; ++k) e[k] = to_metric(ref::sub(x[k + 1], x[0]), Q);
    o[0] = to_metric(ref::sub(x[2], x[1]), Q);
    if (D == 3) {
      o[1] = to_metric(ref::sub(x[3], x[1]), Q);
      o[2] = to_metric(ref::sub(x[3], x[2]), Q);
    }
    r = quality_of<D>(e, o, &s);
  }
  if ((unsigned)(bexp(s) - 423) > 1200u) return quality_ref<D>(x, &Q);  // s outside [2^-600, 2^600]
  return r;
}

// Anisotropic and log-interpolated fields: the element takes the transform of
// its vertex with the largest determinant (the first such).  PRE: from the
// vertices' records, else (no memory for them) computed in place.
// FP64-rate bound: 1024^2 square, both kernels 0.34 ms in the pass and 0.58 in
// the calls, against 3.25 ms with every transform computed per element and the
// full 3 x 3 products.
template <int D, bool LOG, bool PRE, bool PASS = false>
__global__ void __launch_bounds__(kBlock) k_quality(DevMesh m, const double* __restrict__ sizes,
                                                    const double* __restrict__ frames,
                                                    const double* __restrict__ logm, const double* __restrict__ xf,
                                                    const unsigned char* __restrict__ bad, double* __restrict__ q,
                                                    DevStatus* st) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m.T) return;
  int id[D + 1];
#pragma unroll
  for (int a = 0; a <= D; ++a) id[a] = __ldg(m.ev + (size_t)(D + 1) * e + a);
  M3 Q;
  double maxJ = -1.0;
  int pick = -1;
  bool failed = false;
  if constexpr (!PRE)
    Q = M3{};
#pragma unroll
  for (int a = 0; a <= D; ++a) {
    if constexpr (PRE) {
      const double cj = __ldg(xf + kXf * (size_t)id[a] + 9);
      bool larger;
      if constexpr (D == 2) {  // a length: not negative, ordered as its bits (a NaN is past infinity's)
        const long long b = __double_as_longlong(cj);
        larger = (unsigned long long)b <= 0x7ff0000000000000ull && (pick < 0 || b > __double_as_longlong(maxJ));
      } else {
        larger = cj > maxJ;
      }
      if (larger) {
        maxJ = cj;
        pick = id[a];
      }
      if (LOG) failed = failed || bad[id[a]];
    } else {
      bool ok = true;
      const M3 c = vertex_transform<LOG>(sizes, frames, logm, id[a], &ok);
      failed = failed || !ok;
      const double cj = ref::jacobian_det(c, D);
      if (cj > maxJ) {
        maxJ = cj;
        Q = c;
      }
    }
  }
  if (LOG && failed && atomicCAS(&st->code, 0, SPRG_EEIGEN) == 0) st->where = e;
  if constexpr (PRE) {
#pragma unroll
    for (int k = 0; k < 9; ++k) Q.m[k / 3][k % 3] = pick < 0 ? 0.0 : __ldg(xf + kXf * (size_t)pick + k);
  }
  V3 x[D + 1];
#pragma unroll
  for (int a = 0; a <= D; ++a) x[a] = load_xyz(m.xyz, id[a]);
  q[e] = element_quality<D, PASS>(x, Q);
}

template <int D>
__device__ __noinline__ double iso_quality_ref(const V3* x, const double* sz) {
  M3 Q{};
  double maxJ = -1.0;
  const double N[1] = {1.0};
  for (int a = 0; a <= D; ++a) {
    const double h[3] = {sz[a], sz[a], sz[a]};
    double R[9];
    identity9(R);
    const M3 c = ref::get_transform(h, R, N, 1);
    const double cj = ref::jacobian_det(c, D);
    if (cj > maxJ) {
      maxJ = cj;
      Q = c;
    }
  }
  return quality_ref<D>(x, &Q);
}

// Isotropic field: the transform is 1 / h on the diagonal and the vertex with
// the largest determinant the one with the smallest size.  Sizes whose high
// words differ by more than one are ordered by them; closer ones by the
// determinants themselves (RN(i RN(i i)) in space, RN(i i) in the plane),
// whose rounding may make two sizes equal.  Sizes that are not ordinary
// positive numbers take the sequence itself.
template <int D>
__global__ void __launch_bounds__(kBlock) k_quality_iso(DevMesh m, const double* __restrict__ size,
                                                        double* __restrict__ q) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m.T) return;
  int id[D + 1];
  double sz[D + 1];
  V3 x[D + 1];
  bool fine = true;
#pragma unroll
  for (int a = 0; a <= D; ++a) {
    id[a] = __ldg(m.ev + (size_t)(D + 1) * e + a);
    sz[a] = __ldg(size + id[a]);
    fine = fine && ordinary(sz[a]) && __double2hiint(sz[a]) > 0;
  }
#pragma unroll
  for (int a = 0; a <= D; ++a) x[a] = load_xyz(m.xyz, id[a]);
  double r = 0, s = 0;
  if (fine) {
    auto det = [](double h) {
      const double i = __drcp_rn(h);
      return D == 3 ? i * (i * i) : i * i;
    };
    double h = sz[0];
#pragma unroll
    for (int a = 1; a <= D; ++a) {
      const int gap = __double2hiint(h) - __double2hiint(sz[a]);
      if (gap > 1 || (gap >= -1 && det(sz[a]) > det(h))) h = sz[a];
    }
    const double i = __drcp_rn(h);
    V3 ev[3], o[3];
#pragma unroll
    for (int k = 0; k < D; ++k) ev[k] = ref::scale(ref::sub(x[k + 1], x[0]), i);
    o[0] = ref::scale(ref::sub(x[2], x[1]), i);
    if (D == 3) {
      o[1] = ref::scale(ref::sub(x[3], x[1]), i);
      o[2] = ref::scale(ref::sub(x[3], x[2]), i);
    }
    r = quality_of<D>(ev, o, &s);
  }
  if (!fine || (unsigned)(bexp(s) - 423) > 1200u) r = iso_quality_ref<D>(x, sz);
  q[e] = r;
}

}  // namespace

size_t vertex_transform_bytes(int V) { return sizeof(double) * kXf * (size_t)V; }

void launch_quality_f64(const DevMesh& m, const double* size, const double* sizes, const double* frames,
                        const double* logm, double* xf, unsigned char* bad, bool pass, double* q, DevStatus* st,
                        cudaStream_t s) {
  if (!m.T) return;
  const int ge = nblk(m.T), gv = nblk(m.V);
  if (size) {
    if (m.dim == 3) k_quality_iso<3><<<ge, kBlock, 0, s>>>(m, size, q);
    else k_quality_iso<2><<<ge, kBlock, 0, s>>>(m, size, q);
    return;
  }
  auto transforms = [&](auto kernel) { kernel<<<gv, kBlock, 0, s>>>(m.V, sizes, frames, logm, xf, bad); };
  auto quality = [&](auto kernel) { kernel<<<ge, kBlock, 0, s>>>(m, sizes, frames, logm, xf, bad, q, st); };
  if (m.dim == 3) {
    if (xf) transforms(logm ? k_vertex_transforms<3, true> : k_vertex_transforms<3, false>);
    if (logm) quality(xf ? k_quality<3, true, true> : k_quality<3, true, false>);
    else quality(xf ? k_quality<3, false, true> : k_quality<3, false, false>);
  } else {
    if (xf) transforms(logm ? k_vertex_transforms<2, true> : k_vertex_transforms<2, false>);
    if (logm) quality(xf ? k_quality<2, true, true> : k_quality<2, true, false>);
    else quality(!xf ? k_quality<2, false, false> : pass ? k_quality<2, false, true, true> : k_quality<2, false, true>);
  }
}

}  // namespace sprg
