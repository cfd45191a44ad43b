// FP64 element and edge kernels of the parity form: the per-mesh element records,
// the integration-point gradients taken from them, errors and sizes, lengths.
//
// Compiled with -fmad=false.  Records, gradients and the lengths of given sizes
// are bitwise the reference's operation order (sprg_refmath.cuh): operations
// whose result the reference's own sequence fixes in advance are left out
// (products with the shape gradients' 0, 1 and -1, sums with 0), and quotients by
// one common divisor come from its rounded reciprocal with exact residuals.
// Errors and their powers (k_error) and the pass's lengths (k_measure_mark) are
// sums and quotients in an order of their own, with fused operations.
#include "sprg_internal.h"
#include "sprg_metric_f64.cuh"
#include "sprg_reduce.cuh"

namespace sprg {

using ref::M3;
using ref::V3;

namespace {

constexpr int kBlock = 256;

inline int nblk(long n, int b = kBlock) { return (int)((n + b - 1) / b); }

__device__ __forceinline__ V3 load_xyz(const double* __restrict__ xyz, int v) {
  return V3{{xyz[3 * (size_t)v], xyz[3 * (size_t)v + 1], xyz[3 * (size_t)v + 2]}};
}

template <int D>
__device__ __forceinline__ void load_ids(const int* __restrict__ ev, int e, int* id) {
  if (D == 3) {
    const int4 t = __ldg(reinterpret_cast<const int4*>(ev) + e);
    id[0] = t.x; id[1] = t.y; id[2] = t.z; id[3] = t.w;
  } else {
    for (int a = 0; a < 3; ++a) id[a] = __ldg(ev + 3 * (size_t)e + a);
  }
}

// One element's geometry: the rows of J^-1 (D columns each; the third column
// of a triangle's pseudo-inverse is 0), dV = det J, and the longest edge
// (apf::measure).  Record planes: J^-1 row-major (3 D planes), dV, h, and on
// tets the first vertex's shape gradient (the negated row sums); plane k of
// element e at k T + e.
template <int D>
struct ElemRec {
  static constexpr int kPlanes = 3 * D + (D == 3 ? 5 : 2);
  double v[kPlanes];
};

// the reference's own sequence; a row of J^-1 with a value that is not finite
// becomes all NaN (the reference multiplies every row by shape gradients
// that contain 0, so its gradients' component is NaN there)
template <int D>
__device__ __noinline__ void elem_record_ref(const V3* x, double* out) {
  const M3 J = ref::jacobian(x, D + 1, D);
  const M3 ji = ref::jacobian_inverse(J, D);
  for (int i = 0; i < 3; ++i) {
    bool fine = true;
    for (int j = 0; j < D; ++j) fine = fine && bexp(ji.m[i][j]) != 0x7ff;
    for (int j = 0; j < D; ++j) out[D * i + j] = fine ? ji.m[i][j] : __longlong_as_double(0x7ff8000000000000ll);
  }
  out[3 * D] = ref::jacobian_det(J, D);
  double h = 0;
  for (int p = 0; p <= D; ++p)
    for (int q = p + 1; q <= D; ++q) {
      const V3 xe[2] = {x[p], x[q]};
      const M3 Je = ref::jacobian(xe, 2, 1);
      double l = 0;
      l += 2 * ref::jacobian_det(Je, 1);
      h = (h < l) ? l : h;
    }
  out[3 * D + 1] = h;
}

// Tets: J is three coordinate differences (the shape gradients are 0, 1 and
// -1), the determinant reuses the first row of cofactors, the nine quotients
// share one reciprocal, and the longest edge takes one square root (rounding
// is monotone): about 150 FP64 operations against 450 written out.
// Exponents outside the safe range (degenerate, inverted to nothing, not
// finite) take the sequence itself.
__device__ __forceinline__ void tet_record(const V3* x, double* out) {
  double m[3][3];
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int k = 0; k < 3; ++k) m[r][k] = x[r + 1].v[k] - x[0].v[k];
  V3 col[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) col[k] = V3{{m[0][k], m[1][k], m[2][k]}};
  const V3 c0 = ref::cross(col[1], col[2]), c1 = ref::cross(col[2], col[0]), c2 = ref::cross(col[0], col[1]);
  double det = m[0][0] * c0.v[0];
  det += m[1][0] * c0.v[1];
  det += m[2][0] * c0.v[2];
  // an exponent check per quotient: the divisor in [2^-400, 2^400], the
  // dividend 0 or in [2^-500, 2^500]
  bool safe = bexp(det) >= 623 && bexp(det) <= 1423;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double c[3] = {c0.v[k], c1.v[k], c2.v[k]};
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const int ex = bexp(c[r]);
      safe = safe && ex <= 1523 && (ex >= 523 || c[r] == 0.0);
    }
  }
  double hh = 0;
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    const double d = m[r][0] * m[r][0] + m[r][1] * m[r][1] + m[r][2] * m[r][2];
    hh = (hh < d) ? d : hh;
  }
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    const int p = 1 + r, q = 1 + (r + 1) % 3;
    const double a = x[q].v[0] - x[p].v[0], b = x[q].v[1] - x[p].v[1], c = x[q].v[2] - x[p].v[2];
    const double d = a * a + b * b + c * c;
    hh = (hh < d) ? d : hh;
  }
  if (!safe || bexp(hh) > 2000) {
    elem_record_ref<3>(x, out);
    return;
  }
  const double y = __drcp_rn(det);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    out[k] = quotient(c0.v[k], det, y);
    out[3 + k] = quotient(c1.v[k], det, y);
    out[6 + k] = quotient(c2.v[k], det, y);
  }
  out[9] = det;
  out[10] = sqrt(hh);
}

template <int D>
__device__ __forceinline__ void elem_record_of(const DevMesh& m, const int* id, double* out) {
  V3 x[D + 1];
#pragma unroll
  for (int a = 0; a <= D; ++a) x[a] = load_xyz(m.xyz, id[a]);
  if constexpr (D == 3) {
    tet_record(x, out);
#pragma unroll
    for (int r = 0; r < 3; ++r) out[11 + r] = -out[3 * r] - out[3 * r + 1] - out[3 * r + 2];
  } else {
    elem_record_ref<D>(x, out);
  }
}

// per mesh; FP64-rate bound (the operations above), 8 kPlanes bytes written
template <int D>
__global__ void __launch_bounds__(kBlock) k_elem_records(DevMesh m, double* __restrict__ geo) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m.T) return;
  int id[D + 1];
  load_ids<D>(m.ev, e, id);
  double r[ElemRec<D>::kPlanes];
  elem_record_of<D>(m, id, r);
#pragma unroll
  for (int k = 0; k < ElemRec<D>::kPlanes; ++k) geo[(size_t)k * m.T + e] = r[k];
}

// per mesh: the gradients of the listed patches' elements, a warp per patch
__global__ void __launch_bounds__(kBlock) k_listed_records(DevMesh m, PatchWeights pw, double* __restrict__ g) {
  const int it = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (it >= pw.n) return;
  for (int i = lane; i < pw.wn[it]; i += 32) {
    int id[4];
    load_ids<3>(m.ev, pw.el[(size_t)it * pw.stride + i], id);
    double r[ElemRec<3>::kPlanes];
    elem_record_of<3>(m, id, r);
    double* o = g + 12 * (pw.woff[it] + i);
#pragma unroll
    for (int k = 0; k < 9; ++k) o[k] = r[k];
#pragma unroll
    for (int k = 0; k < 3; ++k) o[9 + k] = r[11 + k];
  }
}

// ---------------------------------------------------------------------
// spr::getGradIPField (spr/sprGetGradIPField.cc:15-65): the gradients of the
// shape functions are J^-1's columns and, for the first vertex, the negated
// sum of each row (the reference's products with 1, 0 and -1); the sums over
// the vertices keep its order.  With the per-mesh records a scalar field
// costs 21 FP64 operations and 136 bytes a tet, 0.22 ms for the 5.3M tets of
// a 96^3 box (3.3 TB/s; 0.28 ms with the first vertex's gradients summed here,
// 27 operations and 112 bytes) against 2.76 ms with the sequence written out; without them (no memory for the records) they are
// computed in place.
// ---------------------------------------------------------------------
template <int D, int NC, bool REC>
__global__ void __launch_bounds__(kBlock) k_grad_ip(DevMesh m, const double* __restrict__ geo,
                                                    const double* __restrict__ f, double* __restrict__ ip) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m.T) return;
  int id[D + 1];
  load_ids<D>(m.ev, e, id);
  double j[ElemRec<D>::kPlanes];
  if constexpr (REC) {
#pragma unroll
    for (int k = 0; k < 3 * D; ++k) j[k] = __ldcs(geo + (size_t)k * m.T + e);
    if (D == 3)
#pragma unroll
      for (int k = 0; k < 3; ++k) j[ElemRec<D>::kPlanes - 3 + k] = __ldcs(geo + (size_t)(11 + k) * m.T + e);
  } else {
    elem_record_of<D>(m, id, j);
  }
  double u[D + 1][NC];
#pragma unroll
  for (int a = 0; a <= D; ++a)
#pragma unroll
    for (int c = 0; c < NC; ++c) u[a][c] = __ldg(f + (size_t)id[a] * NC + c);
  // a triangle in a z = const plane: the z row of J^-1 is 0, and so are its
  // gradients of finite values
  bool flat = false;
  if (D == 2 && all_zero(j[2 * D], j[2 * D + 1], 0.0, 0.0)) {
    flat = true;
#pragma unroll
    for (int a = 0; a <= D; ++a)
#pragma unroll
      for (int c = 0; c < NC; ++c) flat = flat && bexp(u[a][c]) != 0x7ff;
  }
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    if (D == 2 && r == 2 && flat) {
      for (int c = 0; c < NC; ++c) ip[(size_t)e * 3 * NC + NC * r + c] = 0.0;
      break;
    }
    if (D == 2 && r == 2) asm volatile("");  // a branch, not selects
    const double g0 = D == 3 ? j[ElemRec<D>::kPlanes - 3 + r] : -j[D * r] - j[D * r + 1];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      double g = g0 * u[0][c];
#pragma unroll
      for (int k = 0; k < D; ++k) g += j[D * r + k] * u[k + 1][c];
      ip[(size_t)e * 3 * NC + NC * r + c] = g;
    }
  }
}

// ---------------------------------------------------------------------
// Element errors (SelfProduct / ElementError, spr/sprEstimateError.cc:98-170)
// and the powers of them the size field takes.
// ---------------------------------------------------------------------
// Per element: err = |eps - eps*(IP)|^2 w dV, and in
// esize h err^(-1/(D+2)) (mode 0; the size factor follows in k_esize) or the
// power alone (mode 1).  The two integrals are summed per thread over a fixed
// grid, then per block in a fixed order; with `done` (zero between launches)
// the last block also reduces the blocks' partials and computes the size
// factor.  FP64-rate bound: about 34 operations a tet, 0.34 ms at 5.3M tets
// (2.36 ms with pow, the Jacobian and one tree reduction per 256 elements).
template <int D, int NC, bool REC>
__global__ void __launch_bounds__(kBlock) k_error(DevMesh m, const double* __restrict__ geo,
                                                  const double* __restrict__ ip, const double* __restrict__ rec,
                                                  double* __restrict__ err, double* __restrict__ esize,
                                                  double* __restrict__ partials, unsigned* __restrict__ done, int mode,
                                                  double adapt_ratio, double target, double* __restrict__ out3) {
  after_previous(geo, ip, rec);
  __shared__ double sh[2 * (kBlock / 32)];
  double self_sum = 0, g_sum = 0;
  double N[4];
  ref::ip_shape_values(D, N);
  const double w = ref::ip_weight(D);
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < m.T; e += gridDim.x * blockDim.x) {
    int id[D + 1];
    load_ids<D>(m.ev, e, id);
    double dV, h;
    if constexpr (REC) {
      dV = __ldcs(geo + (size_t)(3 * D) * m.T + e);
      h = __ldcs(geo + (size_t)(3 * D + 1) * m.T + e);
    } else {
      double r[ElemRec<D>::kPlanes];
      elem_record_of<D>(m, id, r);
      dV = r[3 * D];
      h = r[3 * D + 1];
    }
    double vv = 0, dd = 0;
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      const double b = __ldcs(ip + (size_t)e * NC + k);
      double v2 = __ldg(rec + (size_t)id[0] * NC + k), dv;
      if (D == 3) {
        // every shape value is 1/4: v2 is four times the value here (exact), the
        // sixteenth of its square is taken once per thread
#pragma unroll
        for (int a = 1; a <= D; ++a) v2 += __ldg(rec + (size_t)id[a] * NC + k);
        dv = fma(-0.25, v2, b);
      } else {
        v2 *= N[0];
#pragma unroll
        for (int a = 1; a <= D; ++a) v2 += __ldg(rec + (size_t)id[a] * NC + k) * N[a];
        dv = b - v2;
      }
      vv = fma(v2, v2, vv);
      dd = fma(dv, dv, dd);
    }
    const double wdv = w * dV, er = dd * wdv;
    self_sum = fma(vv, wdv, self_sum);
    err[e] = er;
    double q, g;
    error_powers<D>(er, q, g);
    g_sum += g;
    esize[e] = mode == 0 ? h * q : q;
  }
  if (D == 3) self_sum *= 0.0625;
  double s1 = self_sum, s2 = g_sum;
  rd_block_sum2(s1, s2, sh);
  if (threadIdx.x == 0) {
    partials[2 * blockIdx.x] = s1;
    partials[2 * blockIdx.x + 1] = s2;
  }
  if (!done) return;
  __shared__ bool last;
  if (threadIdx.x == 0) {
    __threadfence();  // this block's partials before its count
    last = atomicAdd(done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  rd_size_factor(partials, gridDim.x, mode, adapt_ratio, target, D, out3, sh);
  if (threadIdx.x == 0) *done = 0;
}

// element sizes from the size factor, in place: h err^(-1/(D+2)) sf
// (getSPRSizeField), or the clamped target size (getTargetSPRSizeField)
template <int D, bool REC>
__global__ void __launch_bounds__(kBlock) k_esize(DevMesh m, const double* __restrict__ geo,
                                                  const double* __restrict__ out3, int mode, double alpha, double beta,
                                                  double* __restrict__ esize) {
  after_previous(geo, out3, esize);
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m.T) return;
  const double sf = out3[2];
  if (mode == 0) {
    esize[e] = esize[e] * sf;
    return;
  }
  double h;
  if constexpr (REC) {
    h = __ldcs(geo + (size_t)(3 * D + 1) * m.T + e);
  } else {
    int id[D + 1];
    load_ids<D>(m.ev, e, id);
    double r[ElemRec<D>::kPlanes];
    elem_record_of<D>(m, id, r);
    h = r[3 * D + 1];
  }
  double h_new = sf * esize[e] * h;
  if (h_new < alpha * h) h_new = alpha * h;
  if (h_new > beta * h) h_new = beta * h;
  esize[e] = h_new;
}

__global__ void __launch_bounds__(kBlock) k_average(DevMesh m, const double* __restrict__ esize,
                                                    double* __restrict__ size) {
  after_previous(esize);
  int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= m.V) return;
  int b = m.a_off[v], e = m.a_off[v + 1];
  double s = 0;
  for (int k = b; k < e; ++k) s += esize[m.a_el[k]];
  s /= (double)(size_t)(e - b);
  size[v] = s;
}

// ---------------------------------------------------------------------
// Isotropic edge lengths (ma::makeSizeField(m, size) + measure)
// ---------------------------------------------------------------------
// given sizes: the lengths themselves, bitwise
__global__ void __launch_bounds__(kBlock) k_measure_iso(DevMesh m, const double* __restrict__ size,
                                                        double* __restrict__ L) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m.E) return;
  const int2 v = __ldg(reinterpret_cast<const int2*>(m.edv) + e);
  L[e] = iso_length(load_xyz(m.xyz, v.x), load_xyz(m.xyz, v.y), __ldg(size + v.x), __ldg(size + v.y));
}

// half an edge's Euclidean length
__device__ __forceinline__ double half_length(const DevMesh& m, int2 v) {
  const V3 d = ref::sub(load_xyz(m.xyz, v.y), load_xyz(m.xyz, v.x));
  return 0.5 * sqrt(fma(d.v[0], d.v[0], fma(d.v[1], d.v[1], d.v[2] * d.v[2])));
}

// per mesh: half the edges' Euclidean lengths
__global__ void __launch_bounds__(kBlock) k_edge_records(DevMesh m, double* __restrict__ len) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m.E) return;
  const int2 v = __ldg(reinterpret_cast<const int2*>(m.edv) + e);
  len[e] = half_length(m, v);
}

// The pass's lengths and marks.  Only the marks leave the pass, so the lengths
// need not be the sequence's bits, but they are as near the exact ones (0.83
// units of 2^-53 rms, the sequence 0.83 to 0.84; (|d| / 2) (h0 + h1) / (h0 h1) as
// it stands 1.09): with the ends' sizes a, b
//   |d| / 2 (1 / h0 + 1 / h1) = |d| / 2 (a + b) / (a b + K (a - b)^2),  K = N0 N1,
// the quotient from the hardware's reciprocal (2^-20 at least) and one Newton
// step, its residual with the denominator's rounding corrected before the
// product: 15 FP64 operations with the per-mesh half lengths, 55 for the sequence.
// Sizes more than about 2.8 apart (K (a - b)^2 then carries two roundings of its
// own), lengths within 1e-6 of 0.5 or 1.5, and exponents outside [-300, 300] take
// iso_length, so every mark is that of the bitwise length.  The comparisons
// and windows are integer ones on the bits (FP64 comparisons use the FP64
// pipe).  96^3 box, 6.3M edges: 0.99 ms for the reference's sequence plus
// 0.03 ms for marking from the stored lengths, 0.18 ms here.
template <bool REC>
__global__ void __launch_bounds__(kBlock) k_measure_mark(DevMesh m, const double* __restrict__ len,
                                                         const double* __restrict__ size, double* __restrict__ L,
                                                         uint32_t* __restrict__ split,
                                                         uint32_t* __restrict__ collapse) {
  after_previous(len, size);
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  bool sp = false, co = false;
  if (e < m.E) {
    const int2 v = __ldg(reinterpret_cast<const int2*>(m.edv) + e);
    const double sa = __ldg(size + v.x), sb = __ldg(size + v.y);
    double d;
    if constexpr (REC) d = __ldcs(len + e);
    else d = half_length(m, v);
    const double K = (1.0 - 0.577350269189626) / 2.0 * ((1.0 + 0.577350269189626) / 2.0);
    const double sum = sa + sb, df = sa - sb, p = K * df * df, den = fma(sa, sb, p);
    const double den_err = fma(sa, sb, -den) + p;
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(den));
    y = fma(y, fma(-den, y, 1.0), y);
    const double q = sum * y, c = fma(-q, den_err, fma(-den, q, sum)) * y;
    double l = fma(d, q, d * c);
    const int ha = __double2hiint(sa), hb = __double2hiint(sb), e0 = ha >> 20, e1 = hb >> 20, hl = __double2hiint(l);
    // hl >> 20 is the biased exponent of a positive length, negative for a
    // negative one; 0x3ff80000 is 1.5's high word, 0x3fe00000 0.5's
    if (min(min(e0, e1), hl >> 20) < 723 || max(max(e0, e1), hl >> 20) > 1323 || abs(ha - hb) > 0x180000 ||
        (unsigned)(hl - 0x3ff7ffff) < 2u || (unsigned)(hl - 0x3fdfffff) < 2u) {
      l = iso_length(load_xyz(m.xyz, v.x), load_xyz(m.xyz, v.y), sa, sb);
      sp = l > 1.5;
      co = l < .5;
    } else {
      sp = hl > 0x3ff80000;
      co = hl < 0x3fdfffff;
    }
    L[e] = l;
  }
  const unsigned bs = __ballot_sync(0xffffffffu, sp), bc = __ballot_sync(0xffffffffu, co);
  if ((threadIdx.x & 31) == 0 && e < m.E) {
    split[e >> 5] = bs;
    collapse[e >> 5] = bc;
  }
}

// blocks of the error kernel: eight per SM, so that a thread takes several
// elements and the reductions stay a small share
constexpr int kErrorGrid = 152 * 8;

}  // namespace

int elem_record_planes(int dim) { return dim == 3 ? ElemRec<3>::kPlanes : ElemRec<2>::kPlanes; }

void launch_elem_records(const DevMesh& m, double* geo, cudaStream_t s) {
  if (!m.T) return;
  if (m.dim == 3) k_elem_records<3><<<nblk(m.T), kBlock, 0, s>>>(m, geo);
  else k_elem_records<2><<<nblk(m.T), kBlock, 0, s>>>(m, geo);
}

void launch_listed_records(const DevMesh& m, const PatchWeights& pw, double* g, cudaStream_t s) {
  if (pw.n) k_listed_records<<<nblk((long)pw.n * 32), kBlock, 0, s>>>(m, pw, g);
}

void launch_grad_ip_f64(const DevMesh& m, const double* geo, const double* f, int ncin, double* ip, cudaStream_t s) {
  if (!m.T) return;
  auto go = [&](auto kernel) { kernel<<<nblk(m.T), kBlock, 0, s>>>(m, geo, f, ip); };
  if (m.dim == 3) {
    if (ncin == 1) go(geo ? k_grad_ip<3, 1, true> : k_grad_ip<3, 1, false>);
    else go(geo ? k_grad_ip<3, 3, true> : k_grad_ip<3, 3, false>);
  } else {
    if (ncin == 1) go(geo ? k_grad_ip<2, 1, true> : k_grad_ip<2, 1, false>);
    else go(geo ? k_grad_ip<2, 3, true> : k_grad_ip<2, 3, false>);
  }
}

int error_blocks(int T) { return nblk(T) < kErrorGrid ? nblk(T) : kErrorGrid; }

void launch_error_f64(const DevMesh& m, const double* geo, const double* ip, int nc, const double* rec, double* err,
                      double* esize, double* partials, int n_blocks, unsigned* done, int mode, double adapt_ratio,
                      double target, double* out3, cudaStream_t s) {
  if (!n_blocks) return;
  auto go = [&](auto kernel) {
    launch_after(m.early, kernel, n_blocks, kBlock, s, m, geo, ip, rec, err, esize, partials, done, mode, adapt_ratio, target, out3);
  };
  if (m.dim == 3) {
    if (nc == 3) go(geo ? k_error<3, 3, true> : k_error<3, 3, false>);
    else go(geo ? k_error<3, 9, true> : k_error<3, 9, false>);
  } else {
    if (nc == 3) go(geo ? k_error<2, 3, true> : k_error<2, 3, false>);
    else go(geo ? k_error<2, 9, true> : k_error<2, 9, false>);
  }
}

void launch_esize_f64(const DevMesh& m, const double* geo, const double* out3, int mode, double alpha, double beta,
                      double* esize, cudaStream_t s) {
  if (!m.T) return;
  auto go = [&](auto kernel) { launch_after(m.early, kernel, nblk(m.T), kBlock, s, m, geo, out3, mode, alpha, beta, esize); };
  if (m.dim == 3) go(geo ? k_esize<3, true> : k_esize<3, false>);
  else go(geo ? k_esize<2, true> : k_esize<2, false>);
}

void launch_average(const DevMesh& m, const double* esize, double* size, cudaStream_t s) {
  if (m.V) launch_after(m.early, k_average, nblk(m.V), kBlock, s, m, esize, size);
}

void launch_measure_iso_f64(const DevMesh& m, const double* size, double* L, cudaStream_t s) {
  if (m.E) k_measure_iso<<<nblk(m.E), kBlock, 0, s>>>(m, size, L);
}

void launch_edge_records(const DevMesh& m, double* len, cudaStream_t s) {
  if (m.E) k_edge_records<<<nblk(m.E), kBlock, 0, s>>>(m, len);
}

void launch_measure_mark_f64(const DevMesh& m, const double* len, const double* size, double* L, uint32_t* split,
                             uint32_t* collapse, cudaStream_t s) {
  if (!m.E) return;
  launch_after(m.early, len ? k_measure_mark<true> : k_measure_mark<false>, nblk(m.E), kBlock, s, m, len, size, L, split, collapse);
}

}  // namespace sprg
