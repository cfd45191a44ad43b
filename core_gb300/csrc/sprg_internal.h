// Internal declarations shared by the CUDA translation units of the
// estimate-and-mark library.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <string>
#include <utility>

#include "spr_gb300.h"

namespace sprg {

// Device view of the flattened mesh.  All index arrays are int32.
struct DevMesh {
  int dim;             // 2 or 3
  int nn;              // vertices per element (dim + 1)
  int ne_el;           // edges per element (3 or 6)
  int V, T, E;
  const double* xyz;   // V x 3 (FP64 master copy)
  const int* xyzq;     // V x 4 (X, Y, Z, 0): 32-bit fixed point on the frame, the learned form's records
  const int* ev;       // T x nn  (getDownward(e,0) order)
  const int* edv;      // E x 2
  const int* p_off;    // V + 1, patch CSR: elements of each vertex, ascending
  const int* p_el;
  const int* a_off;    // V + 1, averaging CSR (reference getAdjacent order)
  const int* a_el;
  bool early;          // launches of this pass: see launch_after
};

// A batch of independent meshes flattened into one context (disjoint union,
// entity ids offset per mesh).  n = 0: a single mesh.  Per mesh k:
// vertices [voff[k], voff[k+1]); error-kernel segments [segoff[k],
// segoff[k+1]) of seg (element ranges that never cross a mesh); the size
// factor of mesh k at out3[4 k + 2].
struct BatchView {
  int n;
  const int* voff;
  const int2* seg;
  const int* segoff;
  const double* ratios;
};

// mesh of vertex v (binary search over the vertex offsets)
__device__ __forceinline__ int batch_mesh(const BatchView& b, int v) {
  int lo = 0, hi = b.n;  // voff[lo] <= v < voff[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(b.voff + mid) <= v) lo = mid;
    else hi = mid;
  }
  return lo;
}

// the size factor that applies at vertex v
__device__ __forceinline__ double batch_sf(const BatchView& b, const double* out3, int v) {
  return b.n ? out3[4 * batch_mesh(b, v) + 2] : out3[2];
}

// Programmatic dependent launch: a kernel launched with launch_after may be set
// up while the kernel before it on the stream drains; it calls
// after_previous() before it reads anything a kernel before it wrote.  On a
// small mesh the launch gaps are as long as the kernels.  The first statement
// lets the kernel after this one be set up in turn (once every block of this
// one has started), the second waits until the one before is complete and
// its writes are visible; both do nothing in an ordinary launch.
// early (DevMesh::early, set per pass): whether to.  Direct passes gain 14 to
// 18 us at 3k tets (FP32, learned, FP64), 13 at 1.6M and 7 at 3.1M (the host's
// launches and the kernels' set-up overlap), passes being captured into a
// graph 4 us at 3k and nothing from 0.5M; at 5.3M tets both lose 30 to 50 of
// about 300 us (waiting blocks take the slots that the tail of the kernel
// before would fill), so the lines lie at 3M and 1M tets.
// The kernel's inputs that a kernel before it (back to the last ordinary launch)
// wrote go through it: a pointer to const with __restrict__ is memory that does
// not change during the kernel, so the compiler may move its loads above the
// wait; values that come out of an asm behind it cannot be used earlier.
template <class... P>
__device__ __forceinline__ void after_previous(P&... p) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  (void)(([&] { asm volatile("" : "+l"(p)::"memory"); }(), 0) + ... + 0);
}
template <class... P, class... A>
inline void launch_after_smem(bool early, void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t s,
                              A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = early ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
template <class... P, class... A>
inline void launch_after(bool early, void (*kernel)(P...), int grid, int block, cudaStream_t s, A&&... args) {
  launch_after_smem(early, kernel, grid, block, 0, s, std::forward<A>(args)...);
}

// The vertex and lane of a thread where LANES consecutive threads take a vertex.
// 64 bits: a mesh may have 2^31 - 1 vertices, LANES times as many threads, and
// threads past the last.
struct VertexLane {
  long v;
  int lane;
};
template <int LANES>
__host__ __device__ inline VertexLane vertex_lane(unsigned block, int threads, int thread) {
  const long i = (long)block * threads + thread;
  return VertexLane{i / LANES, (int)(i % LANES)};
}

// Device status word written by kernels (first error wins).
struct DevStatus {
  int code;        // SPRG_OK or SPRG_E*
  int where;       // entity index that raised it
};

// The listed patches' per-mesh FP64 weights: n patches; patch it: vertex v[it],
// elements el + it stride, wn[it] weights at w + woff[it], or -1 where the
// growth or the rank test failed (SPRG_EPATCH in st).  g (tets, optional): with
// each weight its element's gradient, 12 doubles (J^-1 by rows, then the first
// vertex's shape gradient)
struct PatchWeights {
  int n, stride;
  const int* v;
  const int* el;
  const long long* woff;
  const double* w;
  const int* wn;
  const double* g;
  DevStatus* st;
};

// Expansion work list for patches that need growth or are too large for the
// register path.
struct ExpandList {
  int* items;   // vertex ids
  int* count;   // device counter
  int cap;
};

// ---- FP64 element kernels (sprg_elem_f64.cu) --------------------------
// per-mesh element records: elem_record_planes(dim) planes of T doubles
// (J^-1 row-major, D columns a row; det J; the longest edge; tets: the first
// vertex's shape gradient)
int elem_record_planes(int dim);
void launch_elem_records(const DevMesh& m, double* geo, cudaStream_t s);
// the gradients of the listed patches' elements into g (PatchWeights::g)
void launch_listed_records(const DevMesh& m, const PatchWeights& pw, double* g, cudaStream_t s);
// geo: the records, or null to compute them in place
void launch_grad_ip_f64(const DevMesh& m, const double* geo, const double* f, int ncin, double* ip, cudaStream_t s);
// per-element errors, their powers in esize (k_error) and deterministic block
// partials (2 per block, error_blocks(T) blocks); mode 0: SPR, 1: target.
// done (one unsigned, zero between launches): the last block also computes
// the size factor into out3, as launch_size_factor does; null: it does not
void launch_error_f64(const DevMesh& m, const double* geo, const double* ip, int nc, const double* rec, double* err,
                      double* esize, double* partials, int n_blocks, unsigned* done, int mode, double adapt_ratio,
                      double target, double* out3, cudaStream_t s);
int error_blocks(int T);
// element sizes, in place on the error kernel's esize
void launch_esize_f64(const DevMesh& m, const double* geo, const double* out3, int mode, double alpha, double beta,
                      double* esize, cudaStream_t s);
void launch_average(const DevMesh& m, const double* esize, double* size, cudaStream_t s);
// isotropic lengths of given sizes, bitwise the reference's
void launch_measure_iso_f64(const DevMesh& m, const double* size, double* L, cudaStream_t s);
// per mesh, half the Euclidean edge lengths (E doubles); the pass's lengths (not
// the sequence's bits but near 0.5 and 1.5) with the predicate bitmaps, len null:
// in place
void launch_edge_records(const DevMesh& m, double* len, cudaStream_t s);
void launch_measure_mark_f64(const DevMesh& m, const double* len, const double* size, double* L, uint32_t* split,
                             uint32_t* collapse, cudaStream_t s);

// ---- kernel launchers (sprg_kernels_f64.cu) ---------------------------
// Triangles (tets recover through launch_qr_weights / launch_recover_w64):
// xl: patches that need growth; big: patches above the thread-per-vertex
// size (fitted by the warp path inside launch_recover_f64, which may add to
// xl).  The factors of the thread path's patches are per mesh: qc
// tri_factor_planes() and rr tri_r_planes() planes of V doubles, code V
// bytes; launch_tri_factor fills them and both lists (counters zero on
// entry).  qc null: launch_recover_f64 factors in place and fills the lists
// itself.  any_big: the big list may hold vertices.
struct TriFactor {
  double* qc;
  double* rr;
  unsigned char* code;
};
int tri_factor_planes();
int tri_r_planes();
void launch_tri_factor(const DevMesh& m, TriFactor tf, ExpandList xl, ExpandList big, cudaStream_t s);
// pw: the listed patches (n = 0: left to the caller)
void launch_recover_f64(const DevMesh& m, const double* ip, int nc, double* rec, TriFactor tf, ExpandList xl,
                        ExpandList big, bool any_big, const PatchWeights& pw, cudaStream_t s);
// Patches on the expansion list: grow as the reference does, then fit.
// The list length is read on the device (no host round trip).
// slab: expand_grid() * expand_max_elems() * (4 + nc + 1) doubles.
// nc 0: growth and rank tests alone (ip and rec unused).
// cache_* (optional): record each listed vertex's final element set
// (expand_max_elems() ints per list slot).
void launch_expand_f64(const DevMesh& m, const double* ip, int nc, double* rec, ExpandList xl, double* slab,
                       DevStatus* st, cudaStream_t s, int* cache_v = nullptr, int* cache_n = nullptr,
                       int* cache_el = nullptr);
// Triangles with patches on the warp path: one QR fit per cached listed vertex
// (patch growth depends on geometry only).
void launch_cached_fit_f64(const DevMesh& m, const double* ip, int nc, double* rec, int n_cached, const int* cache_v,
                           const int* cache_n, const int* cache_el, double* slab, DevStatus* st, cudaStream_t s);
// Per-mesh weights of the cached patches (w = Q1 R^-T t from the fit's
// QR; woff: each patch's offset into w, wn: its size or -1 where the rank
// test fails)
void launch_cached_weights_f64(const DevMesh& m, int n_cached, const int* cache_v, const int* cache_n,
                               const int* cache_el, const long long* woff, double* w, int* wn, double* slab,
                               cudaStream_t s);
int expand_max_elems();
int expand_grid();
// Sum partials in fixed order, compute size factor.  mode 0: SPR; 1: target.
void launch_size_factor(const double* partials, int n_blocks, int mode, double adapt_ratio, double target,
                        int dim, double* out3, cudaStream_t s);
// split / collapse (optional): the predicate bitmaps of the lengths, bit e of
// split = L[e] > 1.5, of collapse = L[e] < 0.5
void launch_measure_aniso_f64(const DevMesh& m, const double* sizes, const double* frames, double* L, uint32_t* split,
                              uint32_t* collapse, cudaStream_t s);
void launch_mark(int E, const double* L, int which, int* flags, unsigned long long* count, DevStatus* st,
                 cudaStream_t s);
// markEntities semantics from a predicate bitmap
void launch_apply_bits(int E, const uint32_t* bits, int which, int* flags, unsigned long long* count,
                       DevStatus* st, cudaStream_t s);
// the collapse and split passes in one sweep (counts[0] split, counts[1] collapse)
// skip (device int, or null): when nonzero the flags stay unchanged
void launch_apply_marks(int E, const uint32_t* split_bits, const uint32_t* collapse_bits, int* flags,
                        unsigned long long* counts, DevStatus* st, const int* skip, cudaStream_t s);
// MA sweeps around the marks.  kind: 0 identity size field, 1 isotropic
// (size), 2 anisotropic (sizes, frames), 3 log-interpolated anisotropic
// (logm); pairs: n x 2 vertex ids, or NULL for the mesh's edges (n = E);
// st records SPRG_EEIGEN when an eigen iteration fails
void launch_measure_pairs(const DevMesh& m, int kind, long long n, const int* pairs, const double* size,
                          const double* sizes, const double* frames, const double* logm, double* L, DevStatus* st,
                          cudaStream_t s);
// LogAnisoSizeField: per-vertex log-metric (V x 9) of sizes and frames; kind
// 3 of launch_measure_pairs and the logm argument of launch_quality_f64 read it
void launch_log_metric(int V, const double* sizes, const double* frames, double* logm, cudaStream_t s);
// *out = bits of max(0, the positive values of x) (NaN ignored)
void launch_max_positive(long long n, const double* x, unsigned long long* out, cudaStream_t s);
// deterministic sum: partials holds sum_partials_count() doubles
int sum_partials_count();
void launch_sum(long long n, const double* x, double* partials, double* out, cudaStream_t s);
// first index (in *first, all ones if none) holding the minimum of the
// values below `start`; *key is scratch
void launch_first_min_below(long long n, const double* x, double start, unsigned long long* key,
                            unsigned long long* first, cudaStream_t s);
void launch_mark_quality(int T, const double* q, double good, int* flags, unsigned long long* count, DevStatus* st,
                         cudaStream_t s);
// Mixed-precision anisotropic pass.  Triangle patch weights (FP64, patch
// CSR layout) with the listed vertices (weights not covering them) in lst;
// FP32 metric records (12 floats per
// vertex: h, frame) and quality records (FP32 vertex transforms and
// determinants; ambiguous choices that matter are decided in FP64);
// FP32 edge measure writing the mark bitmaps and the
// edges within their error bound of 0.5 / 1.5 (guard); the guard's FP64
// re-measure fixing those bits; FP32 qualities.
// n_big (zero before): the refined weights of the FP64 anisotropic pass, with the count of
// the patches of more elements than the weights take; null: the mixed pass's
void launch_tri_weights(const DevMesh& m, double* w, unsigned char* listed, ExpandList lst, int* n_big, cudaStream_t s);
// qrec: quality_rec_bytes() per vertex
void launch_metric_f32(int V, int dim, const double* sizes, const double* frames, float* out, void* qrec,
                       cudaStream_t s);
int quality_rec_bytes();
// crec: the FP32 path's coordinate records in the frame x' = (x - c) s + 1
// (frame_scale = s); flat (a mesh in the z = 0 plane, the operator's two-row
// form): met and crec are that form's flat_met and flat_rec
void launch_measure_aniso_f32(const DevMesh& m, bool flat, const float* met, const float4* crec, double frame_scale,
                              uint32_t* split, uint32_t* collapse, int* guard, int* gcount, int gcap, cudaStream_t s);
// sizes / frames: the FP64 metric, or null to rebuild the guarded edges'
// ends from the Hessian H (hessian_metric_vertex, the FP64 pass's bits)
void launch_measure_guard_f64(const DevMesh& m, const double* sizes, const double* frames, const double* H,
                              double eps, double hmin, double hmax, const int* guard, const int* gcount, int gcap,
                              uint32_t* split, uint32_t* collapse, cudaStream_t s);
// sizes / frames as for the guard (the FP64 determinants of tie-breaks)
// two launches: FP32 qualities (listing the elements whose vertex pick the
// FP32 determinants leave open), then the FP64 tie-breaks; cj64: V doubles,
// tie_items: T ints, tie_count: one int (scratch, cleared here)
void launch_quality_aniso_f32(const DevMesh& m, bool flat, const void* qrec, const float4* crec, double frame_scale,
                              const double* sizes, const double* frames, const double* H, double eps, double hmin,
                              double hmax, double* cj64, int* tie_items, int* tie_count, double* q, cudaStream_t s);
// Triangle recovery-of-gradient operator (per mesh, FP64): K_va over the
// patch vertices, tri_operator_slots() slots per vertex (kidx ints, kval 3
// doubles each, a plane of V per slot; klen counts; patches that are not fans
// are added to the listed set)
int tri_operator_slots();
// kc: components per operator slot, 3, or 2 for a mesh in the z = 0 plane
void launch_tri_operator(const DevMesh& m, int kc, const double* w, unsigned char* listed, ExpandList lst, int* kidx,
                         double* kval, int* klen, cudaStream_t s);
// applied to a scalar (ncin 1 -> V x 3) or a VECTOR field (ncin 3 -> V x 9, and
// from that Hessian the FP32 metric records, 12 floats in met, and quality
// records: FP64 decisions, FP32 magnitudes) at every vertex, the listed ones
// through their patches' weights
void launch_apply_operator(const DevMesh& m, int ncin, int kc, const unsigned char* listed, const int* kidx,
                           const double* kval, const int* klen, const double* f, double* out, const PatchWeights& ls,
                           double eps, double hmin, double hmax, float* met, void* qrec, float4* flat_rec, cudaStream_t s);
// incremental mesh update: dst[ids[r] * width + j] = vals[r * width + j];
// the coordinates' bounding box as order keys (3 minima, 3 maxima)
void launch_scatter_rows_f64(long long n, int width, const int* ids, const double* vals, double* dst, cudaStream_t s);
void launch_scatter_rows_i32(long long n, int width, const int* ids, const int* vals, int* dst, cudaStream_t s);
void launch_bbox(int V, const double* xyz, unsigned long long* keys, cudaStream_t s);
// *bad += the number of entries of a outside [0, limit)
void launch_count_out_of_range(long long n, const int* a, int limit, unsigned long long* bad, cudaStream_t s);
double key_to_double(unsigned long long k);
// FP64 SPR weights of tet patches (per mesh, the reference's QR; listed
// patches in lst) and the FP64 recovery from them
void launch_qr_weights(const DevMesh& m, double* w, unsigned char* listed, ExpandList lst, cudaStream_t s);
// (the listed ones through pw; redo, triangles: scratch for V items a recovery and a
// count that is zero before a pass's first); returns the number of launches
int launch_recover_w64(const DevMesh& m, const double* ip, int nc, const double* w, const unsigned char* listed,
                        const PatchWeights& pw, double* rec, ExpandList redo, cudaStream_t s);
// FP64 guard band of the FP32 path: re-decide the listed edges' bits.
struct GuardScratch {
  int* stamp;      // V ints, persistent (de-duplication stamps)
  int* stamp_id;   // device counter: this pass's stamp id (starts at 1; the decide stage bumps it)
  int* fit_items;  // fit_cap ints
  int* fit_count;  // zero before the measure kernel
  int fit_cap;
  double* rec64;   // V x 3 doubles (FP64 recovered values of collected vertices)
  const double* w64;            // FP64 SPR weights in patch-CSR order
  const unsigned char* listed;  // patches on the FP64 reference path
  const double* rec_ref;        // their FP64 reference results (V x 3)
  const double2* geo64;         // per element {det J, h_max} in FP64
};
// unresolved[0]: edges left to the FP32 decision.  After the measure kernel,
// which collects the vertices, two stages in order: 0 fits, 1 decide.
constexpr int kGuardMaxTets = 96;  // elements around one end vertex
constexpr int kGuardStages = 2;
void launch_guard_stage(int stage, const DevMesh& m, const double* u, const double* out3, const int* items,
                        const int* count, int cap, uint32_t* split, uint32_t* collapse, int* unresolved,
                        GuardScratch g, BatchView bv, cudaStream_t s);
// per-mesh size factors of a batch (SPR mode) from segment partials
void launch_size_factor_batch(const double* partials, BatchView bv, int dim, double* out4, cudaStream_t s);
// FP64 qualities (sprg_quality_f64.cu) under the field `size` (isotropic),
// `sizes` and `frames`, or the log-metrics `logm`; xf / bad:
// vertex_transform_bytes(V) and V bytes of scratch for the vertices'
// transforms (null: computed per element), not used for the isotropic field
size_t vertex_transform_bytes(int V);
void launch_quality_f64(const DevMesh& m, const double* size, const double* sizes, const double* frames,
                        const double* logm, double* xf, unsigned char* bad, bool pass, double* q, DevStatus* st, cudaStream_t s);
// anisotropic metric (sizes V x 3, frames V x 9) from a nodal Hessian (V x 9)
void launch_hessian_metric(const DevMesh& m, const double* H, double eps, double hmin, double hmax, double* sizes,
                           double* frames, cudaStream_t s);

// ---- adjacency builders (sprg_kernels_f64.cu) ---------------------------
// Ascending vertex->element CSR via counting sort on the device.
// off must hold V + 1 ints, el T * nn ints, tmp V ints, scan
// offset_scan_bytes(V) (taken before a mesh is given up: the offsets are
// built by the scan, and counts left in their place would be read as offsets).
cudaError_t launch_build_v2e(const DevMesh& m, int* off, int* el, int* tmp, void* scan, size_t scan_bytes,
                             cudaStream_t s);
// V counts and a zero -> V + 1 offsets, in place
size_t offset_scan_bytes(int V);
cudaError_t launch_offset_scan(int V, int* off, void* scan, size_t scan_bytes, cudaStream_t s);
// Sort each CSR segment ascending (segments are short).
void launch_sort_segments(int V, const int* off, int* el, cudaStream_t s);
// X = rint((x - c) s 2^30) per coordinate (c the frame's corner, s its scale)
void launch_xyz_to_fixed(const DevMesh& m, const double* frame, int* xyzq, cudaStream_t s);

}  // namespace sprg
