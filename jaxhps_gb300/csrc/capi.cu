// C ABI of the native HPS library (declarations: include/jaxhps_gb300.h).
//
// Each stage entry point validates its arguments, carves the caller's
// workspace, and enqueues the kernel sequence of that stage on the given
// stream.  No device memory is allocated here.
#include <stdarg.h>
#include <stdio.h>
#include <string.h>

#include <atomic>
#include <vector>
#include <string>

#include "../../include/jaxhps_gb300.h"
#include "hps_common.cuh"
#include "hps_internal.h"

namespace hps {

template <class T, class CT>
cudaError_t leaf_assemble(int n_leaves, int n_pts, int row0, int n_rows, int col_split, int n_ops,
                          const double* ops, const CT* coeffs, T* out_lo, long long ld_lo, long long s_lo,
                          T* out_hi, long long ld_hi, long long s_hi, cudaStream_t st);
template <class T>
cudaError_t set_rows(int batch, int rows, int cols, const T* src, long long lds, T* dst, long long ldd,
                     long long sd, cudaStream_t st);
template <class T>
cudaError_t row_equilibrate(int batch, int n, T* A, long long lda, long long sA, double* s, cudaStream_t st);
template <class T>
cudaError_t col_scale(int batch, int n, T* X, long long ldx, long long sX, const double* s, cudaStream_t st);
template <class T>
cudaError_t row_scale(int batch, int rows, int cols, T* X, const double* s, cudaStream_t st);
template <class T>
cudaError_t balance_rows(int nm, int n, int ne, int ns, T* D, T* C, T* dh, double* s, cudaStream_t st);
template <class T>
cudaError_t perm_gather(int batch, int n, int nr, int nc, const T* M, long long sM, const int* perm, int r0, int c0,
                        T* out, long long sO, cudaStream_t st);
template <class T>
cudaError_t perm_scatter(int batch, int n, int nr, int nc, T* M, long long sM, const int* perm, int r0, int c0,
                         const T* in, long long sI, int add_identity, cudaStream_t st);
template <class T>
cudaError_t add_identity(int batch, int n, T* X, long long sX, cudaStream_t st);
cudaError_t refine_points_3d(int n_nodes, int p, const double* bounds, const double* cheb, const int* perm,
                             double* pts, cudaStream_t st);
cudaError_t refine_points_2d(int n_nodes, int p, const double* bounds, const double* cheb, const int* perm,
                             double* pts, cudaStream_t st);
cudaError_t refine_check_2d(int n_nodes, int p, const double* fv, const int* perm, const int* iperm,
                            const double* Ilo, const double* Ihi, const double* wref, const double* bounds,
                            double* diff, double* ref, double* l2, cudaStream_t st);
template <class T>
cudaError_t panel_map(int mode, int batch, int n_out, int n_other, int m_len, const int* tab, const T* M, const T* in,
                      long long ld_in, long long s_in, T* out, long long ld_out, long long s_out, cudaStream_t st);
template <class T>
cudaError_t scale_batched(int batch, long long n_per, const double* scale, T* x, cudaStream_t st);
int mlp_param_count();
cudaError_t mlp_sample_points(int n, const double* bounds, double* pts, cudaStream_t st);
cudaError_t mlp_features(int n, const double* fvals, const int* depth, double inv_scale, float* X, cudaStream_t st);
cudaError_t mlp_forward(int n, const float* X, const float* P, float* H1, float* H2, float* logit, cudaStream_t st);
cudaError_t mlp_bce(int n, const float* logit, const float* y, float wpos, float* dlogit, float* loss,
                    cudaStream_t st);
cudaError_t mlp_backward(int n, const float* X, const float* P, const float* H1, const float* H2,
                         const float* dlogit, float* G, cudaStream_t st);
cudaError_t mlp_adam(float* P, const float* G, float* M, float* V, float lr, float b1, float b2, float eps, int step,
                     cudaStream_t st);
cudaError_t refine_check_3d(int n_nodes, int p, const double* fv, const int* perm, const int* iperm,
                            const double* Ilo, const double* Ihi, const double* wref, const double* bounds,
                            double* diff, double* ref, double* l2, cudaStream_t st);
template <class T>
cudaError_t merge_gather(int n_merges, int nch, int nb, int n_int, int n_ext, int ns, const T* Tc, const T* hc,
                         const int* int_c, const int* int_l, const int* ext_c, const int* ext_l,
                         const int* loc, T* D, T* C, T* B, T* Tout, T* dh, T* hext, int skip_zero,
                         cudaStream_t st);
template <class T>
cudaError_t merge_gather_iti(int n_merges, int nch, int nb, int n_int, int n_ext, int ns, const T* Rc, const T* hc,
                             const int* int_c, const int* int_l, const int* ext_c, const int* ext_l, T* D, T* C, T* B,
                             T* Tout, T* dh, T* hext, int skip_zero, cudaStream_t st);
template <class T>
cudaError_t down_scatter(int n_merges, int nch, int nb, int n_ext, int n_int, int ns, const int* code,
                         const T* gpar, const T* gint, T* gch, cudaStream_t st);
template <class S, class D>
cudaError_t convert(long long n, const S* src, D* dst, cudaStream_t st);
cudaError_t residual_2d(int n_leaves, int p, int q, int nsrc, int n_ops, unsigned long long kinds, const double* coeffs,
                        const double* inv_half, const double* D1, const double* D2, const double* Pside,
                        const double* Qside, const int* perm, const double* u_int, const double* g,
                        const double* f, float* r_int, double* r_int64, float* r_lo, double* flux, double* u_full,
                        int need_uy, cudaStream_t st, const float* u_int32 = nullptr);
cudaError_t accumulate_pair_max(long long n, const float* x, float* hi, float* lo, double* out, cudaStream_t st);
cudaError_t assemble_u_pair_2d(int n_leaves, int p, int q, int nsrc, const double* Pside, const float* u_hi,
                               const float* u_lo, const double* g, double* u_full, cudaStream_t st);
cudaError_t flux_combine(long long n_nodes, int nsrc, const int* nbr, const double* flux, float* hcorr, int n_bdry,
                         const int* bdry_node, const double* g_given, const double* g_state, float* r_bdry,
                         cudaStream_t st);
cudaError_t accumulate(long long n, const float* x, double* y, cudaStream_t st);
cudaError_t accumulate_max(long long n, int pairs, const float* x, double* y, double* out, cudaStream_t st);
cudaError_t interp_rows(long long n_rows, int n_src, const double* to, const double* src, const double* w,
                        double* out, int rpg, int transposed, cudaStream_t st);
cudaError_t gather_cols(long long n_groups, int n_in, int n_out, const int* idx, const double* in, double* out,
                        cudaStream_t st);
cudaError_t interp_leaf_nodes(int dim, long long n_leaves, int p, const double* bounds, const double* ref, double* nodes,
                              double* wts, cudaStream_t st);
cudaError_t interp_from_leaves(int dim, long long n_t, int nsrc, const double* tpts, int p, const double* bounds,
                               const double* nodes, const double* wts, const int* rearr, const int* cells,
                               const int* nc, const double* lo, const double* h, const double* f, double* out,
                               cudaStream_t st);
cudaError_t residual_iti_2d(int n_leaves, int p, int q, int nsrc, int n_ops, unsigned long long kinds, int cplx,
                            double eta, const void* coeffs, const double* inv_half, const double* D1,
                            const double* D2, const double* Pside, const double* Qside, const int* perm,
                            const void* u, const void* t_in, const void* f, void* r, void* t_out, int need_uy,
                            cudaStream_t st);
cudaError_t iti_combine(long long n_nodes, int nsrc, const int* nbr, const void* t_out, const void* t_in, void* hcorr,
                        int n_bdry, const int* bdry_node, const void* t_given, void* r_bdry, cudaStream_t st);
cudaError_t jx_update_2d(int n_leaves, int p, int q, int nsrc, int n_ops, unsigned long long kinds,
                         const double* coeffs, const double* inv_half, const double* D1, const double* D2,
                         const double* Pside, const double* Qside, const int* perm, const float* du, const float* dg,
                         double* r_int, float* r32, double* flux, int need_uy, cudaStream_t st);
bool jx_df_supported(int p, int q);
size_t jx_df_prep_floats(int n_leaves, int p, int q, int n_ops);
cudaError_t jx_df_prepare(int n_leaves, int p, int q, int n_ops, unsigned long long kinds, const double* coeffs,
                          const double* inv_half, const double* D1, const double* D2, const double* Pside,
                          const double* Qside, const int* perm, float* prep, cudaStream_t st);
cudaError_t jx_df_update_2d(int n_leaves, int p, int q, int nsrc, int n_ops, unsigned long long kinds,
                            const float* prep, const double* inv_half, const int* perm, const float* du,
                            const float* dg, float* r_hi, float* r_lo, double* flux, int need_uy, cudaStream_t st);
cudaError_t assemble_u_2d(int n_leaves, int p, int q, int nsrc, const double* Pside, const double* u_int,
                          const double* g, double* u_full, cudaStream_t st);
cudaError_t interior_f32(long long n_leaves, int pp, int ncb, int nsrc, const double* f, float* r32, cudaStream_t st);

static thread_local std::string g_last_error;
static std::atomic<long long> g_launches{0};

void note_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

// ---- live profiler: event pairs around the launches of the armed classes ----
constexpr int N_KC = 8;
struct Profiler {
  unsigned mask = 0;
  std::vector<cudaEvent_t> ev;  // 2 per slot
  std::vector<int> slot_cls;
  int used = 0;
  double work[N_KC] = {0};
  long long launches[N_KC] = {0};
};
static Profiler g_prof;

// Scopes nest (an inversion's panel kernels and GEMM updates): only the
// outermost records, so no launch is counted twice.
static thread_local int g_prof_depth = 0;

ProfScope::ProfScope(int cls, cudaStream_t s, double w) : on(false), st(s), slot(-1) {
  if (++g_prof_depth > 1) return;
  if (cls <= 0 || cls >= N_KC || !(g_prof.mask & (1u << cls))) return;
  if (g_prof.used * 2 + 2 > (int)g_prof.ev.size()) {
    for (int i = 0; i < 256; ++i) {
      cudaEvent_t e;
      if (cudaEventCreate(&e) != cudaSuccess) return;
      g_prof.ev.push_back(e);
    }
  }
  slot = g_prof.used++;
  if ((int)g_prof.slot_cls.size() < g_prof.used) g_prof.slot_cls.resize(g_prof.used);
  g_prof.slot_cls[slot] = cls;
  on = true;
  g_prof.work[cls] += w;
  g_prof.launches[cls] += 1;
  cudaEventRecord(g_prof.ev[2 * slot], st);
}

ProfScope::~ProfScope() {
  if (on) cudaEventRecord(g_prof.ev[2 * slot + 1], st);
  --g_prof_depth;
}

void set_error(const char* fmt, ...) {
  char buf[1024];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  g_last_error = buf;
}

static size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

// Carves consecutive 256-byte aligned regions out of a workspace.
struct Carver {
  unsigned char* p;
  size_t used = 0;
  explicit Carver(void* base) : p(reinterpret_cast<unsigned char*>(base)) {}
  void* take(size_t bytes) {
    void* r = p ? p + used : nullptr;
    used += al256(bytes);
    return r;
  }
};

#define HPS_CHECK(...)                                                             \
  do {                                                                             \
    cudaError_t _e = (__VA_ARGS__);                                                    \
    if (_e != cudaSuccess) {                                                       \
      set_error("%s failed: %s (%s:%d)", #__VA_ARGS__, cudaGetErrorString(_e), __FILE__, \
                __LINE__);                                                         \
      return HPS_ERR_CUDA;                                                         \
    }                                                                              \
  } while (0)

// ---------------------------------------------------------------------------
// Leaf DtN
// ---------------------------------------------------------------------------
// FP64 and complex128 leaves: the rows of A_ii and of W = -A_ie P are brought
// to one scale before the elimination (powers of two: exact), the inverse's
// columns back afterwards.  Collocation rows near the leaf's boundary are
// about p^2 / 2 times those at its centre, so the inverse's columns and W's
// rows are graded the opposite way, and the digit products (gemm_f64_tc.cu),
// which keep a row's or column's entries relative to its largest, would drop
// what the small ones carry: against long double Y is off by 5.8e-16 with the
// scaling, 8.3e-16 without, and was by 7.8e-16 from FP64 chains (T: 0.96e-15,
// 1.02e-15, 1.81e-15; 42 leaves of seven problems, p = 9 to 16).
static bool leaf_rows_scaled(int dtype) { return dtype == F64 || dtype == C128; }

// The dtype field of the stage arguments: element type and HPS_INVERSE_REFINED.
static int base_dtype(int dtype) { return dtype & ~HPS_INVERSE_REFINED; }
static bool wants_refined(int dtype, int n, const int* info) {
  return (dtype & HPS_INVERSE_REFINED) && info && inverse_refined_takes(base_dtype(dtype), n);
}
static size_t stage_inverse_bytes(int dtype, int n, int batch, const int* info) {
  return wants_refined(dtype, n, info) ? inverse_refined_workspace_bytes(base_dtype(dtype), n, batch)
                                       : inverse_workspace_bytes(base_dtype(dtype), n, batch);
}
template <class T>
static cudaError_t stage_inverse(int dtype, int n, T* X, int batch, int* info, void* ws, size_t bytes, cudaStream_t st,
                                 int flags) {
  const long long nn = (long long)n * n;
  if constexpr (DTypeOf<T>::value == F64 || DTypeOf<T>::value == C128) {
    if (wants_refined(dtype, n, info))
      return inverse_refined<T>(n, X, n, nn, X, n, nn, batch, info, ws, bytes, st);
  }
  return inverse_batched<T>(n, X, n, nn, X, n, nn, batch, info, ws, bytes, st, flags);
}

static size_t leaf_dtn_ws(const hps_leaf_dtn_args* a, Carver* cv) {
  const size_t es = dtype_size(base_dtype(a->dtype));
  const int n_i = a->n_pts - a->n_cb;
  cv->take(es * (size_t)a->n_leaves * n_i * a->n_cb);      // A_ie
  cv->take(es * (size_t)a->n_leaves * n_i * a->n_gauss);   // W = -A_ie P
  cv->take(stage_inverse_bytes(a->dtype, n_i, a->n_leaves, a->info));
  if (leaf_rows_scaled(base_dtype(a->dtype))) cv->take(sizeof(double) * (size_t)a->n_leaves * n_i);
  return cv->used + 256;
}

template <class T>
static int leaf_dtn_impl(const hps_leaf_dtn_args* a, cudaStream_t st) {
  const int nl = a->n_leaves, np = a->n_pts, ncb = a->n_cb, ng = a->n_gauss, ns = a->nsrc;
  const int ni = np - ncb;
  unsigned char* wsb = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(a->workspace) + 255) & ~uintptr_t(255));
  Carver cv(wsb);
  T* Aie = (T*)cv.take(sizeof(T) * (size_t)nl * ni * ncb);
  T* W = (T*)cv.take(sizeof(T) * (size_t)nl * ni * ng);
  const size_t invb = stage_inverse_bytes(a->dtype, ni, nl, a->info);
  void* invws = cv.take(invb);
  constexpr int dt = DTypeOf<T>::value;
  double* rscale = leaf_rows_scaled(dt) ? (double*)cv.take(sizeof(double) * (size_t)nl * ni) : nullptr;
  T* Aii = (T*)a->Aii_inv;
  cudaError_t e;
  if (a->coef_complex)
    e = leaf_assemble<T, c128>(nl, np, ncb, ni, ncb, a->n_ops, a->ops, (const c128*)a->coeffs, Aie, ncb,
                               (long long)ni * ncb, Aii, ni, (long long)ni * ni, st);
  else
    e = leaf_assemble<T, double>(nl, np, ncb, ni, ncb, a->n_ops, a->ops, (const double*)a->coeffs, Aie, ncb,
                                 (long long)ni * ncb, Aii, ni, (long long)ni * ni, st);
  HPS_CHECK(e);
  const T one_ = one<T>(), zero_ = zero<T>(), mone = make_scalar<T>(-1.0, 0.0);
  const T* P = (const T*)a->P;
  const T* Q = (const T*)a->Q;
  T* Y = (T*)a->Y;
  // W = -A_ie P
  HPS_CHECK(gemm_batched<T>(ni, ng, ncb, mone, Aie, ncb, (long long)ni * ncb, P, ng, 0, zero_, nullptr, 0, 0, W,
                            ng, (long long)ni * ng, nl, st));
  if (rscale) {
    HPS_CHECK(row_equilibrate<T>(nl, ni, Aii, ni, (long long)ni * ni, rscale, st));
    HPS_CHECK(row_scale<T>(nl, ni, ng, W, rscale, st));
  }
  // the leaf blocks may use the tensor-memory kernel (FP32, 64 < n <= 224)
  HPS_CHECK(stage_inverse<T>(a->dtype, ni, Aii, nl, a->info, invws, invb, st, INV_TENSOR_MEMORY));
  // Y[n_cb:] = A_ii^-1 W ;  Y[:n_cb] = P
  HPS_CHECK(gemm_batched<T>(ni, ng, ni, one_, Aii, ni, (long long)ni * ni, W, ng, (long long)ni * ng, zero_,
                            nullptr, 0, 0, Y + (size_t)ncb * ng, ng, (long long)np * ng, nl, st));
  HPS_CHECK(set_rows<T>(nl, ncb, ng, P, ng, Y, ng, (long long)np * ng, st));
  if (rscale) HPS_CHECK(col_scale<T>(nl, ni, Aii, ni, (long long)ni * ni, rscale, st));
  // T = Q Y
  HPS_CHECK(gemm_batched<T>(ng, ng, np, one_, Q, np, 0, Y, ng, (long long)np * ng, zero_, nullptr, 0, 0,
                            (T*)a->T, ng, (long long)ng * ng, nl, st));
  if (ns > 0 && a->source && a->v) {
    T* v = (T*)a->v;
    const T* f = (const T*)a->source;
    HPS_CHECK(gemm_batched<T>(ni, ns, ni, one_, Aii, ni, (long long)ni * ni, f + (size_t)ncb * ns, ns,
                              (long long)np * ns, zero_, nullptr, 0, 0, v + (size_t)ncb * ns, ns,
                              (long long)np * ns, nl, st));
    HPS_CHECK(set_rows<T>(nl, ncb, ns, nullptr, 0, v, ns, (long long)np * ns, st));
    if (a->h)
      HPS_CHECK(gemm_batched<T>(ng, ns, np, one_, Q, np, 0, v, ns, (long long)np * ns, zero_, nullptr, 0, 0,
                                (T*)a->h, ns, (long long)ng * ns, nl, st));
  }
  return HPS_OK;
}

// ---------------------------------------------------------------------------
// Leaf ItI
// ---------------------------------------------------------------------------
static size_t leaf_iti_ws(const hps_leaf_iti_args* a, Carver* cv) {
  cv->take(stage_inverse_bytes(a->dtype, a->n_pts, a->n_leaves, a->info));
  cv->take(sizeof(double) * (size_t)a->n_leaves * a->n_pts);
  return cv->used + 256;
}

template <class T>
static int leaf_iti_impl(const hps_leaf_iti_args* a, cudaStream_t st) {
  const int nl = a->n_leaves, np = a->n_pts, ncb = a->n_cb, ng = a->n_gauss, ns = a->nsrc;
  const int ni = np - ncb;
  unsigned char* wsb = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(a->workspace) + 255) & ~uintptr_t(255));
  Carver cv(wsb);
  const size_t invb = stage_inverse_bytes(a->dtype, np, nl, a->info);
  void* invws = cv.take(invb);
  double* rscale = (double*)cv.take(sizeof(double) * (size_t)nl * np);
  T* Bm = (T*)a->B_inv;
  const long long sB = (long long)np * np;
  HPS_CHECK(set_rows<T>(nl, ncb, np, (const T*)a->G, np, Bm, np, sB, st));
  cudaError_t e;
  if (a->coef_complex)
    e = leaf_assemble<T, c128>(nl, np, ncb, ni, 0, a->n_ops, a->ops, (const c128*)a->coeffs, nullptr, 0, 0,
                               Bm + (size_t)ncb * np, np, sB, st);
  else
    e = leaf_assemble<T, double>(nl, np, ncb, ni, 0, a->n_ops, a->ops, (const double*)a->coeffs, nullptr, 0, 0,
                                 Bm + (size_t)ncb * np, np, sB, st);
  HPS_CHECK(e);
  // inv(B) = inv(diag(s) B) diag(s): the impedance rows (~p^2/h) and the PDE
  // rows (~p^4/h^2) are brought to one scale before elimination
  HPS_CHECK(row_equilibrate<T>(nl, np, Bm, np, sB, rscale, st));
  HPS_CHECK(stage_inverse<T>(a->dtype, np, Bm, nl, a->info, invws, invb, st, 0));
  HPS_CHECK(col_scale<T>(nl, np, Bm, np, sB, rscale, st));
  const T one_ = one<T>(), zero_ = zero<T>();
  HPS_CHECK(gemm_batched<T>(np, ng, ncb, one_, Bm, np, sB, (const T*)a->P, ng, 0, zero_, nullptr, 0, 0,
                            (T*)a->Y, ng, (long long)np * ng, nl, st));
  HPS_CHECK(gemm_batched<T>(ng, ng, np, one_, (const T*)a->QH, np, 0, (const T*)a->Y, ng, (long long)np * ng,
                            zero_, nullptr, 0, 0, (T*)a->T, ng, (long long)ng * ng, nl, st));
  if (ns > 0 && a->source && a->v) {
    HPS_CHECK(gemm_batched<T>(np, ns, ni, one_, Bm + ncb, np, sB, (const T*)a->source + (size_t)ncb * ns, ns,
                              (long long)np * ns, zero_, nullptr, 0, 0, (T*)a->v, ns, (long long)np * ns, nl,
                              st));
    if (a->h)
      HPS_CHECK(gemm_batched<T>(ng, ns, np, one_, (const T*)a->QH, np, 0, (const T*)a->v, ns,
                                (long long)np * ns, zero_, nullptr, 0, 0, (T*)a->h, ns, (long long)ng * ns, nl,
                                st));
  }
  return HPS_OK;
}

// ---------------------------------------------------------------------------
// Merge level (DtN)
// ---------------------------------------------------------------------------
static size_t merge_ws(const hps_merge_args* a, Carver* cv) {
  const size_t es = dtype_size(base_dtype(a->dtype));
  const size_t nm = (size_t)a->n_merges;
  if (!a->D_inv) cv->take(es * nm * a->n_int * a->n_int);
  cv->take(es * nm * a->n_int * a->n_ext);                       // C
  cv->take(es * nm * a->n_ext * a->n_int);                       // B
  cv->take(es * nm * a->n_int * (a->nsrc > 0 ? a->nsrc : 1));    // dh
  if (a->n_x > 0) {
    // two-colour inverse: D12, D21, W, P (n_x^2 each) and W's inverse scratch
    for (int k = 0; k < 4; ++k) cv->take(es * nm * a->n_x * a->n_x);
    cv->take(stage_inverse_bytes(a->dtype, a->n_x, a->n_merges, a->info));
  } else {
    cv->take(stage_inverse_bytes(a->dtype, a->n_int, a->n_merges, a->info));
  }
  if (leaf_rows_scaled(base_dtype(a->dtype))) cv->take(sizeof(double) * nm * a->n_int);   // balance_rows
  return cv->used + 256;
}

// The rectangles of C (c_form) or B as groups, one per exterior range with the
// interface ranges as its segments: the products of a whole merge are then one
// launch, each with its full K (3D: 72 products of one face each took 20 to 36
// us apiece, bound by a single tile's latency, and read and wrote S and T_out
// three times).  64 leaves of 8^2, whole build and solve: 3.2 -> 1.8 ms, 8 x 8
// leaves of 10^3 27.8 -> 22.1 ms, no size found where the single products are
// faster.  0 where the ranges are not the same or disjoint, or too many.
static int rect_groups(const hps_merge_args* a, bool c_form, int other, GemmGroup* g) {
  const int n = c_form ? a->n_c_rects : a->n_b_rects;
  const int* r = c_form ? a->c_rects : a->b_rects;
  int ng = 0;
  for (int k = 0; k < n; ++k) {
    const int* q = r + 5 * k;
    const int i0 = c_form ? q[0] : q[2], li = c_form ? q[1] : q[3], e0 = c_form ? q[2] : q[0], le = c_form ? q[3] : q[1];
    int j = 0;
    for (; j < ng; ++j) {
      const int f0 = c_form ? g[j].n0 : g[j].m0, lf = c_form ? g[j].n : g[j].m;
      if (f0 == e0 && lf == le) break;
      if (e0 < f0 + lf && f0 < e0 + le) return 0;
    }
    if (j == ng) {
      if (ng == GEMM_GROUPS) return 0;
      GemmGroup& x = g[ng++];
      x.segs = 0;
      (c_form ? x.n0 : x.m0) = e0;
      (c_form ? x.n : x.m) = le;
      (c_form ? x.m0 : x.n0) = 0;
      (c_form ? x.m : x.n) = other;
    }
    GemmGroup& x = g[j];
    // ranges side by side are one segment
    if (x.segs > 0 && x.k0[x.segs - 1] + x.len[x.segs - 1] == i0) {
      x.len[x.segs - 1] += li;
      continue;
    }
    if (x.segs == GEMM_SEGS) return 0;
    x.k0[x.segs] = i0;
    x.len[x.segs++] = li;
  }
  return ng;
}

template <class T>
static cudaError_t run_groups(const GemmGroup* g, int ng, double alpha, const T* A, long long lda, long long sA, const T* B,
                              long long ldb, long long sB, bool add, T* D, long long ldd, long long sD, int batch,
                              cudaStream_t st) {
  if constexpr (DTypeOf<T>::value == F64 || DTypeOf<T>::value == C128)
    return gemm_groups<T>(g, ng, alpha, A, lda, sA, B, ldb, sB, 1.0, add ? D : nullptr, ldd, sD, D, ldd, sD, batch, st);
  else
    return gemm_groups_simt<T>(g, ng, make_scalar<T>(alpha, 0.0), A, lda, sA, B, ldb, sB, add, D, ldd, sD, batch, st);
}

template <class T>
static int merge_impl(const hps_merge_args* a, cudaStream_t st, bool iti) {
  const int nm = a->n_merges, ni = a->n_int, ne = a->n_ext, ns = a->nsrc;
  unsigned char* wsb = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(a->workspace) + 255) & ~uintptr_t(255));
  Carver cv(wsb);
  T* D = a->D_inv ? (T*)a->D_inv : (T*)cv.take(sizeof(T) * (size_t)nm * ni * ni);
  T* C = (T*)cv.take(sizeof(T) * (size_t)nm * ni * ne);
  T* B = (T*)cv.take(sizeof(T) * (size_t)nm * ne * ni);
  if (a->B_out) B = (T*)a->B_out;
  T* dh = (T*)cv.take(sizeof(T) * (size_t)nm * ni * (ns > 0 ? ns : 1));
  const int nx = a->n_x;
  T *X12 = nullptr, *X21 = nullptr, *Wm = nullptr, *Pm = nullptr;
  if (nx > 0) {
    X12 = (T*)cv.take(sizeof(T) * (size_t)nm * nx * nx);
    X21 = (T*)cv.take(sizeof(T) * (size_t)nm * nx * nx);
    Wm = (T*)cv.take(sizeof(T) * (size_t)nm * nx * nx);
    Pm = (T*)cv.take(sizeof(T) * (size_t)nm * nx * nx);
  }
  const size_t invb = stage_inverse_bytes(a->dtype, nx > 0 ? nx : ni, nm, a->info);
  void* invws = cv.take(invb);
  double* rscale = leaf_rows_scaled(DTypeOf<T>::value) ? (double*)cv.take(sizeof(double) * (size_t)nm * ni) : nullptr;
  const bool with_h = ns > 0 && a->h_children && a->h_out && a->g_tilde;
  // with the block rectangles, the zero blocks of C (and of B unless B is
  // returned) are never read: the gather leaves them unwritten
  const bool rects_on = a->n_c_rects > 0 && a->n_b_rects > 0;
  const int skip_zero = rects_on ? (1 | (a->B_out ? 0 : 2)) : 0;
  if (iti)
    HPS_CHECK(merge_gather_iti<T>(nm, a->nch, a->nb, ni, ne, with_h ? ns : 0, (const T*)a->T_children,
                                  with_h ? (const T*)a->h_children : nullptr, a->int_c, a->int_l, a->ext_c, a->ext_l,
                                  D, C, B, (T*)a->T_out, dh, (T*)a->h_out, skip_zero, st));
  else
    HPS_CHECK(merge_gather<T>(nm, a->nch, a->nb, ni, ne, with_h ? ns : 0, (const T*)a->T_children,
                              with_h ? (const T*)a->h_children : nullptr, a->int_c, a->int_l, a->ext_c, a->ext_l,
                              a->loc, D, C, B, (T*)a->T_out, dh, (T*)a->h_out, skip_zero, st));
  const T one_ = one<T>(), zero_ = zero<T>(), mone = make_scalar<T>(-1.0, 0.0);
  // an impedance merge's rows are an identity's and a contraction's: of one scale
  const bool balanced = rscale && !iti && f64_products_on_tensor_cores();
  if constexpr (DTypeOf<T>::value == F64 || DTypeOf<T>::value == C128) {
    if (balanced) HPS_CHECK(balance_rows<T>(nm, ni, ne, with_h ? ns : 0, D, C, with_h ? dh : nullptr, rscale, st));
  }
  if (nx > 0) {
    // D = [[I, D12], [D21, I]] in colour order; W = I - D12 D21,
    // D^-1 = [[W^-1, -W^-1 D12], [-D21 W^-1, I + D21 W^-1 D12]]
    const long long sD = (long long)ni * ni, sx = (long long)nx * nx;
    const int* cp = a->colour_perm;
    HPS_CHECK(perm_gather<T>(nm, ni, nx, nx, D, sD, cp, 0, nx, X12, sx, st));
    HPS_CHECK(perm_gather<T>(nm, ni, nx, nx, D, sD, cp, nx, 0, X21, sx, st));
    HPS_CHECK(gemm_batched<T>(nx, nx, nx, mone, X12, nx, sx, X21, nx, sx, zero_, nullptr, 0, 0, Wm, nx, sx, nm, st));
    HPS_CHECK(add_identity<T>(nm, nx, Wm, sx, st));
    HPS_CHECK(stage_inverse<T>(a->dtype, nx, Wm, nm, a->info, invws, invb, st, 0));
    HPS_CHECK(gemm_batched<T>(nx, nx, nx, mone, Wm, nx, sx, X12, nx, sx, zero_, nullptr, 0, 0, Pm, nx, sx, nm, st));
    HPS_CHECK(perm_scatter<T>(nm, ni, nx, nx, D, sD, cp, 0, 0, Wm, sx, 0, st));
    HPS_CHECK(perm_scatter<T>(nm, ni, nx, nx, D, sD, cp, 0, nx, Pm, sx, 0, st));
    HPS_CHECK(gemm_batched<T>(nx, nx, nx, mone, X21, nx, sx, Wm, nx, sx, zero_, nullptr, 0, 0, X12, nx, sx, nm, st));
    HPS_CHECK(perm_scatter<T>(nm, ni, nx, nx, D, sD, cp, nx, 0, X12, sx, 0, st));
    HPS_CHECK(gemm_batched<T>(nx, nx, nx, mone, X21, nx, sx, Pm, nx, sx, zero_, nullptr, 0, 0, Wm, nx, sx, nm, st));
    HPS_CHECK(perm_scatter<T>(nm, ni, nx, nx, D, sD, cp, nx, nx, Wm, sx, 1, st));
  } else {
    // interface matrices: the recursive block inversion may serve FP32
    HPS_CHECK(stage_inverse<T>(a->dtype, ni, D, nm, a->info, invws, invb, st, INV_BLOCK_RECURSIVE));
  }
  T* S = (T*)a->S;
  const long long sDD = (long long)ni * ni, sC = (long long)ni * ne, sB = (long long)ne * ni, sT = (long long)ne * ne;
  const bool rects = a->n_c_rects > 0 && a->n_b_rects > 0;
  GemmGroup groups[GEMM_GROUPS];
  // FP64: on the digit kernel, or not at all.  FP32: where no block is long
  // enough for the tensor cores' products (from 128 on), which are faster there.
  bool grouped = f64_products_on_tensor_cores();
  if (DTypeOf<T>::value == F32 || DTypeOf<T>::value == C64) {
    grouped = gemm_simt_blocks();
    for (int k = 0; rects_on && k < a->n_c_rects; ++k) grouped = grouped && a->c_rects[5 * k + 1] < 128;
    for (int k = 0; rects_on && k < a->n_b_rects; ++k) grouped = grouped && a->b_rects[5 * k + 3] < 128;
  }
  // S = -D^-1 C
  int ng = rects && grouped ? rect_groups(a, true, ni, groups) : 0;
  if (ng) {
    HPS_CHECK(run_groups<T>(groups, ng, -1.0, D, ni, sDD, C, ne, sC, false, S, ne, sC, nm, st));
  } else if (rects) {
    for (int r = 0; r < a->n_c_rects; ++r) {
      const int* q = a->c_rects + 5 * r;   // i0, n_i, e0, n_e, first
      HPS_CHECK(gemm_batched<T>(ni, q[3], q[1], mone, D + q[0], ni, sDD, C + (long long)q[0] * ne + q[2], ne, sC,
                                q[4] ? zero_ : one_, q[4] ? nullptr : S + q[2], ne, sC, S + q[2], ne, sC, nm, st));
    }
  } else {
    HPS_CHECK(gemm_batched<T>(ni, ne, ni, mone, D, ni, sDD, C, ne, sC, zero_, nullptr, 0, 0, S, ne, sC, nm, st));
  }
  // T_out = A + B S
  if (a->T_out) {
    T* To = (T*)a->T_out;
    ng = rects && grouped ? rect_groups(a, false, ne, groups) : 0;
    if (ng) {
      HPS_CHECK(run_groups<T>(groups, ng, 1.0, B, ni, sB, S, ne, sC, true, To, ne, sT, nm, st));
    } else if (rects) {
      for (int r = 0; r < a->n_b_rects; ++r) {
        const int* q = a->b_rects + 5 * r;   // e0, n_e, i0, n_i, first
        HPS_CHECK(gemm_batched<T>(q[1], ne, q[3], one_, B + (long long)q[0] * ni + q[2], ni, sB,
                                  S + (long long)q[2] * ne, ne, sC, one_, To + (long long)q[0] * ne, ne, sT,
                                  To + (long long)q[0] * ne, ne, sT, nm, st));
      }
    } else {
      HPS_CHECK(gemm_batched<T>(ne, ne, ni, one_, B, ni, sB, S, ne, sC, one_, To, ne, sT, To, ne, sT, nm, st));
    }
  }
  if (with_h) {
    T* gt = (T*)a->g_tilde;
    T* ho = (T*)a->h_out;
    const long long sg = (long long)ni * ns, sh = (long long)ne * ns;
    HPS_CHECK(gemm_batched<T>(ni, ns, ni, mone, D, ni, sDD, dh, ns, sg, zero_, nullptr, 0, 0, gt, ns, sg, nm, st));
    ng = rects && (ns <= 8 || grouped) ? rect_groups(a, false, ns, groups) : 0;
    if (ng && ns <= 8) {
      HPS_CHECK(skinny_groups<T>(groups, ng, ne, ns, B, ni, sB, gt, ns, sg, ho, ns, sh, nm, st));
    } else if (ng) {
      HPS_CHECK(run_groups<T>(groups, ng, 1.0, B, ni, sB, gt, ns, sg, true, ho, ns, sh, nm, st));
    } else if (rects) {
      for (int r = 0; r < a->n_b_rects; ++r) {
        const int* q = a->b_rects + 5 * r;
        HPS_CHECK(gemm_batched<T>(q[1], ns, q[3], one_, B + (long long)q[0] * ni + q[2], ni, sB,
                                  gt + (long long)q[2] * ns, ns, sg, one_, ho + (long long)q[0] * ns, ns, sh,
                                  ho + (long long)q[0] * ns, ns, sh, nm, st));
      }
    } else {
      HPS_CHECK(gemm_batched<T>(ne, ns, ni, one_, B, ni, sB, gt, ns, sg, one_, ho, ns, sh, ho, ns, sh, nm, st));
    }
  }
  if (balanced && (a->D_inv || a->BD_inv)) HPS_CHECK(col_scale<T>(nm, ni, D, ni, sDD, rscale, st));
  // B D^-1
  if (a->BD_inv) {
    T* BD = (T*)a->BD_inv;
    ng = rects && grouped ? rect_groups(a, false, ni, groups) : 0;
    if (ng) {
      HPS_CHECK(run_groups<T>(groups, ng, 1.0, B, ni, sB, D, ni, sDD, false, BD, ni, sB, nm, st));
    } else if (rects) {
      for (int r = 0; r < a->n_b_rects; ++r) {
        const int* q = a->b_rects + 5 * r;
        T* o = BD + (long long)q[0] * ni;
        HPS_CHECK(gemm_batched<T>(q[1], ni, q[3], one_, B + (long long)q[0] * ni + q[2], ni, sB,
                                  D + (long long)q[2] * ni, ni, sDD, q[4] ? zero_ : one_, q[4] ? nullptr : o, ni, sB,
                                  o, ni, sB, nm, st));
      }
    } else {
      HPS_CHECK(gemm_batched<T>(ne, ni, ni, one_, B, ni, sB, D, ni, sDD, zero_, nullptr, 0, 0, BD, ni, sB, nm, st));
    }
  }
  return HPS_OK;
}

// ---------------------------------------------------------------------------
// Down level
// ---------------------------------------------------------------------------
template <class T>
static int down_impl(const hps_down_args* a, cudaStream_t st) {
  const int nm = a->n_merges, ni = a->n_int, ne = a->n_ext, ns = a->nsrc;
  const T one_ = one<T>();
  HPS_CHECK(gemm_batched<T>(ni, ns, ne, one_, (const T*)a->S, ne, (long long)ni * ne, (const T*)a->g_parent, ns,
                            (long long)ne * ns, one_, (const T*)a->g_tilde, ns, (long long)ni * ns, (T*)a->g_int,
                            ns, (long long)ni * ns, nm, st));
  HPS_CHECK(down_scatter<T>(nm, a->nch, a->nb, ne, ni, ns, a->code, (const T*)a->g_parent, (const T*)a->g_int,
                            (T*)a->g_children, st));
  return HPS_OK;
}

template <class T>
static int gemm_entry(bool digits, int m, int n, int k, const double* alpha, const void* A, long long lda, long long sA,
                      const void* B, long long ldb, long long sB, const double* beta, const void* C, long long ldc,
                      long long sC, void* D, long long ldd, long long sD, int batch, void* stream) {
  const T al = make_scalar<T>(alpha ? alpha[0] : 1.0, alpha ? alpha[1] : 0.0);
  const T be = make_scalar<T>(beta ? beta[0] : 0.0, beta ? beta[1] : 0.0);
  HPS_CHECK(gemm_batched<T>(m, n, k, al, (const T*)A, lda, sA, (const T*)B, ldb, sB, be, (const T*)C, ldc, sC,
                            (T*)D, ldd, sD, batch, (cudaStream_t)stream, digits));
  return HPS_OK;
}

template <class T>
static int inverse_entry(int n, const void* A, long long lda, long long sA, void* X, long long ldx, long long sX,
                         int batch, int* info, void* ws, size_t wsb, void* stream, int flags) {
  HPS_CHECK(inverse_batched<T>(n, (const T*)A, lda, sA, (T*)X, ldx, sX, batch, info, ws, wsb,
                               (cudaStream_t)stream, flags));
  return HPS_OK;
}

template <class T>
static int up_impl(const hps_up_args* a, cudaStream_t st) {
  const int nm = a->n_merges, ni = a->n_int, ne = a->n_ext, ns = a->nsrc;
  const T one_ = one<T>(), zero_ = zero<T>(), mone = make_scalar<T>(-1.0, 0.0);
  if (a->flags & HPS_UP_ITI)
    HPS_CHECK(merge_gather_iti<T>(nm, a->nch, a->nb, ni, ne, ns, nullptr, (const T*)a->h_children, a->int_c,
                                  a->int_l, a->ext_c, a->ext_l, nullptr, nullptr, nullptr, nullptr, (T*)a->dh,
                                  (T*)a->h_out, 0, st));
  else
    HPS_CHECK(merge_gather<T>(nm, a->nch, a->nb, ni, ne, ns, nullptr, (const T*)a->h_children, a->int_c, a->int_l,
                              a->ext_c, a->ext_l, nullptr, nullptr, nullptr, nullptr, nullptr, (T*)a->dh,
                              (T*)a->h_out, 0, st));
  HPS_CHECK(gemm_batched<T>(ni, ns, ni, mone, (const T*)a->D_inv, ni, (long long)ni * ni, (const T*)a->dh, ns,
                            (long long)ni * ns, zero_, nullptr, 0, 0, (T*)a->g_tilde, ns, (long long)ni * ns, nm,
                            st));
  if (a->flags & HPS_UP_B_IS_BD_INV)
    HPS_CHECK(gemm_batched<T>(ne, ns, ni, mone, (const T*)a->B, ni, (long long)ne * ni, (const T*)a->dh, ns,
                              (long long)ni * ns, one_, (T*)a->h_out, ns, (long long)ne * ns, (T*)a->h_out, ns,
                              (long long)ne * ns, nm, st));
  else
    HPS_CHECK(gemm_batched<T>(ne, ns, ni, one_, (const T*)a->B, ni, (long long)ne * ni, (const T*)a->g_tilde, ns,
                              (long long)ni * ns, one_, (T*)a->h_out, ns, (long long)ne * ns, (T*)a->h_out, ns,
                              (long long)ne * ns, nm, st));
  return HPS_OK;
}

template <class T>
static int panel_map_entry(int mode, int batch, int n_out, int n_other, int m_len, const int* tab, const void* M,
                           const void* in, long long ld_in, long long s_in, void* out, long long ld_out,
                           long long s_out, void* stream) {
  HPS_CHECK(panel_map<T>(mode, batch, n_out, n_other, m_len, tab, (const T*)M, (const T*)in, ld_in, s_in, (T*)out,
                         ld_out, s_out, (cudaStream_t)stream));
  return HPS_OK;
}

template <class T>
static int scale_entry(int batch, long long n_per, const double* scale, void* x, void* stream) {
  HPS_CHECK(scale_batched<T>(batch, n_per, scale, (T*)x, (cudaStream_t)stream));
  return HPS_OK;
}

}  // namespace hps

using namespace hps;

#define DISPATCH(dt, FN, ...)                                                  \
  switch (dt) {                                                                \
    case HPS_F64: return FN<double>(__VA_ARGS__);                              \
    case HPS_F32: return FN<float>(__VA_ARGS__);                               \
    case HPS_C128: return FN<c128>(__VA_ARGS__);                               \
    case HPS_C64: return FN<c64>(__VA_ARGS__);                                 \
    default: set_error("unknown dtype %d", (int)(dt)); return HPS_ERR_ARG;     \
  }

extern "C" {

const char* hps_version(void) { return "jaxhps_gb300 0.1.0 (sm_103a)"; }

long long hps_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }

int hps_gemm_policy(int policy) { return set_gemm_policy(policy); }

int hps_gemm_tune_set(int M, int N, int K, int batch, int variant) {
  if (gemm_tune_set(M, N, K, batch, variant) != 0) {
    set_error("hps_gemm_tune_set: variant %d out of range", variant);
    return HPS_ERR_ARG;
  }
  return HPS_OK;
}

int hps_gemm_tune_clear(void) {
  gemm_tune_clear();
  return HPS_OK;
}

int hps_gemm_force_variant(int variant) { return gemm_force_variant(variant); }

long long hps_gemm_shapes(int mode, long long* out, long long cap) { return gemm_shapes(mode, out, cap); }

int hps_interp_rows(long long n_rows, int n_src, const double* to_pts, const double* src_pts,
                    const double* src_weights, double* out, int rows_per_group, int transposed, void* stream) {
  if (n_rows < 0 || n_src <= 0 || !to_pts || !src_pts || !src_weights || !out || rows_per_group <= 0 ||
      (transposed && n_rows % rows_per_group != 0)) {
    set_error("hps_interp_rows: invalid arguments");
    return HPS_ERR_ARG;
  }
  HPS_CHECK(interp_rows(n_rows, n_src, to_pts, src_pts, src_weights, out, rows_per_group, transposed,
                        (cudaStream_t)stream));
  return HPS_OK;
}

int hps_gather_cols(long long n_groups, int n_in, int n_out, const int* idx, const double* in, double* out,
                    void* stream) {
  if (n_groups < 0 || n_in <= 0 || n_out <= 0 || !idx || !in || !out) {
    set_error("hps_gather_cols: invalid arguments");
    return HPS_ERR_ARG;
  }
  HPS_CHECK(gather_cols(n_groups, n_in, n_out, idx, in, out, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_interp_leaf_nodes(int dim, long long n_leaves, int p, const double* leaf_bounds, const double* ref_nodes,
                          double* leaf_nodes, double* leaf_weights, void* stream) {
  if ((dim != 2 && dim != 3) || n_leaves < 0 || p < 2 || !leaf_bounds || !ref_nodes || !leaf_nodes || !leaf_weights) {
    set_error("hps_interp_leaf_nodes: invalid arguments");
    return HPS_ERR_ARG;
  }
  HPS_CHECK(interp_leaf_nodes(dim, n_leaves, p, leaf_bounds, ref_nodes, leaf_nodes, leaf_weights,
                              (cudaStream_t)stream));
  return HPS_OK;
}

int hps_interp_from_leaves(int dim, long long n_targets, int nsrc, const double* targets, int p,
                           const double* leaf_bounds, const double* leaf_nodes, const double* leaf_weights,
                           const int* rearrange, const int* cells, const int* n_cells, const double* cell_origin,
                           const double* cell_size, const double* f, double* out, void* stream) {
  if ((dim != 2 && dim != 3) || n_targets < 0 || nsrc <= 0 || p < 2 || p > 32 || !targets || !leaf_bounds ||
      !leaf_nodes || !leaf_weights || !rearrange || !cells || !n_cells || !cell_origin || !cell_size || !f || !out) {
    set_error("hps_interp_from_leaves: invalid arguments");
    return HPS_ERR_ARG;
  }
  for (int a = 0; a < dim; ++a)
    if (n_cells[a] <= 0 || !(cell_size[a] > 0.0)) {
      set_error("hps_interp_from_leaves: invalid cell table");
      return HPS_ERR_ARG;
    }
  HPS_CHECK(interp_from_leaves(dim, n_targets, nsrc, targets, p, leaf_bounds, leaf_nodes, leaf_weights, rearrange,
                               cells, n_cells, cell_origin, cell_size, f, out, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_gemm_tc_status(void) { return gemm_tc_error(); }

int hps_gemm_tc_status_reset(void) { return gemm_tc_error_reset(); }

int hps_inverse_policy(int policy) { return set_inverse_tc_policy(policy); }

int hps_inverse_block_policy(int policy) { return set_inverse_rec_policy(policy); }

int hps_set_spin_limits(long long panel_barrier_polls, long long tc_wait_polls, long long* prev_panel,
                        long long* prev_tc) {
  cudaError_t e = set_panel_spin_limit(panel_barrier_polls, prev_panel);
  if (e == cudaSuccess) e = set_tc_spin_limit(tc_wait_polls, prev_tc);
  if (e == cudaSuccess) e = set_itc_spin_limit(tc_wait_polls, nullptr);
  if (e != cudaSuccess) {
    set_error("hps_set_spin_limits: %s", cudaGetErrorString(e));
    return HPS_ERR_CUDA;
  }
  return HPS_OK;
}

int hps_profile_begin(int class_mask) {
  g_prof.mask = (unsigned)class_mask;
  g_prof.used = 0;
  for (int c = 0; c < N_KC; ++c) {
    g_prof.work[c] = 0.0;
    g_prof.launches[c] = 0;
  }
  return HPS_OK;
}

int hps_profile_end(double* total_ms, long long* launches, double* work) {
  double tot[N_KC] = {0};
  for (int i = 0; i < g_prof.used; ++i) {
    float ms = 0.f;
    if (cudaEventSynchronize(g_prof.ev[2 * i + 1]) != cudaSuccess ||
        cudaEventElapsedTime(&ms, g_prof.ev[2 * i], g_prof.ev[2 * i + 1]) != cudaSuccess) {
      set_error("hps_profile_end: event query failed");
      g_prof.mask = 0;
      return HPS_ERR_CUDA;
    }
    tot[g_prof.slot_cls[i]] += ms;
  }
  for (int c = 0; c < N_KC; ++c) {
    if (total_ms) total_ms[c] = tot[c];
    if (launches) launches[c] = g_prof.launches[c];
    if (work) work[c] = g_prof.work[c];
  }
  g_prof.mask = 0;
  g_prof.used = 0;
  return HPS_OK;
}

int hps_last_error(char* buf, size_t len) {
  if (buf && len) {
    strncpy(buf, g_last_error.c_str(), len - 1);
    buf[len - 1] = 0;
  }
  return (int)g_last_error.size();
}

int hps_gemm_batched(int dtype, int m, int n, int k, const double* alpha, const void* A, long long lda,
                     long long strideA, const void* B, long long ldb, long long strideB, const double* beta,
                     const void* C, long long ldc, long long strideC, void* D, long long ldd, long long strideD,
                     int batch, void* stream) {
  if (m < 0 || n < 0 || k < 0 || batch < 0 || (!A && m * k > 0) || (!B && k * n > 0) || (!D && m * n > 0)) {
    set_error("hps_gemm_batched: invalid arguments");
    return HPS_ERR_ARG;
  }
  DISPATCH(dtype & ~HPS_PRODUCT_DIGITS, gemm_entry, (dtype & HPS_PRODUCT_DIGITS) != 0, m, n, k, alpha, A, lda, strideA,
           B, ldb, strideB, beta, C, ldc, strideC, D, ldd, strideD, batch, stream)
}

size_t hps_inverse_workspace_size(int dtype, int n, int batch) {
  return inverse_workspace_bytes(dtype, n, batch);
}


int hps_inverse_batched(int dtype, int n, const void* A, long long lda, long long strideA, void* X, long long ldx,
                        long long strideX, int batch, int* info, void* workspace, size_t workspace_bytes,
                        void* stream) {
  if (n < 0 || batch < 0 || !A || !X) {
    set_error("hps_inverse_batched: invalid arguments");
    return HPS_ERR_ARG;
  }
  if (workspace_bytes < inverse_workspace_bytes(dtype, n, batch)) {
    set_error("hps_inverse_batched: workspace too small (%zu < %zu)", workspace_bytes,
              inverse_workspace_bytes(dtype, n, batch));
    return HPS_ERR_WORKSPACE;
  }
  DISPATCH(dtype, inverse_entry, n, A, lda, strideA, X, ldx, strideX, batch, info, workspace, workspace_bytes,
           stream, 0)
}

int hps_inverse_interface(int dtype, int n, const void* A, long long lda, long long strideA, void* X, long long ldx,
                          long long strideX, int batch, int* info, void* workspace, size_t workspace_bytes,
                          void* stream) {
  if (n < 0 || batch < 0 || !A || !X) {
    set_error("hps_inverse_interface: invalid arguments");
    return HPS_ERR_ARG;
  }
  if (workspace_bytes < inverse_workspace_bytes(dtype, n, batch)) {
    set_error("hps_inverse_interface: workspace too small (%zu < %zu)", workspace_bytes,
              inverse_workspace_bytes(dtype, n, batch));
    return HPS_ERR_WORKSPACE;
  }
  DISPATCH(dtype, inverse_entry, n, A, lda, strideA, X, ldx, strideX, batch, info, workspace, workspace_bytes,
           stream, INV_BLOCK_RECURSIVE)
}

int hps_convert(int ds, int dd, long long n, const void* src, void* dst, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (!src || !dst || n < 0) {
    set_error("hps_convert: invalid arguments");
    return HPS_ERR_ARG;
  }
  if (ds == HPS_F64 && dd == HPS_F32) HPS_CHECK(convert<double, float>(n, (const double*)src, (float*)dst, st));
  else if (ds == HPS_F32 && dd == HPS_F64) HPS_CHECK(convert<float, double>(n, (const float*)src, (double*)dst, st));
  else if (ds == HPS_C128 && dd == HPS_C64) HPS_CHECK(convert<c128, c64>(n, (const c128*)src, (c64*)dst, st));
  else if (ds == HPS_C64 && dd == HPS_C128) HPS_CHECK(convert<c64, c128>(n, (const c64*)src, (c128*)dst, st));
  else {
    set_error("hps_convert: unsupported pair %d -> %d", ds, dd);
    return HPS_ERR_ARG;
  }
  return HPS_OK;
}

size_t hps_local_solve_dtn_workspace_size(const hps_leaf_dtn_args* a) {
  Carver cv(nullptr);
  return leaf_dtn_ws(a, &cv);
}

int hps_local_solve_dtn(const hps_leaf_dtn_args* a, void* stream) {
  if (!a || a->n_leaves <= 0 || a->n_pts <= a->n_cb || a->n_cb <= 0 || a->n_gauss <= 0 || a->n_ops <= 0 ||
      !a->ops || !a->coeffs || !a->P || !a->Q || !a->Y || !a->T || !a->Aii_inv) {
    set_error("hps_local_solve_dtn: invalid arguments");
    return HPS_ERR_ARG;
  }
  if (a->nsrc > 0 && (!a->source || !a->v || !a->h)) {
    set_error("hps_local_solve_dtn: nsrc > 0 needs source, v and h");
    return HPS_ERR_ARG;
  }
  if (a->workspace_bytes < hps_local_solve_dtn_workspace_size(a)) {
    set_error("hps_local_solve_dtn: workspace too small (%zu < %zu)", a->workspace_bytes,
              hps_local_solve_dtn_workspace_size(a));
    return HPS_ERR_WORKSPACE;
  }
  DISPATCH(base_dtype(a->dtype), leaf_dtn_impl, a, (cudaStream_t)stream)
}

size_t hps_local_solve_iti_workspace_size(const hps_leaf_iti_args* a) {
  Carver cv(nullptr);
  return leaf_iti_ws(a, &cv);
}

int hps_local_solve_iti(const hps_leaf_iti_args* a, void* stream) {
  if (!a || a->n_leaves <= 0 || a->n_pts <= a->n_cb || a->n_cb <= 0 || a->n_gauss <= 0 || a->n_ops <= 0 ||
      !a->ops || !a->coeffs || !a->G || !a->P || !a->QH || !a->Y || !a->T || !a->B_inv ||
      (base_dtype(a->dtype) != HPS_C128 && base_dtype(a->dtype) != HPS_C64)) {
    set_error("hps_local_solve_iti: invalid arguments");
    return HPS_ERR_ARG;
  }
  if (a->nsrc > 0 && (!a->source || !a->v || !a->h)) {
    set_error("hps_local_solve_iti: nsrc > 0 needs source, v and h");
    return HPS_ERR_ARG;
  }
  if (a->workspace_bytes < hps_local_solve_iti_workspace_size(a)) {
    set_error("hps_local_solve_iti: workspace too small");
    return HPS_ERR_WORKSPACE;
  }
  if (base_dtype(a->dtype) == HPS_C128) return leaf_iti_impl<c128>(a, (cudaStream_t)stream);
  return leaf_iti_impl<c64>(a, (cudaStream_t)stream);
}

size_t hps_merge_level_dtn_workspace_size(const hps_merge_args* a) {
  Carver cv(nullptr);
  return merge_ws(a, &cv);
}

// Rectangles of the block-structured merge products: in bounds, and over the
// exterior index each range is written first by the rectangle marked `first`
// and only accumulated afterwards, with every exterior index covered.
static bool rects_ok(int n, const int* r, int n_int, int n_ext, bool c_form) {
  std::vector<char> done(n_ext, 0);
  for (int k = 0; k < n; ++k) {
    const int* q = r + 5 * k;
    const int i0 = c_form ? q[0] : q[2], li = c_form ? q[1] : q[3];
    const int e0 = c_form ? q[2] : q[0], le = c_form ? q[3] : q[1];
    if (i0 < 0 || li <= 0 || i0 + li > n_int || e0 < 0 || le <= 0 || e0 + le > n_ext || (q[4] != 0 && q[4] != 1))
      return false;
    for (int e = e0; e < e0 + le; ++e) {
      if ((bool)done[e] == (bool)q[4]) return false;
      done[e] = 1;
    }
  }
  for (int e = 0; e < n_ext; ++e)
    if (!done[e]) return false;
  return true;
}

static int check_merge_rects(const hps_merge_args* a, const char* who) {
  if (a->n_c_rects == 0 && a->n_b_rects == 0) return HPS_OK;
  if (a->n_c_rects <= 0 || a->n_b_rects <= 0 || !a->c_rects || !a->b_rects ||
      !rects_ok(a->n_c_rects, a->c_rects, a->n_int, a->n_ext, true) ||
      !rects_ok(a->n_b_rects, a->b_rects, a->n_int, a->n_ext, false)) {
    set_error("%s: invalid block rectangles", who);
    return HPS_ERR_ARG;
  }
  return HPS_OK;
}

int hps_merge_level_dtn(const hps_merge_args* a, void* stream) {
  if (!a || a->n_merges <= 0 || a->nch <= 0 || a->nb <= 0 || a->n_int <= 0 || a->n_ext <= 0 || !a->T_children ||
      !a->int_c || !a->int_l || !a->ext_c || !a->ext_l || !a->loc || !a->S) {
    set_error("hps_merge_level_dtn: invalid arguments");
    return HPS_ERR_ARG;
  }
  if (a->workspace_bytes < hps_merge_level_dtn_workspace_size(a)) {
    set_error("hps_merge_level_dtn: workspace too small (%zu < %zu)", a->workspace_bytes,
              hps_merge_level_dtn_workspace_size(a));
    return HPS_ERR_WORKSPACE;
  }
  if (check_merge_rects(a, "hps_merge_level_dtn") != HPS_OK) return HPS_ERR_ARG;
  if (a->n_x != 0) {
    set_error("hps_merge_level_dtn: the two-colour inverse applies to ItI merges only");
    return HPS_ERR_ARG;
  }
  DISPATCH(base_dtype(a->dtype), merge_impl, a, (cudaStream_t)stream, false)
}

int hps_merge_level_iti(const hps_merge_args* a, void* stream) {
  if (!a || a->n_merges <= 0 || a->nch <= 0 || a->nb <= 0 || a->n_int <= 0 || a->n_ext <= 0 || !a->T_children ||
      !a->int_c || !a->int_l || !a->ext_c || !a->ext_l || !a->S) {
    set_error("hps_merge_level_iti: invalid arguments");
    return HPS_ERR_ARG;
  }
  if (a->workspace_bytes < hps_merge_level_dtn_workspace_size(a)) {
    set_error("hps_merge_level_iti: workspace too small (%zu < %zu)", a->workspace_bytes,
              hps_merge_level_dtn_workspace_size(a));
    return HPS_ERR_WORKSPACE;
  }
  if (check_merge_rects(a, "hps_merge_level_iti") != HPS_OK) return HPS_ERR_ARG;
  if (a->n_x < 0 || (a->n_x > 0 && (2 * a->n_x != a->n_int || !a->colour_perm))) {
    set_error("hps_merge_level_iti: two-colour structure needs n_x = n_int / 2 and colour_perm");
    return HPS_ERR_ARG;
  }
  DISPATCH(base_dtype(a->dtype), merge_impl, a, (cudaStream_t)stream, true)
}

int hps_up_level(const hps_up_args* a, void* stream) {
  if (!a || a->n_merges <= 0 || a->nsrc <= 0 || !a->h_children || !a->D_inv || !a->B || !a->dh || !a->g_tilde ||
      !a->h_out || !a->int_c || !a->int_l || !a->ext_c || !a->ext_l) {
    set_error("hps_up_level: invalid arguments");
    return HPS_ERR_ARG;
  }
  DISPATCH(a->dtype, up_impl, a, (cudaStream_t)stream)
}

static int pack_kinds(int n_ops, const int* op_kind, unsigned long long* kinds, int* need_uy) {
  // op kinds packed 4 bits each; D_xy needs the u_y field on the whole grid
  if (n_ops > 10) {
    set_error("residual: at most 10 operators");
    return HPS_ERR_ARG;
  }
  *kinds = 0;
  *need_uy = 0;
  for (int o = 0; o < n_ops; ++o) {
    if (op_kind[o] < 0 || op_kind[o] > 5) {
      set_error("residual: bad op kind %d", op_kind[o]);
      return HPS_ERR_ARG;
    }
    *kinds |= (unsigned long long)op_kind[o] << (4 * o);
    if (op_kind[o] == 1) *need_uy = 1;
  }
  return HPS_OK;
}

static int pack_op_kinds(const hps_residual2d_args* a, unsigned long long* kinds, int* need_uy) {
  return pack_kinds(a->n_ops, a->op_kind, kinds, need_uy);
}

int hps_residual_iti_2d(const hps_residual_iti2d_args* a, void* stream) {
  if (!a || a->n_leaves <= 0 || a->p < 3 || a->q <= 0 || a->nsrc <= 0 || a->n_ops <= 0 || !a->coeffs ||
      !a->inv_half || !a->D1 || !a->D2 || !a->Pside || !a->Qside || !a->perm || !a->u || !a->t_in || !a->r ||
      !a->t_out) {
    set_error("hps_residual_iti_2d: invalid arguments");
    return HPS_ERR_ARG;
  }
  if (a->n_leaves > 2147483647 || (a->nsrc + 15) / 16 > 65535) {
    set_error("hps_residual_iti_2d: too many right-hand sides");
    return HPS_ERR_ARG;
  }
  unsigned long long kinds = 0;
  int need_uy = 0;
  if (pack_kinds(a->n_ops, a->op_kind, &kinds, &need_uy) != HPS_OK) return HPS_ERR_ARG;
  cudaError_t e = residual_iti_2d(a->n_leaves, a->p, a->q, a->nsrc, a->n_ops, kinds, a->coef_complex, a->eta,
                                  a->coeffs, a->inv_half, a->D1, a->D2, a->Pside, a->Qside, a->perm, a->u, a->t_in,
                                  a->f, a->r, a->t_out, need_uy, (cudaStream_t)stream);
  if (e == cudaErrorInvalidValue) {
    set_error("hps_residual_iti_2d: p, q too large for the shared-memory layout");
    return HPS_ERR_ARG;
  }
  HPS_CHECK(e);
  return HPS_OK;
}

int hps_residual_update_2d(const hps_residual2d_args* a, const float* du, const float* dg, void* stream) {
  if (!a || a->n_leaves <= 0 || a->p < 3 || a->q <= 0 || a->nsrc <= 0 || a->n_ops <= 0 || !a->coeffs ||
      !a->inv_half || !a->D1 || !a->D2 || !a->Pside || !a->Qside || !a->perm || !du || !dg || !a->r_int ||
      !a->r_int64 || !a->flux) {
    set_error("hps_residual_update_2d: invalid arguments");
    return HPS_ERR_ARG;
  }
  if ((a->nsrc + 15) / 16 > 65535) {
    set_error("hps_residual_update_2d: too many right-hand sides");
    return HPS_ERR_ARG;
  }
  unsigned long long kinds = 0;
  int need_uy = 0;
  if (pack_op_kinds(a, &kinds, &need_uy) != HPS_OK) return HPS_ERR_ARG;
  HPS_CHECK(jx_update_2d(a->n_leaves, a->p, a->q, a->nsrc, a->n_ops, kinds, a->coeffs, a->inv_half, a->D1, a->D2,
                         a->Pside, a->Qside, a->perm, du, dg, a->r_int64, a->r_int, a->flux, need_uy,
                         (cudaStream_t)stream));
  return HPS_OK;
}

int hps_residual_df_supported(int p, int q) { return jx_df_supported(p, q) ? 1 : 0; }

int hps_mapped_pointer(const void* host, void** device) {
  if (!host || !device) {
    set_error("hps_mapped_pointer: invalid arguments");
    return HPS_ERR_ARG;
  }
  *device = nullptr;
  const cudaError_t e = cudaHostGetDevicePointer(device, const_cast<void*>(host), 0);
  if (e != cudaSuccess) {
    cudaGetLastError();
    *device = nullptr;
    set_error("hps_mapped_pointer: not page-locked host memory mapped for the device (%s)", cudaGetErrorString(e));
    return HPS_ERR_ARG;
  }
  return HPS_OK;
}

size_t hps_residual_df_prep_size(int n_leaves, int p, int q, int n_ops) {
  if (n_leaves <= 0 || n_ops <= 0 || n_ops > 10 || !jx_df_supported(p, q)) return 0;
  return jx_df_prep_floats(n_leaves, p, q, n_ops) * sizeof(float);
}

static int check_df_args(const hps_residual2d_args* a, const char* who) {
  if (!a || a->n_leaves <= 0 || a->p < 3 || a->q <= 0 || a->nsrc <= 0 || a->n_ops <= 0 || !a->inv_half ||
      !a->perm) {
    set_error("%s: invalid arguments", who);
    return HPS_ERR_ARG;
  }
  if (!jx_df_supported(a->p, a->q)) {
    set_error("%s: p = %d, q = %d not supported (q = p - 2 with p in 8, 10, 12, 14, 16)", who, a->p, a->q);
    return HPS_ERR_ARG;
  }
  return HPS_OK;
}

int hps_residual_df_prepare(const hps_residual2d_args* a, float* prep, void* stream) {
  if (check_df_args(a, "hps_residual_df_prepare") != HPS_OK) return HPS_ERR_ARG;
  if (!prep || !a->coeffs || !a->D1 || !a->D2 || !a->Pside || !a->Qside) {
    set_error("hps_residual_df_prepare: invalid arguments");
    return HPS_ERR_ARG;
  }
  unsigned long long kinds = 0;
  int need_uy = 0;
  if (pack_op_kinds(a, &kinds, &need_uy) != HPS_OK) return HPS_ERR_ARG;
  HPS_CHECK(jx_df_prepare(a->n_leaves, a->p, a->q, a->n_ops, kinds, a->coeffs, a->inv_half, a->D1, a->D2, a->Pside,
                          a->Qside, a->perm, prep, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_residual_update_2d_df(const hps_residual2d_args* a, const float* prep, const float* du, const float* dg,
                              float* r_lo, void* stream) {
  if (check_df_args(a, "hps_residual_update_2d_df") != HPS_OK) return HPS_ERR_ARG;
  if (!prep || !du || !dg || !a->r_int || !r_lo || !a->flux) {
    set_error("hps_residual_update_2d_df: invalid arguments");
    return HPS_ERR_ARG;
  }
  if ((a->nsrc + 15) / 16 > 65535) {
    set_error("hps_residual_update_2d_df: too many right-hand sides");
    return HPS_ERR_ARG;
  }
  unsigned long long kinds = 0;
  int need_uy = 0;
  if (pack_op_kinds(a, &kinds, &need_uy) != HPS_OK) return HPS_ERR_ARG;
  HPS_CHECK(jx_df_update_2d(a->n_leaves, a->p, a->q, a->nsrc, a->n_ops, kinds, prep, a->inv_half, a->perm, du, dg,
                            a->r_int, r_lo, a->flux, need_uy, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_assemble_u_2d(int n_leaves, int p, int q, int nsrc, const double* Pside, const double* u_int,
                      const double* g, double* u_full, void* stream) {
  if (n_leaves <= 0 || p < 3 || q <= 0 || nsrc <= 0 || !Pside || !u_int || !g || !u_full) {
    set_error("hps_assemble_u_2d: invalid arguments");
    return HPS_ERR_ARG;
  }
  HPS_CHECK(assemble_u_2d(n_leaves, p, q, nsrc, Pside, u_int, g, u_full, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_refine_points_3d(int n_nodes, int p, const double* bounds, const double* cheb, const int* perm,
                         double* pts, void* stream) {
  if (n_nodes < 0 || p < 2 || !bounds || !cheb || !perm || !pts) {
    set_error("hps_refine_points_3d: invalid arguments");
    return HPS_ERR_ARG;
  }
  if (n_nodes == 0) return HPS_OK;
  HPS_CHECK(refine_points_3d(n_nodes, p, bounds, cheb, perm, pts, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_refine_check_3d(int n_nodes, int p, const double* f_values, const int* perm, const int* iperm,
                        const double* interp_lo, const double* interp_hi, const double* cc_weights,
                        const double* bounds, double* diff_max, double* ref_max, double* l2_err, void* stream) {
  if (n_nodes < 0 || p < 2 || p > 16 || !f_values || !perm || !iperm || !interp_lo || !interp_hi || !cc_weights ||
      !bounds || !diff_max || !ref_max) {
    set_error("hps_refine_check_3d: invalid arguments (2 <= p <= 16)");
    return HPS_ERR_ARG;
  }
  if (n_nodes == 0) return HPS_OK;
  HPS_CHECK(refine_check_3d(n_nodes, p, f_values, perm, iperm, interp_lo, interp_hi, cc_weights, bounds, diff_max,
                            ref_max, l2_err, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_refine_points_2d(int n_nodes, int p, const double* bounds, const double* cheb, const int* perm,
                         double* pts, void* stream) {
  if (n_nodes < 0 || p < 2 || !bounds || !cheb || !perm || !pts) {
    set_error("hps_refine_points_2d: invalid arguments");
    return HPS_ERR_ARG;
  }
  if (n_nodes == 0) return HPS_OK;
  HPS_CHECK(refine_points_2d(n_nodes, p, bounds, cheb, perm, pts, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_refine_check_2d(int n_nodes, int p, const double* f_values, const int* perm, const int* iperm,
                        const double* interp_lo, const double* interp_hi, const double* cc_weights,
                        const double* bounds, double* diff_max, double* ref_max, double* l2_err, void* stream) {
  if (n_nodes < 0 || p < 2 || p > 64 || !f_values || !perm || !iperm || !interp_lo || !interp_hi || !cc_weights ||
      !bounds || !diff_max || !ref_max) {
    set_error("hps_refine_check_2d: invalid arguments (2 <= p <= 64)");
    return HPS_ERR_ARG;
  }
  if (n_nodes == 0) return HPS_OK;
  HPS_CHECK(refine_check_2d(n_nodes, p, f_values, perm, iperm, interp_lo, interp_hi, cc_weights, bounds, diff_max,
                            ref_max, l2_err, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_panel_map(int dtype, int mode, int batch, int n_out, int n_other, int m_len, const int* table,
                  const void* M, const void* in, long long ld_in, long long stride_in, void* out, long long ld_out,
                  long long stride_out, void* stream) {
  if ((mode != 0 && mode != 1) || batch < 0 || n_out < 0 || n_other < 0 || (batch > 0 && (!table || !in || !out))) {
    set_error("hps_panel_map: invalid arguments");
    return HPS_ERR_ARG;
  }
  switch (dtype) {
    case HPS_F64: return panel_map_entry<double>(mode, batch, n_out, n_other, m_len, table, M, in, ld_in, stride_in,
                                                 out, ld_out, stride_out, stream);
    case HPS_F32: return panel_map_entry<float>(mode, batch, n_out, n_other, m_len, table, M, in, ld_in, stride_in,
                                                out, ld_out, stride_out, stream);
    case HPS_C128: return panel_map_entry<c128>(mode, batch, n_out, n_other, m_len, table, M, in, ld_in, stride_in,
                                                out, ld_out, stride_out, stream);
    case HPS_C64: return panel_map_entry<c64>(mode, batch, n_out, n_other, m_len, table, M, in, ld_in, stride_in,
                                              out, ld_out, stride_out, stream);
    default: set_error("hps_panel_map: unknown dtype %d", dtype); return HPS_ERR_ARG;
  }
}

int hps_scale_batched(int dtype, int batch, long long n_per, const double* scale, void* x, void* stream) {
  if (batch < 0 || n_per < 0 || (batch > 0 && (!scale || !x))) {
    set_error("hps_scale_batched: invalid arguments");
    return HPS_ERR_ARG;
  }
  DISPATCH(dtype, scale_entry, batch, n_per, scale, x, stream)
}

int hps_mlp_param_count(void) { return mlp_param_count(); }

int hps_mlp_sample_points(int n, const double* bounds, double* pts, void* stream) {
  if (n < 0 || (n > 0 && (!bounds || !pts))) {
    set_error("hps_mlp_sample_points: invalid arguments");
    return HPS_ERR_ARG;
  }
  HPS_CHECK(mlp_sample_points(n, bounds, pts, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_mlp_features(int n, const double* f_samples, const int* depth, double scale, float* X, void* stream) {
  if (n < 0 || !(scale != 0.0) || (n > 0 && (!f_samples || !depth || !X))) {
    set_error("hps_mlp_features: invalid arguments (scale must be non-zero)");
    return HPS_ERR_ARG;
  }
  HPS_CHECK(mlp_features(n, f_samples, depth, 1.0 / scale, X, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_mlp_forward(int n, const float* X, const float* params, float* H1, float* H2, float* logit, void* stream) {
  if (n < 0 || (n > 0 && (!X || !params || !logit))) {
    set_error("hps_mlp_forward: invalid arguments");
    return HPS_ERR_ARG;
  }
  HPS_CHECK(mlp_forward(n, X, params, H1, H2, logit, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_mlp_bce(int n, const float* logit, const float* labels, float pos_weight, float* dlogit, float* loss_sum,
                void* stream) {
  if (n < 0 || (n > 0 && (!logit || !labels || !dlogit))) {
    set_error("hps_mlp_bce: invalid arguments");
    return HPS_ERR_ARG;
  }
  HPS_CHECK(mlp_bce(n, logit, labels, pos_weight, dlogit, loss_sum, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_mlp_backward(int n, const float* X, const float* params, const float* H1, const float* H2,
                     const float* dlogit, float* grad, void* stream) {
  if (n < 0 || (n > 0 && (!X || !params || !H1 || !H2 || !dlogit || !grad))) {
    set_error("hps_mlp_backward: invalid arguments");
    return HPS_ERR_ARG;
  }
  HPS_CHECK(mlp_backward(n, X, params, H1, H2, dlogit, grad, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_mlp_adam(float* params, const float* grad, float* m, float* v, float lr, float beta1, float beta2, float eps,
                 int step, void* stream) {
  if (!params || !grad || !m || !v || step < 1) {
    set_error("hps_mlp_adam: invalid arguments");
    return HPS_ERR_ARG;
  }
  HPS_CHECK(mlp_adam(params, grad, m, v, lr, beta1, beta2, eps, step, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_iti_combine(long long n_nodes, int nsrc, const int* nbr, const void* t_out, const void* t_in, void* hcorr,
                    int n_bdry, const int* bdry_node, const void* t_given, void* r_bdry, void* stream) {
  if (n_nodes <= 0 || nsrc <= 0 || !nbr || !t_out || !t_in || !hcorr || n_bdry < 0 ||
      (n_bdry > 0 && (!bdry_node || !r_bdry))) {
    set_error("hps_iti_combine: invalid arguments");
    return HPS_ERR_ARG;
  }
  HPS_CHECK(iti_combine(n_nodes, nsrc, nbr, t_out, t_in, hcorr, n_bdry, bdry_node, t_given, r_bdry,
                        (cudaStream_t)stream));
  return HPS_OK;
}

int hps_assemble_rows_complex(int n_leaves, int n_pts, int row0, int n_rows, int n_ops, const double* ops,
                              const void* coeffs, void* out, long long ld, long long stride, void* stream) {
  if (n_leaves <= 0 || n_pts <= 0 || row0 < 0 || n_rows <= 0 || row0 + n_rows > n_pts || n_ops <= 0 || !ops ||
      !coeffs || !out || ld < n_pts || stride < (long long)n_rows * ld) {
    set_error("hps_assemble_rows_complex: invalid arguments");
    return HPS_ERR_ARG;
  }
  HPS_CHECK(leaf_assemble<c128, c128>(n_leaves, n_pts, row0, n_rows, n_pts, n_ops, ops, (const c128*)coeffs,
                                      (c128*)out, ld, stride, nullptr, 0, 0, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_assemble_rows(int n_leaves, int n_pts, int row0, int n_rows, int n_ops, const double* ops,
                      const double* coeffs, double* out, long long ld, long long stride, void* stream) {
  if (n_leaves <= 0 || n_pts <= 0 || row0 < 0 || n_rows <= 0 || row0 + n_rows > n_pts || n_ops <= 0 || !ops ||
      !coeffs || !out || ld < n_pts || stride < (long long)n_rows * ld) {
    set_error("hps_assemble_rows: invalid arguments");
    return HPS_ERR_ARG;
  }
  HPS_CHECK(leaf_assemble<double, double>(n_leaves, n_pts, row0, n_rows, n_pts, n_ops, ops, coeffs, out, ld, stride,
                                          nullptr, 0, 0, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_interior_f32(long long n_leaves, int n_pts, int n_cb, int nsrc, const double* f, float* r32, void* stream) {
  if (n_leaves <= 0 || n_pts <= n_cb || nsrc <= 0 || !f || !r32) {
    set_error("hps_interior_f32: invalid arguments");
    return HPS_ERR_ARG;
  }
  HPS_CHECK(interior_f32(n_leaves, n_pts, n_cb, nsrc, f, r32, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_residual_2d(const hps_residual2d_args* a, void* stream) {
  if (!a || a->n_leaves <= 0 || a->p < 3 || a->q <= 0 || a->nsrc <= 0 || a->n_ops <= 0 ||
      !a->coeffs || !a->inv_half || !a->D1 || !a->D2 || !a->Pside || !a->Qside || !a->perm || !a->u_int || !a->g ||
      !a->r_int || !a->flux) {
    set_error("hps_residual_2d: invalid arguments");
    return HPS_ERR_ARG;
  }
  if (a->n_leaves > 2147483647 || (a->nsrc + 15) / 16 > 65535) {
    set_error("hps_residual_2d: too many right-hand sides");
    return HPS_ERR_ARG;
  }
  unsigned long long kinds = 0;
  int need_uy = 0;
  if (pack_op_kinds(a, &kinds, &need_uy) != HPS_OK) return HPS_ERR_ARG;
  HPS_CHECK(residual_2d(a->n_leaves, a->p, a->q, a->nsrc, a->n_ops, kinds, a->coeffs, a->inv_half, a->D1, a->D2,
                        a->Pside, a->Qside, a->perm, a->u_int, a->g, a->f, a->r_int, a->r_int64, nullptr, a->flux,
                        a->u_full, need_uy, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_residual_2d_df(const hps_residual2d_args* a, const float* u_int32, float* r_lo, void* stream) {
  if (!a || a->n_leaves <= 0 || a->p < 3 || a->q <= 0 || a->nsrc <= 0 || a->n_ops <= 0 ||
      !a->coeffs || !a->inv_half || !a->D1 || !a->D2 || !a->Pside || !a->Qside || !a->perm ||
      (!a->u_int && !u_int32) || !a->g || !a->r_int || !r_lo || !a->flux) {
    set_error("hps_residual_2d_df: invalid arguments");
    return HPS_ERR_ARG;
  }
  if (a->n_leaves > 2147483647 || (a->nsrc + 15) / 16 > 65535) {
    set_error("hps_residual_2d_df: too many right-hand sides");
    return HPS_ERR_ARG;
  }
  unsigned long long kinds = 0;
  int need_uy = 0;
  if (pack_op_kinds(a, &kinds, &need_uy) != HPS_OK) return HPS_ERR_ARG;
  HPS_CHECK(residual_2d(a->n_leaves, a->p, a->q, a->nsrc, a->n_ops, kinds, a->coeffs, a->inv_half, a->D1, a->D2,
                        a->Pside, a->Qside, a->perm, a->u_int, a->g, a->f, a->r_int, a->r_int64, r_lo, a->flux,
                        a->u_full, need_uy, (cudaStream_t)stream, u_int32));
  return HPS_OK;
}

int hps_accumulate_max_df(long long n, const float* x, float* y_hi, float* y_lo, double* out, void* stream) {
  if (n < 0 || n % 4 || !x || !y_hi || !y_lo || !out) {
    set_error("hps_accumulate_max_df: invalid arguments (n a multiple of 4, 16-byte aligned arrays)");
    return HPS_ERR_ARG;
  }
  HPS_CHECK(accumulate_pair_max(n, x, y_hi, y_lo, out, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_assemble_u_2d_df(int n_leaves, int p, int q, int nsrc, const double* Pside, const float* u_hi,
                         const float* u_lo, const double* g, double* u_full, void* stream) {
  if (n_leaves <= 0 || p < 3 || q <= 0 || nsrc <= 0 || !Pside || !u_hi || !u_lo || !g || !u_full) {
    set_error("hps_assemble_u_2d_df: invalid arguments");
    return HPS_ERR_ARG;
  }
  HPS_CHECK(assemble_u_pair_2d(n_leaves, p, q, nsrc, Pside, u_hi, u_lo, g, u_full, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_flux_combine(long long n_nodes, int nsrc, const int* nbr, const double* flux, float* hcorr, int n_bdry,
                     const int* bdry_node, const double* g_given, const double* g_state, float* r_bdry,
                     void* stream) {
  if (n_nodes <= 0 || nsrc <= 0 || !nbr || !flux || !hcorr || (n_bdry > 0 && (!bdry_node || !g_state || !r_bdry))) {
    set_error("hps_flux_combine: invalid arguments");
    return HPS_ERR_ARG;
  }
  HPS_CHECK(flux_combine(n_nodes, nsrc, nbr, flux, hcorr, n_bdry, bdry_node, g_given, g_state, r_bdry,
                         (cudaStream_t)stream));
  return HPS_OK;
}

int hps_accumulate_max(long long n, int pairs, const float* x, double* y, double* out, void* stream) {
  if (n < 0 || !x || !y || !out || (pairs && n % 2)) {
    set_error("hps_accumulate_max: invalid arguments");
    return HPS_ERR_ARG;
  }
  HPS_CHECK(accumulate_max(n, pairs, x, y, out, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_accumulate(long long n, const float* x, double* y, void* stream) {
  if (n < 0 || (n > 0 && (!x || !y))) {
    set_error("hps_accumulate: invalid arguments");
    return HPS_ERR_ARG;
  }
  HPS_CHECK(accumulate(n, x, y, (cudaStream_t)stream));
  return HPS_OK;
}

int hps_down_level(const hps_down_args* a, void* stream) {
  if (!a || a->n_merges <= 0 || a->nsrc <= 0 || !a->S || !a->g_parent || !a->code || !a->g_int ||
      !a->g_children) {
    set_error("hps_down_level: invalid arguments");
    return HPS_ERR_ARG;
  }
  DISPATCH(a->dtype, down_impl, a, (cudaStream_t)stream)
}

}  // extern "C"
