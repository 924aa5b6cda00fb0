// noalloc.cu — gpdhg_convergence_noalloc: termination statistics of a candidate solution
// computed without allocating any memory.
//
// Who needs it: callers that may not allocate on the GPU at the moment they want a
// solution checked — code inside a host that owns all device memory through its own pool
// (a Julia CUDA.jl or PyTorch caching allocator that must not be bypassed), a serving path
// with a fixed memory budget, or a process whose device memory is exhausted by design. They
// pass device pointers to the problem vectors, the candidate and its two products, and get
// back the reference's ConvergenceInformation.
//
// The call is synchronous: it ends by copying the statistics to the host and waiting for its
// stream. It therefore cannot run on a stream that is being captured into a CUDA graph; such a
// call is refused with GPDHG_ERR_NOT_SUPPORTED before any other CUDA call, which leaves the
// caller's capture intact.
//
// Scratch: one file-scope device array (kScratchDoubles doubles, 89.3 KiB), which every GPU
// that loads the library holds until the process exits. Its device address is looked up with
// cudaGetSymbolAddress, with the device current, on the first call in each CUDA context (once
// per device, again only if that device's context was destroyed and re-created, since the
// module and its symbol are reloaded then). Every call reuses the same array: each call
// overwrites all partials it reads, so nothing needs clearing, and calls that overlap on the
// GPU (two streams, or two host threads) race on it.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>

#include "eval_kernels.cuh"
#include "host_logic.h"

namespace gpdhg {
namespace {

constexpr long long kNoallocMaxLength = 1LL << 24;                     // n and m at most
// Elements per CTA: as few as one per thread, and about one wave of 4 CTAs on each of 152 SMs for
// both sides together on long vectors; either side then takes at most kNoallocCtas CTAs, for which the
// scratch has room.
constexpr int kNoallocCtas = 600;
constexpr int noalloc_item(long long n, long long m) {
  constexpr long long wave = (long long)kBlock * kNoallocCtas;
  return kBlock * (int)std::max<long long>(1, (n + m + wave - 1) / wave);
}
constexpr int noalloc_items(long long len, int item) { return (int)((len + item - 1) / item); }
static_assert(noalloc_items(kNoallocMaxLength, noalloc_item(kNoallocMaxLength, 0)) <= kNoallocCtas &&
              noalloc_items(kNoallocMaxLength, noalloc_item(kNoallocMaxLength, 1)) <= kNoallocCtas &&
              noalloc_items(kBlock * kNoallocCtas, noalloc_item(kBlock * kNoallocCtas, 0)) <= kNoallocCtas,
              "the scratch holds every CTA's partials");
constexpr int kQn = 10, kQm = 9;
constexpr int kScratchDoubles = (kQn + kQm) * kNoallocCtas + 32;

static __device__ __align__(256) double g_noalloc_scratch[kScratchDoubles];

enum { kA_LuSq = 0, kA_LuMax, kA_Cx, kA_XMax, kA_XSq, kA_RcvSq, kA_RcvMax, kA_Contrib, kA_CSq, kA_CMax };
constexpr unsigned kAMax = (1u << kA_LuMax) | (1u << kA_XMax) | (1u << kA_RcvMax) | (1u << kA_CMax);
enum { kB_CvSq = 0, kB_CvMax, kB_DrSq, kB_DrMax, kB_By, kB_YMax, kB_YSq, kB_BSq, kB_BMax };
constexpr unsigned kBMax = (1u << kB_CvMax) | (1u << kB_DrMax) | (1u << kB_YMax) | (1u << kB_BMax);

// Column side: bound violations, objective, reduced costs of g = c - A'y (the statistics of
// compute_primal_residual!, primal_obj and compute_dual_stats!, src/iteration_stats_utils_gpu.jl:71-238).
struct ColumnStats {
  static constexpr int kQ = kQn;
  static constexpr unsigned kMax = kAMax;
  const double *l, *u, *c, *x, *aty;
  __device__ __forceinline__ void operator()(long long j, double* a) const {
    const double xv = x[j], lv = l[j], uv = u[j], cv = c[j];
    const bool fl = bits_finite(lv), fu = bits_finite(uv);
    add_violation<true>(xv, lv, uv, a[kA_LuSq], a[kA_LuMax]);
    a[kA_Cx] = fma(cv, xv, a[kA_Cx]);
    a[kA_XMax] = nan_max(a[kA_XMax], xv);
    a[kA_XSq] = fma(xv, xv, a[kA_XSq]);
    const double g = cv - aty[j];
    const bool kept = keeps_cost(g, fl, fu);
    const double rcv = cost_residual(g, kept);
    add_square(rcv, a[kA_RcvSq]);
    a[kA_RcvMax] = nan_max(a[kA_RcvMax], rcv);
    add_bound_term<true>(g, kept, lv, uv, a[kA_Contrib]);
    a[kA_CSq] = fma(cv, cv, a[kA_CSq]);
    a[kA_CMax] = nan_max(a[kA_CMax], cv);
  }
};

// Row side: constraint violations of A x, dual sign violations, b'y.
struct RowStats {
  static constexpr int kQ = kQm;
  static constexpr unsigned kMax = kBMax;
  const double *b, *y, *ax;
  int neq;
  __device__ __forceinline__ void operator()(long long i, double* a) const {
    const double bv = b[i], yv = y[i];
    const bool ineq = i >= neq;
    const double cv = row_violation(bv - ax[i], ineq);
    add_square(cv, a[kB_CvSq]);
    a[kB_CvMax] = nan_max(a[kB_CvMax], cv);
    const double dr = dual_violation(yv, ineq);
    add_square(dr, a[kB_DrSq]);
    a[kB_DrMax] = nan_max(a[kB_DrMax], dr);
    a[kB_By] = fma(bv, yv, a[kB_By]);
    a[kB_YMax] = nan_max(a[kB_YMax], yv);
    a[kB_YSq] = fma(yv, yv, a[kB_YSq]);
    a[kB_BSq] = fma(bv, bv, a[kB_BSq]);
    a[kB_BMax] = nan_max(a[kB_BMax], bv);
  }
};

// One side's elements, its CTAs and their partials in the scratch.
template <class F>
struct NoallocSide {
  F f;
  long long len;
  int item;         // elements per CTA
  int items;
  double* partials; // quantity q of CTA k at partials[q * items + k]
};

template <class F>
__device__ __forceinline__ void noalloc_item_sums(const NoallocSide<F>& s, int item, double* sh, double* res) {
  double acc[F::kQ];
#pragma unroll
  for (int q = 0; q < F::kQ; ++q) acc[q] = 0.0;
  const long long b = (long long)item * s.item;
  const long long e = b + s.item < s.len ? b + s.item : s.len;
  for (long long i = b + threadIdx.x; i < e; i += kBlock) s.f(i, acc);
  const double r = block_reduce_q<F::kQ, F::kMax>(acc, sh, res);
  if ((int)threadIdx.x < F::kQ) s.partials[(size_t)threadIdx.x * s.items + item] = r;
}

// Both sides in one launch: the columns' CTAs, then the rows'. Bound by the FP64 pipe (88% busy;
// 104 MB at HBM rate would take 15 us): n = 2M, m = 1M took 163 + 47 us in two launches with a
// shuffle tree per quantity and plainly written arithmetic, and takes 50 us.
__global__ void __launch_bounds__(kBlock, 4) noalloc_reduce_kernel(NoallocSide<ColumnStats> n, NoallocSide<RowStats> m) {
  __shared__ double sh[kQn * kBlock];
  __shared__ double res[kQn];
  if ((int)blockIdx.x < n.items) noalloc_item_sums(n, blockIdx.x, sh, res);
  else noalloc_item_sums(m, (int)blockIdx.x - n.items, sh, res);
}

// One CTA per quantity (columns' then rows'), its items in order; rows' results from out + 16. (5 us; two
// CTAs over all quantities in turn took 19 + 15 us.)
__global__ void __launch_bounds__(kBlock) noalloc_finalize_kernel(const double* part_n, int items_n,
                                                                  const double* part_m, int items_m, double* out) {
  __shared__ double sh[32];
  const bool rows = (int)blockIdx.x >= kQn;
  const int q = rows ? (int)blockIdx.x - kQn : (int)blockIdx.x;
  const bool is_max = ((rows ? kBMax : kAMax) >> q) & 1u;
  const int items = rows ? items_m : items_n;
  const double* p = (rows ? part_m : part_n) + (size_t)q * items;
  double a = 0.0;
  for (int k = threadIdx.x; k < items; k += kBlock) a = is_max ? nan_max(a, p[k]) : a + p[k];
  a = is_max ? block_nan_max(a, sh) : block_sum(a, sh);
  if (threadIdx.x == 0) out[(rows ? 16 : 0) + q] = a;
}

using CtxGetIdFn = int (*)(void* ctx, unsigned long long* id);   // cuCtxGetId

// Id of the current CUDA context through the driver entry point (cudart is linked statically,
// libcuda is not); 0 when there is none yet.
unsigned long long current_context_id() {
  static CtxGetIdFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      f = nullptr;
    }
    return reinterpret_cast<CtxGetIdFn>(f);
  }();
  if (!fn) throw Error(GPDHG_ERR_CUDA, "cuCtxGetId is not available from the driver");
  unsigned long long id = 0;
  return fn(nullptr, &id) == 0 ? id : 0ULL;
}

struct ScratchAddress {
  unsigned long long context = 0;
  double* ptr = nullptr;
};
std::mutex g_addr_mutex;
ScratchAddress g_addr[256];

// Device address of the scratch array in the current device's current context: looked up
// once per context, so a device whose context was reset gets the reloaded module's address.
double* scratch_address() {
  int dev = 0;
  CK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 256) throw Error(GPDHG_ERR_CUDA, "device ordinal out of range");
  std::lock_guard<std::mutex> lock(g_addr_mutex);
  ScratchAddress& a = g_addr[dev];
  const unsigned long long ctx = current_context_id();
  if (!a.ptr || ctx == 0 || ctx != a.context) {
    void* p = nullptr;
    CK(cudaGetSymbolAddress(&p, g_noalloc_scratch));   // makes the device's primary context current
    a.ptr = static_cast<double*>(p);
    a.context = current_context_id();
    if (a.context == 0) throw Error(GPDHG_ERR_CUDA, "no current CUDA context after the symbol lookup");
  }
  return a.ptr;
}

}  // namespace
}  // namespace gpdhg

namespace gpdhg {

void convergence_noalloc(int32_t n, int32_t m, int32_t neq, double obj_const, const double* l, const double* u,
                         const double* c, const double* b, const double* x, const double* y, const double* ax,
                         const double* aty, double eps_abs, double eps_rel, void* stream,
                         gpdhg_convergence_information* out) {
  if (!out || !l || !u || !c || !x || !aty) throw Error(GPDHG_ERR_INVALID_ARGUMENT, "required pointer is NULL");
  if (n <= 0 || m < 0 || neq < 0 || neq > m)
    throw Error(GPDHG_ERR_INVALID_ARGUMENT, "need n > 0 and 0 <= num_equalities <= m");
  if (m > 0 && (!b || !y || !ax)) throw Error(GPDHG_ERR_INVALID_ARGUMENT, "row-side pointer is NULL");
  if ((long long)n > kNoallocMaxLength || (long long)m > kNoallocMaxLength)
    throw Error(GPDHG_ERR_INVALID_ARGUMENT,
                "gpdhg_convergence_noalloc handles at most 16,777,216 variables and constraints");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // A capturing stream cannot take the synchronous read-back at the end; refuse before any
  // other CUDA call so that the caller's capture is left valid.
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  const cudaError_t ce = cudaStreamIsCapturing(s, &cap);
  if (ce != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
    if (ce != cudaSuccess) cudaGetLastError();
    throw Error(GPDHG_ERR_NOT_SUPPORTED,
                "gpdhg_convergence_noalloc is synchronous and cannot run on a stream that is being captured");
  }
  double* base = scratch_address();
  double* part_n = base;
  double* part_m = base + (size_t)kQn * kNoallocCtas;
  double* outs = base + (size_t)(kQn + kQm) * kNoallocCtas;
  const int item = noalloc_item(n, m);
  const int in = noalloc_items(n, item), im = noalloc_items(m, item);
  noalloc_reduce_kernel<<<in + im, kBlock, 0, s>>>(
      NoallocSide<ColumnStats>{ColumnStats{l, u, c, x, aty}, n, item, in, part_n},
      NoallocSide<RowStats>{RowStats{b, y, ax, neq}, m, item, im, part_m});
  CK_LAUNCH();
  noalloc_finalize_kernel<<<kQn + kQm, kBlock, 0, s>>>(part_n, in, part_m, im, outs);
  CK_LAUNCH();
  double h[32];
  CK(cudaMemcpyAsync(h, outs, sizeof(h), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  const double* A = h;
  const double* B = h + 16;
  // compute_convergence_information (src/iteration_stats_utils_gpu.jl:251-309) with the
  // CachedQuadraticProgramInfo norms of this problem (src/termination.jl:130-137)
  const double linf_c = A[kA_CMax], l2_c = std::sqrt(A[kA_CSq]);
  const double linf_b = B[kB_BMax], l2_b = std::sqrt(B[kB_BSq]);
  const double eps_ratio = eps_abs / eps_rel;
  gpdhg_convergence_information ci;
  std::memset(&ci, 0, sizeof(ci));
  ci.candidate_type = GPDHG_POINT_TYPE_CURRENT_ITERATE;
  ci.primal_objective = obj_const + A[kA_Cx];
  ci.l_inf_primal_residual = jmax_h(B[kB_CvMax], A[kA_LuMax]);
  ci.l2_primal_residual = std::sqrt(B[kB_CvSq] + A[kA_LuSq]);
  ci.relative_l_inf_primal_residual = ci.l_inf_primal_residual / (eps_ratio + linf_b);
  ci.relative_l2_primal_residual = ci.l2_primal_residual / (eps_ratio + l2_b);
  ci.l_inf_primal_variable = A[kA_XMax];
  ci.l2_primal_variable = std::sqrt(A[kA_XSq]);
  const double dual_res_inf = jmax_h(B[kB_DrMax], A[kA_RcvMax]);
  ci.dual_objective = B[kB_By] + obj_const + A[kA_Contrib];
  ci.l_inf_dual_residual = dual_res_inf;
  ci.l2_dual_residual = std::sqrt(B[kB_DrSq] + A[kA_RcvSq]);
  ci.relative_l_inf_dual_residual = ci.l_inf_dual_residual / (eps_ratio + linf_c);
  ci.relative_l2_dual_residual = ci.l2_dual_residual / (eps_ratio + l2_c);
  ci.l_inf_dual_variable = B[kB_YMax];
  ci.l2_dual_variable = std::sqrt(B[kB_YSq]);
  ci.corrected_dual_objective = dual_res_inf == 0.0 ? ci.dual_objective : -INFINITY;
  const double gap = std::fabs(ci.primal_objective - ci.dual_objective);
  ci.relative_optimality_gap = gap / (eps_ratio + std::fabs(ci.primal_objective) + std::fabs(ci.dual_objective));
  *out = ci;
}

}  // namespace gpdhg
