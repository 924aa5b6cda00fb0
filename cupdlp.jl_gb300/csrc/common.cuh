// common.cuh — shared device/host helpers of libgpdhg (sm_103a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <stdexcept>
#include <string>

#include "gpdhg.h"

namespace gpdhg {

// Phase timing of problem creation and solve set-up, printed to stderr when the environment
// variable GPDHG_TRACE is set (a diagnostic; nothing else reads it).
struct PhaseTrace {
  bool on;
  std::chrono::steady_clock::time_point t;
  PhaseTrace() : on(std::getenv("GPDHG_TRACE") != nullptr), t(std::chrono::steady_clock::now()) {}
  void mark(const char* what) {
    if (!on) return;
    const auto now = std::chrono::steady_clock::now();
    std::fprintf(stderr, "gpdhg trace: %-28s %8.2f ms\n", what,
                 std::chrono::duration<double, std::milli>(now - t).count());
    t = now;
  }
};

// A failure that maps onto one gpdhg_status at the ABI boundary.
struct Error : std::runtime_error {
  gpdhg_status status;
  Error(gpdhg_status s, const std::string& m) : std::runtime_error(m), status(s) {}
};

inline void cuda_check(cudaError_t e, const char* what, const char* file, int line) {
  if (e != cudaSuccess) {
    cudaGetLastError();   // reported here: the launch check of a later call must not find it again
    gpdhg_status s = (e == cudaErrorMemoryAllocation) ? GPDHG_ERR_OUT_OF_MEMORY : GPDHG_ERR_CUDA;
    throw Error(s, std::string(what) + ": " + cudaGetErrorString(e) + " (" + file + ":" + std::to_string(line) + ")");
  }
}
#define CK(call) ::gpdhg::cuda_check((call), #call, __FILE__, __LINE__)
#define CK_LAUNCH() ::gpdhg::cuda_check(cudaGetLastError(), "kernel launch", __FILE__, __LINE__)

// Records what is launched on a stream (and on `side`, a stream for work beside it, which joins it
// through the events) into a graph. Thrown out of, it takes the stream out of capture.
class GraphCapture {
 public:
  cudaStream_t side = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  explicit GraphCapture(cudaStream_t stream, bool with_side = true) : stream_(stream) {
    try {
      if (with_side) {
        CK(cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking));
        CK(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming));
        CK(cudaEventCreateWithFlags(&join, cudaEventDisableTiming));
      }
      CK(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal));
    } catch (...) {
      release();
      throw;
    }
    open_ = true;
  }
  GraphCapture(const GraphCapture&) = delete;
  GraphCapture& operator=(const GraphCapture&) = delete;
  ~GraphCapture() {
    if (open_) {
      cudaGraph_t g = nullptr;
      if (cudaStreamEndCapture(stream_, &g) == cudaSuccess && g) cudaGraphDestroy(g);
      cudaGetLastError();
    }
    release();
  }
  cudaGraphExec_t finish() {
    cudaGraph_t g = nullptr;
    open_ = false;   // whether it succeeds or not
    CK(cudaStreamEndCapture(stream_, &g));
    cudaGraphExec_t ex = nullptr;
    const cudaError_t e = cudaGraphInstantiate(&ex, g, 0);
    cudaGraphDestroy(g);
    cuda_check(e, "cudaGraphInstantiate", __FILE__, __LINE__);
    return ex;
  }

 private:
  cudaStream_t stream_;
  bool open_ = false;
  void release() {
    if (join) cudaEventDestroy(join);
    if (fork) cudaEventDestroy(fork);
    if (side) cudaStreamDestroy(side);
  }
};

constexpr int kBlock = 256;          // threads per CTA of every row-block kernel
constexpr int kStageDepth = 8;                // independent (col, val) loads per thread and item
constexpr int kStage = kBlock * kStageDepth;  // nonzeros staged per item (2048)

// One CTA's share of a CSR matrix: rows [row_begin, row_end) and the schedule used for
// them (see spmv.cuh): staged short rows reduced by groups of `group` lanes, warp-per-row
// register accumulation, one long row streamed by the whole CTA, or long rows by a warp each.
enum ItemMode : int32_t { kItemStaged = 0, kItemWarps = 1, kItemLong = 2, kItemLongWarps = 3 };
struct RowItem {
  int32_t row_begin;
  int32_t row_end;
  int32_t group;
  int32_t mode;
  int32_t nnz_begin;   // row_ptr[row_begin]
  int32_t nnz_count;   // row_ptr[row_end] - row_ptr[row_begin]
};

// A contiguous element range [begin, end) of one instance, reduced by one CTA of the
// segmented FP64 reductions (evaluation statistics, restart scores).
struct SegItem {
  int32_t begin;
  int32_t end;
  int32_t inst;
};

// Device view of a CSR matrix with its row-block schedule.
template <class T>
struct CsrView {
  int32_t nrows;
  int32_t ncols;
  const int32_t* row_ptr;
  const int32_t* col;
  const T* val;
  const RowItem* items;
  int32_t num_items;
};

// Scalar state of the step loop, resident on the device and updated by the last CTA
// of the dual kernel after every step attempt (the host mirrors it between chunks).
struct StepState {
  double tau;              // step size of the next attempt (take_step!'s local step_size)
  double omega;            // primal weight
  double iter_start_tau;   // solver_state.step_size at entry of take_step!: the averaging weight
  double commit_weight;    // averaging weight of the accepted step awaiting its commit
  double kkt_passes;       // cumulative_kkt_passes
  double sum_w_primal;     // sum_primal_solution_weights
  double sum_w_dual;       // sum_dual_solution_weights
  double reduction_exponent;
  double growth_exponent;
  double last_limit;       // diagnostics: last step-size limit
  long long total_iters;   // total_number_iterations (attempts)
  long long count_primal;  // sum_primal_solutions_count
  long long count_dual;    // sum_dual_solutions_count
  long long accepted;
  long long rejected;
  int parity;              // which y / K x buffer is current
  int pending_commit;      // an accepted step whose vector updates are not applied yet
  int done;                // the current chunk is finished
  int numerical_error;
  int accepted_in_chunk;
  int target_in_chunk;
  int attempts_in_chunk;
  int max_attempts_in_chunk;
  unsigned int arrive;     // CTAs of the dual kernel finished in this attempt
  int constant_step;       // ConstantStepsizeParams: every attempt is accepted
  long long primal_spmv;   // attempts whose primal kernel also ran A'y (a commit)
  const double* pow_table; // [1-(k+1)^-r, 1+(k+1)^-g] for k < pow_table_len (device)
  long long pow_table_len;
  double half_over_omega;  // 0.5 / omega, set by the host with omega
  double tto;              // tau / omega, kept by whoever changes tau or omega (the host, the step decision)
  // for an evaluation, set by the host or by the decision that ends a chunk: 1 / sum_w_primal and
  // 1 / sum_w_dual, whether the instance is evaluated, whether it has no average yet (the current
  // point stands in), and (by the host) whether the last restart point's KKT ingredients are needed
  double rcp_w_primal, rcp_w_dual;
  int eval_active, eval_current, eval_restart;
  int restart;             // RestartMode of the restart kernel that follows
  int launch_attempts;     // attempts_in_chunk after which the launch under way has run all of its own
  // when the launch's state arrived, and from then to the decision of its last attempt that did work
  unsigned long long launch_start_ns, launch_ns;
};

// ----------------------------------------------------------------------------------
// Deterministic block reductions (fixed shuffle tree, fixed warp order).
// ----------------------------------------------------------------------------------
template <class T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
// Barrier of a thread-block cluster, for every thread of every CTA: what was written before is
// visible to all after. The aligned forms want the whole warp at the instruction, and the code
// before may have left it diverged (a lane's own branch, the epilogue of the lanes that own rows):
// each brings the warp together first.
__device__ __forceinline__ void cluster_arrive() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// A barrier of the CTA's first `threads` threads (whole warps) under its own number, apart from __syncthreads.
template <int kNumber, int kThreads>
__device__ __forceinline__ void named_barrier() {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"n"(kNumber), "n"(kThreads) : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
  cluster_arrive();
  cluster_wait();
}
// The shared-memory address of p (this CTA's) in CTA `rank` of the cluster, and a store there.
__device__ __forceinline__ unsigned remote_address(const void* p, unsigned rank) {
  unsigned a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void remote_store(unsigned a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void remote_store(unsigned a, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}

// Sum over the CTA; the result is valid in thread 0. `sh` holds >= 32 entries.
template <class T>
__device__ __forceinline__ T block_sum(T v, T* sh) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  T r = T(0);
  if (wid == 0) {
    r = (lane < (int)(blockDim.x >> 5)) ? sh[lane] : T(0);
    r = warp_sum(r);
  }
  return r;
}

// Julia's max/min (used by the reference's kernels) propagate NaN.
__device__ __forceinline__ double jmax(double a, double b) { return (a != a || b != b) ? a + b : (a > b ? a : b); }
__device__ __forceinline__ double jmin(double a, double b) { return (a != a || b != b) ? a + b : (a < b ? a : b); }
__device__ __forceinline__ float jmax(float a, float b) { return (a != a || b != b) ? a + b : (a > b ? a : b); }
__device__ __forceinline__ float jmin(float a, float b) { return (a != a || b != b) ? a + b : (a < b ? a : b); }

inline int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }

// Streaming accesses (read or written once per pass): evict-first in L1 and L2, so the
// vectors gathered by the next kernel stay resident in L2.
template <class T>
__device__ __forceinline__ T lds(const T* p) { return __ldcs(p); }
template <class T>
__device__ __forceinline__ void sts(T* p, T v) { __stcs(p, v); }

// max / min of doubles on the integer pipe (GB300's FP64 pipe is the scarce resource):
// for non-NaN values the sign-magnitude bit pattern maps to an order-preserving int64 key.
__device__ __forceinline__ long long order_key(double v) {
  const long long b = __double_as_longlong(v);
  return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}
__device__ __forceinline__ double imax(double a, double b) { return order_key(a) < order_key(b) ? b : a; }
__device__ __forceinline__ double imin(double a, double b) { return order_key(b) < order_key(a) ? b : a; }
__device__ __forceinline__ float imax(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ float imin(float a, float b) { return fminf(a, b); }

}  // namespace gpdhg
