// batch_kernels.cuh — step and evaluation kernels for many LPs packed into one
// block-diagonal ("segmented") CSR; a lone LP is evaluated by the same kernels.
//
// Every row-block item of the packed A and A' belongs to exactly one instance, and an
// instance's items are built exactly as for a lone solve, so each instance sees the same
// per-CTA sums in the same order as when solved alone: results are bitwise identical
// alone and in a batch. Per-instance scalars live in a StepState array; the last CTA of
// an instance's dual pass (a per-instance arrival counter) takes that instance's
// accept/reject decision. A finished or retired instance's CTAs exit at once.
#pragma once

#include "eval_kernels.cuh"
#include "step_kernels.cuh"

namespace gpdhg {

// ---- segmented FP64 reductions --------------------------------------------------
// A segment item is a contiguous range of at most kSegLen elements of one instance, reduced by a
// cluster of two CTAs of 128 threads into its partials; then one CTA per instance and quantity reduces
// the instance's items in order. (One CTA per instance for all quantities took 15-34 us on
// 1,000-2,000 items, its loads of 25 quantities one after the other; one CTA each takes 6 us.) st
// NULL: every instance is active.
//
// Thread t of the 256 takes the elements t, t + 256, ... of its item; a quantity's 256 sums are added
// by one warp, lane l the entries l, l + 32, ... in order and then a shuffle tree (restart scores
// need this very order: they decide where the solve restarts). The passes are bound by the FP64 pipe
// (a third of their time is the least its arithmetic can take, a sixth the reduction) and by the 4,000
// cycles that one element takes a warp, so:
//   * a thread loads its next element's dozen operands before it works on one (128 registers);
//   * the item's sums are spread over both CTAs (stored into the reducing warp's CTA over
//     distributed shared memory), which on a small LP are two SMs' FP64 pipes instead of one, and on
//     a large one halve the granularity of the last wave;
//   * a warp's up to three sums share the instructions of their trees (6 additions, not 15).
// Times of the column and the row pass, with one CTA of 256 threads per item -> as it is: FP64 20,011 x
// 40,022 18.6 -> 13.4 and 13.6 -> 10.4 us; FP32 90,007 x 180,014 25 -> 20 and 30 -> 22 us;
// transportation 1M columns FP64 90 -> 66 us; power-law FP32 (2M, 1M) 177 -> 150 and 94 -> 87 us. Clusters of
// 4 CTAs of 64 take 67, 152 and 87 us on the last two, of 8 CTAs of 32 twice that; a warp per item 88,
// 203 and 125 us, and 60-72 us on the small ones.
constexpr int kPassCluster = 2;
template <int N, int O>
__device__ __forceinline__ void packed_tree(double* a) {   // N sums over 32 lanes; sum q ends at lane packed_lane
  constexpr int H = (N + 1) / 2;
  const bool up = (threadIdx.x & O) != 0;
#pragma unroll
  for (int w = 0; w < N - H; ++w) {
    const double give = of_bits(up ? bits_of(a[w]) : bits_of(a[w + H]));
    const double keep = of_bits(up ? bits_of(a[w + H]) : bits_of(a[w]));
    a[w] = keep + __shfl_xor_sync(0xffffffffu, give, O);
  }
  if (N - H < H) a[H - 1] += __shfl_xor_sync(0xffffffffu, a[H - 1], O);
  if constexpr (O > 1) packed_tree<H, O / 2>(a);
}
__host__ __device__ constexpr int packed_lane(int n, int q) {
  int lane = 0;
  for (int o = 16; o > 0; o >>= 1) {
    const int h = (n + 1) / 2;
    if (q >= h) {
      lane |= o;
      q -= h;
    }
    n = h;
  }
  return lane;
}
__host__ __device__ constexpr int count_bits(unsigned m) { return m ? (int)(m & 1u) + count_bits(m >> 1) : 0; }
// The quantities in the order of their reduction, sums before maxima: warp g of the cluster's eight
// takes the slots g, g + 8, ...
template <int Q, unsigned MAXMASK>
struct PassSlots {
  static constexpr int kWarps = kBlock / 32;
  static constexpr int kSums = Q - count_bits(MAXMASK);
  static constexpr int kRounds = (Q + kWarps - 1) / kWarps, kSumRounds = (kSums + kWarps - 1) / kWarps;
  __host__ __device__ static constexpr int slot(int q) {
    const int maxima = count_bits(MAXMASK & ((1u << q) - 1u));
    return MAXMASK >> q & 1u ? kSums + maxima : q - maxima;
  }
  __device__ static __forceinline__ int quantity(int s) {
    int q = 0;
#pragma unroll
    for (int k = 0; k < Q; ++k)
      if (slot(k) == s) q = k;
    return q;
  }
};
// F: Params(st, inst), In, load(params, i, in), apply(params, i, in, acc).
template <int Q, unsigned MAXMASK, class F>
__global__ void __launch_bounds__(kBlock / kPassCluster, 2 * kPassCluster)
    seg_reduce_kernel(const SegItem* items, const StepState* st, F f, double* partials, int num_items) {
  using S = PassSlots<Q, MAXMASK>;
  constexpr int W = S::kWarps, V = W / kPassCluster;   // warps of the cluster and of a CTA
  __shared__ double sh[V * S::kRounds][kBlock];
  const int rank = blockIdx.x % kPassCluster, item = blockIdx.x / kPassCluster;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = rank * (kBlock / kPassCluster) + (int)threadIdx.x;
  const SegItem it = items[item];
  if (st && !st[it.inst].eval_active) return;   // the whole cluster
  cluster_arrive();   // waited for before the first store into the other CTA
  const typename F::Params p(st, it.inst);
  double acc[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) acc[q] = 0.0;
  typename F::In in, next;
  int i = it.begin + t;
  if (i < it.end) f.load(p, i, in);
#pragma unroll 1
  for (; i < it.end; i += kBlock) {
    if (i + kBlock < it.end) f.load(p, i + kBlock, next);
    f.apply(p, i, in, acc);
    in = next;
  }
  cluster_wait();
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    constexpr S slots{};
    const int s = slots.slot(q), owner = s % W;
    remote_store(remote_address(&sh[owner % V + V * (s / W)][t], owner / V), acc[q]);
  }
  cluster_barrier();
  const int g = rank * V + warp;
  double sum[S::kSumRounds];
#pragma unroll
  for (int j = 0; j < S::kRounds; ++j) {
    const int s = g + W * j;
    if (j < S::kSumRounds) sum[j] = 0.0;
    if (s >= Q) break;
    const double* c = sh[warp + V * j] + lane;
    double v = c[0];
    if (s < S::kSums) {
#pragma unroll
      for (int w = 1; w < W; ++w) v += c[w * 32];
      if (j < S::kSumRounds) sum[j] = v;
    } else {
#pragma unroll
      for (int w = 1; w < W; ++w) v = nan_max(v, c[w * 32]);
      v = warp_nan_max(v);
      if (lane == 0) partials[(size_t)S::quantity(s) * num_items + item] = v;
    }
  }
  __syncwarp();
  packed_tree<S::kSumRounds, 16>(sum);
#pragma unroll
  for (int j = 0; j < S::kSumRounds; ++j) {
    const int s = g + W * j;
    if (s < S::kSums && lane == packed_lane(S::kSumRounds, j)) partials[(size_t)S::quantity(s) * num_items + item] = sum[0];
  }
}
template <int Q, unsigned MAXMASK, class F>
inline void launch_reduce(const SegItem* items, const StepState* st, const F& f, double* partials, int num_items,
                          cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(kPassCluster * num_items));
  cfg.blockDim = dim3(kBlock / kPassCluster);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kPassCluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  CK(cudaLaunchKernelEx(&cfg, seg_reduce_kernel<Q, MAXMASK, F>, items, st, f, partials, num_items));
}

// Where one side's partials lie and where its results go (quantity q of instance k at
// out[k * kEvalStride + q]).
struct SegSide {
  const int32_t* inst_item_begin;
  const double* partials;
  double* out;
  int num_items;
  int quantities;
  unsigned maxmask;
};
constexpr int kEvalStride = 64;   // results per instance: rows' at 0, columns' at kEvalOutN
constexpr int kEvalOutN = 32;
constexpr int kEvalSpan = 63;     // behind steps: seconds from their last decision to the end of the evaluation
static_assert(kPassMQ <= kEvalOutN && kEvalOutN + kPassNQ <= kEvalSpan && kEvalSpan < kEvalStride, "results do not overlap");
// Grid (instances, quantities of both sides): a grid's first dimension takes any number of
// instances, the others 65,535 at most. The results go straight into the host's pinned memory,
// and so does the state if mirror is given (the first CTA copies it, whether evaluated or not): behind
// the kernel, a copy node cost 4-11 us.
static __global__ void __launch_bounds__(kBlock) seg_finalize_kernel(SegSide a, SegSide b, const StepState* st,
                                                                        StepState* mirror) {
  __shared__ double sh[kBlock], res[1];
  const int inst = blockIdx.x;
  if (mirror && blockIdx.y == 0 && threadIdx.x < kStateWords)
    reinterpret_cast<long long*>(mirror + inst)[threadIdx.x] = reinterpret_cast<const long long*>(st + inst)[threadIdx.x];
  if (st && !st[inst].eval_active) return;
  const bool second = (int)blockIdx.y >= a.quantities;
  const SegSide& s = second ? b : a;
  const int q = (int)blockIdx.y - (second ? a.quantities : 0);
  const bool is_max = (s.maxmask >> q) & 1u;
  const double* p = s.partials + (size_t)q * s.num_items;
  const int k1 = s.inst_item_begin[inst + 1];
  double acc[1] = {0.0};
  for (int k = s.inst_item_begin[inst] + (int)threadIdx.x; k < k1; k += kBlock)
    acc[0] = is_max ? nan_max(acc[0], p[k]) : acc[0] + p[k];
  const double r = is_max ? block_reduce_q<1, 1u>(acc, sh, res) : block_reduce_q<1, 0u>(acc, sh, res);
  if (threadIdx.x == 0) {
    s.out[(size_t)inst * kEvalStride + q] = r;
    if (mirror && blockIdx.y == 0)
      a.out[(size_t)inst * kEvalStride + kEvalSpan] =
          1e-9 * (double)(long long)(global_ns() - st[inst].launch_start_ns - st[inst].launch_ns);
  }
}

// ---- state ------------------------------------------------------------------------
// Copies the instances' states between the device and the host's pinned mirror (one CTA each): a
// kernel starts and ends some 3 us closer to its neighbours than a copy does.
static __global__ void copy_state_kernel(const StepState* src, StepState* dst) {
  if (threadIdx.x < kStateWords)
    reinterpret_cast<long long*>(dst + blockIdx.x)[threadIdx.x] =
        reinterpret_cast<const volatile long long*>(src + blockIdx.x)[threadIdx.x];
  __syncthreads();
  if (threadIdx.x == 0) dst[blockIdx.x].launch_start_ns = global_ns();
}
inline void copy_state(const StepState* src, StepState* dst, int count, cudaStream_t s) {
  copy_state_kernel<<<count, (kStateWords + 31) / 32 * 32, 0, s>>>(src, dst);
  CK_LAUNCH();
}

// ---- restart ----------------------------------------------------------------------
// Restart actions (src/saddle_point_gpu.jl:575-614) of the instances whose StepState::restart is set
// (kRestartToAverage: the average becomes the current point): the averaging sums are cleared and
// the restart point is stored. Elements [0, n) are columns, the rest rows; inst_of NULL: one
// instance. (As up to eleven copies and fills, a restart was mostly launches.)
enum RestartMode : int { kNoRestart = 0, kRestartFromCurrent = 1, kRestartToAverage = 2 };
template <class T>
struct RestartArgs {
  const StepState* st;
  const int32_t* col_inst;
  const int32_t* row_inst;
  int n, m;
  const T *c, *ax, *agrad, *ay, *akx;
  T *x, *kty, *grad, *sx, *rx, *rgrad;
  T *y0, *y1, *kx0, *kx1, *sy, *skx, *ry, *rkx;
};
template <class T>
__global__ void __launch_bounds__(kBlock) restart_kernel(RestartArgs<T> a) {
  const int stride = gridDim.x * blockDim.x;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < a.n; j += stride) {
    const int mode = a.st[a.col_inst ? a.col_inst[j] : 0].restart;
    if (mode == kNoRestart) continue;
    T x = a.x[j], g = a.grad[j];
    if (mode == kRestartToAverage) {
      x = a.ax[j];
      g = a.agrad[j];
      a.x[j] = x;
      a.kty[j] = a.c[j] - g;
      a.grad[j] = g;
    }
    a.sx[j] = T(0);
    a.rx[j] = x;
    a.rgrad[j] = g;
  }
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.m; i += stride) {
    const StepState& q = a.st[a.row_inst ? a.row_inst[i] : 0];
    if (q.restart == kNoRestart) continue;
    T* yc = q.parity ? a.y1 : a.y0;
    T* kc = q.parity ? a.kx1 : a.kx0;
    T y = yc[i], k = kc[i];
    if (q.restart == kRestartToAverage) {
      y = a.ay[i];
      k = a.akx[i];
      yc[i] = y;
      kc[i] = k;
    }
    a.sy[i] = T(0);
    a.skx[i] = T(0);
    a.ry[i] = y;
    a.rkx[i] = k;
  }
}

}  // namespace gpdhg
