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
// A segment item is a contiguous element range of one instance, reduced by one CTA into its
// partials; then one CTA per instance and quantity reduces the instance's items in order. (One
// CTA per instance for all quantities took 15-34 us on 1,000-2,000 items, its loads of 25
// quantities one after the other; one CTA each takes 6 us.) st NULL: every instance is active.
// The passes are bound by the FP64 pipe (62-81% busy) and the latency of a thread's dozen loads, so
// 3 CTAs per SM (80 registers, some spilled in the column pass; 2 CTAs: 110 and 212 us for the two
// column passes below). Cold-cache times, FP64 arithmetic plainly written -> as it is: column pass
// of the transportation LP (1M columns, FP64) 194 -> 101 us, of the power-law LP (2M, FP32) 428 ->
// 189 us, its row pass (1M rows) 127 -> 93 us. (Longer segments, in one wave of CTAs, take 70, 138
// and 70 us, but add the restart scores in another order.)
template <int Q, unsigned MAXMASK, class F>
__global__ void __launch_bounds__(kBlock, 3) seg_reduce_kernel(const SegItem* items, const StepState* st, F f,
                                                            double* partials, int num_items) {
  __shared__ double sh[(Q < kRedChunk ? Q : kRedChunk) * kBlock];
  __shared__ double res[Q];
  const SegItem it = items[blockIdx.x];
  if (st && !st[it.inst].eval_active) return;
  const typename F::Params p(st, it.inst);
  double acc[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) acc[q] = 0.0;
  for (int i = it.begin + threadIdx.x; i < it.end; i += kBlock) f(p, i, acc);
  const double r = block_reduce_q<Q, MAXMASK>(acc, sh, res);
  if ((int)threadIdx.x < Q) partials[(size_t)threadIdx.x * num_items + blockIdx.x] = r;
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
// Grid (quantities of both sides, instances).
static __global__ void __launch_bounds__(kBlock) seg_finalize_kernel(SegSide a, SegSide b, const StepState* st) {
  __shared__ double sh[kBlock], res[1];
  const int inst = blockIdx.y;
  if (st && !st[inst].eval_active) return;
  const bool second = (int)blockIdx.x >= a.quantities;
  const SegSide& s = second ? b : a;
  const int q = (int)blockIdx.x - (second ? a.quantities : 0);
  const bool is_max = (s.maxmask >> q) & 1u;
  const double* p = s.partials + (size_t)q * s.num_items;
  const int k1 = s.inst_item_begin[inst + 1];
  double acc[1] = {0.0};
  for (int k = s.inst_item_begin[inst] + (int)threadIdx.x; k < k1; k += kBlock)
    acc[0] = is_max ? nan_max(acc[0], p[k]) : acc[0] + p[k];
  const double r = is_max ? block_reduce_q<1, 1u>(acc, sh, res) : block_reduce_q<1, 0u>(acc, sh, res);
  if (threadIdx.x == 0) s.out[(size_t)inst * kEvalStride + q] = r;
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
