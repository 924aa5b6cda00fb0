// spmv.cuh — the CSR row-block SpMV shared by every step kernel.
//
// An item (one CTA) covers rows [row_begin, row_end); its `mode` picks the schedule:
//   kItemStaged  short rows whose nonzeros fit the CTA's stage (kStage = 256 x 8), at most
//                one row per group of `group` lanes (1..32) — steps 1-3 below;
//   kItemWarps   up to 8 rows of >= 64 nonzeros, one warp per row: register accumulation
//                (one FMA per nonzero, four independent loads per lane in flight);
//   kItemLong    one row of more than 256 nonzeros, streamed by the whole CTA;
//   kItemLongWarps  up to 8 such rows of at most kStage nonzeros, one per warp, each summed in
//                the order of kItemLong (long_row_dot).
// Staged items:
//   1. the row's own epilogue loads (`pre`) are issued first;
//   2. every thread loads U (col, val) pairs of the item — fully unrolled, independent,
//      coalesced — then issues its U gathers, and stages the products in shared memory
//      (FP64 stages value and gathered entry apart, so the row sum is one FMA per nonzero on
//      GB300's scarce FP64 pipe): U loads in flight per thread instead of one dependent load
//      chain per nonzero;
//   3. after one barrier each group sums its row from shared memory in a fixed order and
//      its lane 0 runs the epilogue (`post`).
// Matrix streams use evict-first loads so the gathered vector stays in L2. The reduction
// order is fixed by the schedule, so results are deterministic.
#pragma once

#include "common.cuh"

namespace gpdhg {


template <class T>
__device__ __forceinline__ T group_sum(T v, int g) {
  for (int o = g >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, g);
  return v;
}

// Row r of M times xg by the 32 lanes of a warp, four independent loads per lane in flight.
template <class T>
__device__ __forceinline__ T warp_row_dot(const CsrView<T>& M, const T* __restrict__ xg, int r, int lane) {
  const int s = M.row_ptr[r], e = M.row_ptr[r + 1];
  T a0 = T(0), a1 = T(0), a2 = T(0), a3 = T(0);
  int k = s + lane;
  for (; k + 96 < e; k += 128) {
    const int c0 = lds(M.col + k), c1 = lds(M.col + k + 32), c2 = lds(M.col + k + 64), c3 = lds(M.col + k + 96);
    const T v0 = lds(M.val + k), v1 = lds(M.val + k + 32), v2 = lds(M.val + k + 64), v3 = lds(M.val + k + 96);
    a0 += v0 * xg[c0];
    a1 += v1 * xg[c1];
    a2 += v2 * xg[c2];
    a3 += v3 * xg[c3];
  }
  for (; k < e; k += 32) a0 += lds(M.val + k) * xg[lds(M.col + k)];
  return warp_sum((a0 + a1) + (a2 + a3));
}

// Row r of M (at most kStage nonzeros) times xg by one warp, in the order of a whole CTA's sum
// (kItemLong): virtual warp w takes the nonzeros 256 q + 32 w + lane in order of q, the warps' sums
// are shuffle trees, added in order of w. The eight trees share their levels' instructions (lanes
// keep half of the quantities at each), 9 additions instead of 40 or, by a CTA, 8 x (8 + 7 + 5):
// on the power-law LPs, whose rows of 257 to 2,048 nonzeros hold most of the matrix, those kept the
// FP64 pipe 74% busy, and a CTA per row is short of loads in flight. A'y of the 500k x 1M LP in FP64
// 209 -> 88 us, of the 1M x 2M LP in FP32 173 -> 101 us.
template <class T>
__device__ __forceinline__ T long_row_dot(const CsrView<T>& M, const T* __restrict__ xg, int r, int lane) {
  constexpr int W = kBlock / 32;
  static_assert(W == 8, "three levels of pairs");
  const unsigned full = 0xffffffffu;
  const int s = M.row_ptr[r], e = M.row_ptr[r + 1];
  T a[W];
#pragma unroll
  for (int w = 0; w < W; ++w) a[w] = T(0);
  for (int base = s; base < e; base += kBlock) {
    int c[W];
    T v[W];
#pragma unroll
    for (int w = 0; w < W; ++w) {
      const int k = base + 32 * w + lane;
      c[w] = k < e ? lds(M.col + k) : -1;
      v[w] = k < e ? lds(M.val + k) : T(0);
    }
    T x[W];
#pragma unroll
    for (int w = 0; w < W; ++w) x[w] = c[w] >= 0 ? xg[c[w]] : T(0);
#pragma unroll
    for (int w = 0; w < W; ++w) {
      if (base + 32 * w >= e) break;   // uniform over the warp
      a[w] = base == s ? fma(v[w], x[w], T(0)) : a[w] + fma(v[w], x[w], T(0));
    }
  }
#pragma unroll
  for (int h = W / 2, o = 16; h > 0; h >>= 1, o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int w = 0; w < h; ++w) {
      const T give = up ? a[w] : a[w + h], keep = up ? a[w + h] : a[w];
      a[w] = keep + __shfl_xor_sync(full, give, o);
    }
  }
  a[0] += __shfl_xor_sync(full, a[0], 2);
  a[0] += __shfl_xor_sync(full, a[0], 1);
  T sum = T(0);
#pragma unroll
  for (int w = 0; w < W; ++w) sum += __shfl_sync(full, a[0], 4 * w);   // lanes 4 w.. hold warp w's
  return sum;
}

// Runs the item's rows. Every thread of the CTA must call it. `stage` holds kStage T, and
// so does `stage2` when T is double (unused otherwise).
template <class T, class Pre, class Post>
__device__ __forceinline__ void spmv_item(const CsrView<T>& M, const T* __restrict__ xg, int item, T* stage,
                                          T* stage2, T* wsum, Pre&& pre, Post&& post) {
  constexpr int U = kStageDepth;
  const RowItem it = M.items[item];
  const int tid = threadIdx.x;
  if (it.mode == kItemLongWarps) {
    const int lane = tid & 31, r = it.row_begin + (tid >> 5);
    if (r < it.row_end) {
      decltype(pre(r)) p{};
      if (lane == 0) p = pre(r);
      const T sum = long_row_dot(M, xg, r, lane);
      if (lane == 0) post(r, sum, p);
    }
    return;
  }
  if (it.mode == kItemWarps) {
    const int lane = tid & 31;
    for (int base = it.row_begin; base < it.row_end; base += kBlock / 32) {
      const int r = base + (tid >> 5);
      if (r < it.row_end) {   // whole warps take this branch together
        decltype(pre(r)) p{};
        if (lane == 0) p = pre(r);
        const T sum = warp_row_dot(M, xg, r, lane);
        if (lane == 0) post(r, sum, p);
      }
    }
    return;
  }
  if (it.mode == kItemLong) {
    // one long row streamed by the whole CTA, U independent loads per thread per round
    const int r = it.row_begin;
    decltype(pre(r)) p{};
    if (tid == 0) p = pre(r);
    const int s = M.row_ptr[r], e = M.row_ptr[r + 1];
    T acc[U];
#pragma unroll
    for (int q = 0; q < U; ++q) acc[q] = T(0);
    for (int base = s; base < e; base += kBlock * U) {
      int c[U];
      T v[U];
#pragma unroll
      for (int q = 0; q < U; ++q) {
        const int k = base + q * kBlock + tid;
        c[q] = k < e ? lds(M.col + k) : 0;
        v[q] = k < e ? lds(M.val + k) : T(0);
      }
#pragma unroll
      for (int q = 0; q < U; ++q)
        if (base + q * kBlock < e) acc[q] += v[q] * xg[c[q]];   // the same for the whole CTA
    }
#pragma unroll
    for (int q = 1; q < U; ++q)
      if (s + q * kBlock < e) acc[0] += acc[q];
    const T a = warp_sum(acc[0]);
    __syncthreads();
    if ((tid & 31) == 0) wsum[tid >> 5] = a;
    __syncthreads();
    if (tid == 0) {
      T sum = T(0);
      for (int w = 0; w < kBlock / 32; ++w) sum += wsum[w];
      post(r, sum, p);
    }
    return;
  }
  const int g = it.group;
  const int lane = tid & (g - 1);
  const int r = it.row_begin + tid / g;
  const bool owner = r < it.row_end && lane == 0;
  decltype(pre(r)) p{};
  if (owner) p = pre(r);
  const int s0 = M.row_ptr[it.row_begin];
  const int cnt = M.row_ptr[it.row_end] - s0;
  {
    int c[U];
    T v[U];
#pragma unroll
    for (int q = 0; q < U; ++q) {
      const int k = q * kBlock + tid;
      c[q] = k < cnt ? lds(M.col + s0 + k) : 0;
      v[q] = k < cnt ? lds(M.val + s0 + k) : T(0);
    }
#pragma unroll
    for (int q = 0; q < U; ++q) {
      const int k = q * kBlock + tid;
      if (k < cnt) {
        if constexpr (sizeof(T) == 8) {
          stage[k] = v[q];
          stage2[k] = xg[c[q]];
        } else {
          stage[k] = v[q] * xg[c[q]];
        }
      }
    }
  }
  __syncthreads();
  T sum = T(0);
  if (r < it.row_end) {
    const int a = M.row_ptr[r] - s0, b = M.row_ptr[r + 1] - s0;
    if constexpr (sizeof(T) == 8) {
      for (int k = a + lane; k < b; k += g) sum += stage[k] * stage2[k];
    } else {
      for (int k = a + lane; k < b; k += g) sum += stage[k];
    }
  }
  sum = group_sum(sum, g);
  if (owner) post(r, sum, p);
}

// y = M x over the row-block items of M. With st non-NULL only the items of instances under evaluation
// (StepState::eval_active) run; row_inst gives the instance of an item's first row (the packed matrix
// of a batch; an item never spans two instances), NULL: one instance.
struct NoPre {};
template <class T>
__global__ void __launch_bounds__(kBlock) spmv_kernel(CsrView<T> M, const T* __restrict__ x, T* y,
                                                      const int32_t* __restrict__ row_inst, const StepState* st) {
  __shared__ T stage[kStage];
  __shared__ T stage2[sizeof(T) == 8 ? kStage : 1];
  __shared__ T wsum[kBlock / 32];
  if ((int)blockIdx.x >= M.num_items) return;
  if (st && !st[row_inst ? row_inst[M.items[blockIdx.x].row_begin] : 0].eval_active) return;
  auto pre = [](int) { return NoPre{}; };
  auto post = [&](int i, T s, const NoPre&) { y[i] = s; };
  spmv_item(M, x, blockIdx.x, stage, stage2, wsum, pre, post);
}

}  // namespace gpdhg
