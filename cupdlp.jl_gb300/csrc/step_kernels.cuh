// step_kernels.cuh — the two fused kernels of one PDHG step attempt.
//
// Reference step (src/primal_dual_hybrid_gradient_gpu.jl:177-413) per attempt:
//   x^ = proj_[l,u](x - (tau/omega)(c - K'y));  dx = x^ - x            (:177-197)
//   K dx                                                               (:225, cuSPARSE)
//   y^ = y + omega tau (b - 2 K dx - K x);  y^[ineq] >= 0;  dy = y^ - y (:232-260)
//   |dy . K dx|, ||dx||, ||dy||                                        (:324-338)
//   accept if tau <= movement / interaction; then x += dx, Kx += K dx, y += dy,
//   K'y = A' y and the four weighted sums (:297-319, src/saddle_point_gpu.jl:131-221);
//   tau <- min((1-(k+1)^-0.3) limit, (1+(k+1)^-0.6) tau)                (:405-409)
//
// Here one attempt is two kernels over warp tiles (tiles.h, tile_spmv.cuh) and no host
// round trip:
//   primal_step_kernel: [if the previous attempt was accepted] K'y = A' y (tiles of A'),
//       x += dx, and the x weighted sum; then the next dx, and per-CTA ||dx||^2. (The
//       average's K'y is formed at evaluation time as A' y-bar, not summed here.)
//   dual_step_kernel:   [if the previous attempt was accepted] the y / Kx weighted sums;
//       then K dx (tiles of A), the projected dual candidate, Kx + K dx into the other half
//       of the double-buffered y / Kx, per-CTA interaction and ||dy||^2 partials; the last
//       CTA of an instance to finish reduces that instance's partials of both kernels in a
//       fixed order and takes the accept/reject and step-size decision, flipping the buffer
//       parity on accept.
//       (A separate decision kernel measured slower: one more kernel boundary per attempt
//       costs more than this CTA's serial tail.)
// Every CTA belongs to one instance; each warp owns whole tiles (row sums in registers,
// the fused epilogue on its rows), so no barrier sits between a warp's loads and its
// arithmetic, and latency is hidden by the many warps resident per SM. A split row's
// contribution to the partials is written to a per-split-row slot by the one warp that
// completes it, so all reductions keep a fixed order.
// So an accepted step costs exactly one pass over A and one over A'; a rejected attempt
// costs one pass over A plus a streaming pass over the n-vectors.
//
// `direct` mode (the FP32 bulk phase): the primal kernel stores the candidate x^ itself
// (in the dx buffer) and the dual kernel forms K x^ = A x^ from scratch, K dx = K x^ - K x,
// and stores K x^ as the next K x. The reference's incremental K x += K dx (:304) is kept
// in FP64 for parity; in FP32 it drifts by ~1e-6 relative, which this mode removes.
#pragma once

#include "common.cuh"
#include "tile_spmv.cuh"
#include "tiles.h"

namespace gpdhg {

enum StepMode : int { kStepNormal = 0, kStepCommitOnly = 1 };

// Programmatic dependent launch (sm_90+): the step kernels are launched with the
// programmatic-serialization attribute, so a kernel's CTAs may start while the previous
// kernel finishes. Everything before pdl_wait() must read only constant data (the tile
// plan); pdl_wait() returns once the previous kernel has completed and its writes are
// visible (immediately when it was launched without the attribute).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" :::); }

template <class T>
struct PrimalArgs {
  CsrView<T> At;         // CSR of A' (rows = variables)
  TileView<T> plan;      // tiles of A'
  const T* c;
  const T* l;
  const T* u;
  T* x;
  T* dx;                 // dx, or x^ in direct mode
  T* kty;
  T* sx;
  const T* y0;
  const T* y1;
  StepState* st;         // one per instance
  double* part_p;        // ||dx||^2 per CTA
  double* part_p_split;  // ||dx||^2 of each split row
  int mode;
  int direct;
};

template <class T>
struct DualArgs {
  CsrView<T> A;          // CSR of A (rows = constraints)
  TileView<T> plan;      // tiles of A
  const int32_t* p_cta_begin;    // primal plan: first CTA of each instance
  const int32_t* p_split_begin;  // primal plan: first split row of each instance
  const T* dx;
  const T* b;
  T* y0;
  T* y1;
  T* kx0;
  T* kx1;
  T* sy;
  T* skx;
  StepState* st_mut;     // one per instance; the instance's last CTA updates it
  const double* part_p;
  const double* part_p_split;
  double* part_d;        // [interaction | ||dy||^2] per CTA (num_ctas each)
  double* part_d_split;  // (interaction, ||dy||^2) of each split row
  int direct;            // dx holds x^ and the row sums are K x^ (see above)
};

// Sums over the CTA of Q <= 8 per-thread partials in a fixed order: out[q] in shared memory, complete
// after the final barrier; `sh` holds Q * kBlock doubles and may be reused by consecutive calls. An
// FP64 addition takes 64 cycles and the pipe 2 lanes per SM and cycle, so FP64 partials go through
// shared memory and warp q adds quantity q: lane l entry l of every warp in warp order, then a
// shuffle tree (12 dependent additions; two quantities one after the other took 2,300 cycles). FP32
// partials: a shuffle tree per warp in FP32, the warp sums added in FP64 in warp order.
// post(q, sum), run by the one thread that has sum q, gives what out[q] takes.
struct KeepSum {
  __device__ __forceinline__ double operator()(int, double sum) const { return sum; }
};
template <int Q, class T, class Post = KeepSum>
__device__ __forceinline__ void cta_sums(const T (&v)[Q], double* out, double* sh, Post post = Post()) {
  static_assert(Q <= kBlock / 32, "one warp per quantity");
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  __syncthreads();  // a previous call's readers are done with sh and out
  if constexpr (sizeof(T) == 8) {
#pragma unroll
    for (int q = 0; q < Q; ++q) sh[q * kBlock + t] = v[q];
    __syncthreads();
    if (warp < Q) {
      const double* c = sh + warp * kBlock + lane;
      double sum = c[0];
#pragma unroll
      for (int w = 1; w < kBlock / 32; ++w) sum += c[32 * w];
      sum = warp_sum(sum);
      if (lane == 0) out[warp] = post(warp, sum);
    }
  } else {
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const T ws = warp_sum(v[q]);
      if (lane == 0) sh[q * 32 + warp] = (double)ws;
    }
    __syncthreads();
    if (warp < Q && lane == 0) {
      double sum = sh[warp * 32];
#pragma unroll
      for (int w = 1; w < kBlock / 32; ++w) sum += sh[warp * 32 + w];
      out[warp] = post(warp, sum);
    }
  }
  __syncthreads();
}

// One lane's epilogue inputs for its row of a tile (issued with the tile's matrix loads).
template <class T>
struct PrimalIn {
  T dx;  // dx (x^ in direct mode); K'y when no commit is pending
  T x;
  T sx;
  T c;
  T l;
  T u;
};

// FP64 step kernels run row epilogues after the CTA's row sums are in shared memory, one row
// per thread (the dual kernel for its warp tiles, the primal kernel for its warp-streamed
// rows). Summed tile by tile, a tile's epilogue (about a dozen FP64 instructions per row) runs
// on only the lanes that own its rows (a handful when rows are longer than a lane's run, one
// for a streamed row), yet every warp-wide FP64 instruction occupies GB300's narrow FP64 pipe
// for the whole warp: on the power-law LP that made the pipe, not memory, the dual's bound
// (79% busy). FP32 keeps the per-tile epilogue (its pipe is wide, and the shared-memory row
// buffer would take L1 from the gathers).
template <class T>
constexpr bool kDenseEpilogue = sizeof(T) == 8;
template <class T>
constexpr int kDenseSlots = kDenseEpilogue<T> ? kTilesPerCtaMax * kTileRows : 1;

// What a primal pass takes from its instance's state: whether an accepted step waits for its
// commit, that step's averaging weight, step_size / primal_weight and the current dual.
template <class T>
struct PrimalScalars {
  bool pending;
  T w;
  T tto;
  const T* yg;
};

// Column j's epilogue inputs.
template <class T>
__device__ __forceinline__ void primal_load(const PrimalArgs<T>& a, bool pending, bool commit_only, int j,
                                            PrimalIn<T>& e) {
  if (!commit_only) {
    e.c = lds(a.c + j);
    e.l = lds(a.l + j);
    e.u = lds(a.u + j);
  }
  if (pending) {
    e.dx = lds(a.dx + j);
    if (!a.direct) e.x = lds(a.x + j);
    e.sx = lds(a.sx + j);
  } else {
    e.x = lds(a.x + j);
    e.dx = lds(a.kty + j);
  }
}
// x^ = proj(x - (tau/omega)(c - K'y)) and dx (:177-197), which is returned; out is what the dual
// pass gathers.
template <class T>
__device__ __forceinline__ T primal_candidate(const PrimalArgs<T>& a, T tto, int j, T xv, T ktyv, const PrimalIn<T>& e,
                                              T& out) {
  T v = xv - tto * (e.c - ktyv);
  v = imin(e.u, imax(e.l, v));   // min(u, max(l, .)) (:192)
  const T d = v - xv;
  out = a.direct ? v : d;
  a.dx[j] = out;                 // gathered by the dual kernel next: a normal (L2-resident) store
  return d;
}
// The accepted step applied to column j with K'y = ktyv; returns the new x.
template <class T>
__device__ __forceinline__ T primal_commit(const PrimalArgs<T>& a, T w, int j, T ktyv, const PrimalIn<T>& e) {
  const T xv = a.direct ? e.dx : e.x + e.dx;   // x += dx (:303)
  sts(a.x + j, xv);
  sts(a.kty + j, ktyv);                         // K'y = A'y (:307)
  sts(a.sx + j, e.sx + xv * w);                 // weighted sum (src/saddle_point_gpu.jl:137)
  return xv;
}

// Shared memory of a CTA's primal work.
template <class T>
struct PrimalShared {
  T rs_all[kBlock / 32][32];
  T wlane[kBlock];
  T lsum[kDenseEpilogue<T> ? kTilesPerCtaMax : 1];   // sums of FP64 warp-streamed rows
};

// One CTA's primal work on its nt staged tiles: the pending commit and the next candidate of
// every row (commit_only: the commit alone). acc takes the thread's share of ||dx||^2.
template <class T>
__device__ __forceinline__ void primal_work(const PrimalArgs<T>& a, const PrimalScalars<T>& sc, PrimalShared<T>& sm,
                                            const Tile* tl, int nt, bool commit_only, T& acc) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool pending = sc.pending;
  const T w = sc.w, tto = sc.tto;
  const T* yg = sc.yg;
  T* rs = sm.rs_all[warp];
  auto load_in = [&](const Tile& t, PrimalIn<T>& e) {
    e = PrimalIn<T>{};
    if (lane < t.rows) primal_load(a, pending, commit_only, t.row_begin + lane, e);
  };
  // the candidate; its ||dx||^2 term goes into the CTA's sum with one FMA, or into the split
  // row's own slot
  auto candidate = [&](int j, T xv, T ktyv, const PrimalIn<T>& e, const Tile& t, bool split) {
    T out;
    const T d = primal_candidate(a, tto, j, xv, ktyv, e, out);
    if (split) {
      a.part_p_split[t.split] = (double)(d * d);
      __threadfence();
    } else {
      acc = fma(d, d, acc);
    }
  };
  // split handling and the fused epilogue of tile t, once its row sums are in rs
  auto finish = [&](const Tile& t, const PrimalIn<T>& e) {
    const bool split = t.split >= 0;
    const int j = t.row_begin + lane;
    if (pending) {
      int rows = t.rows;
      if (split) rows = split_finish(t, a.plan, rs) ? 1 : 0;
      if (lane < rows) {
        const T ktyv = rs[lane];
        const T xv = primal_commit(a, w, j, ktyv, e);
        if (!commit_only) candidate(j, xv, ktyv, e, t, split);
      }
      __syncwarp();
    } else {
      // previous attempt rejected: K'y is unchanged, only the candidate is recomputed
      const int rows = (split && t.piece != t.pieces - 1) ? 0 : t.rows;
      if (lane < rows) candidate(j, e.x, e.dx, e, t, split);
    }
  };
  TileLoad<T> L0;
  PrimalIn<T> E0;
  if (nt > 0 && tl[0].e_log2 <= group_code(1)) {
    // group tiles: 8 / W long rows, W warps each; the group's first warp finishes its row
    const int W = 1 << group_log2(tl[0].e_log2);
    const int q = warp / W, sub = warp % W;
    const bool has = q < nt;
    Tile t{};
    if (has) t = tl[q];
    if (has && sub == 0) load_in(t, E0);
    if (pending) group_row_sum(a.At.col, a.At.val, yg, t, has, W, sub, sm.wlane, rs);
    if (has && sub == 0) finish(t, E0);
  } else if (kDenseEpilogue<T> && nt > 0 && tl[0].e_log2 == kWarpLong) {
    // FP64 CTAs of warp-streamed rows (one row per tile): the warps stream their rows' sums
    // into shared memory, then thread q runs the epilogue of tile q's row, so the FP64
    // instructions of the epilogue run on full warps instead of on each warp's lane 0
    if (pending)
      for (int q = warp; q < nt; q += kBlock / 32) {
        const T sum = long_row_sum(a.At.col, a.At.val, yg, tl[q]);
        if (lane == 0) sm.lsum[q] = sum;
      }
    __syncthreads();
    for (int q = threadIdx.x; q < nt; q += kBlock) {
      const Tile& t = tl[q];
      const int j = t.row_begin;
      PrimalIn<T> e{};
      primal_load(a, pending, commit_only, j, e);
      if (pending) {
        const T ktyv = sm.lsum[q];
        const T xv = primal_commit(a, w, j, ktyv, e);
        if (!commit_only) candidate(j, xv, ktyv, e, t, false);
      } else {
        candidate(j, e.x, e.dx, e, t, false);
      }
    }
  } else {
    // each warp walks its tiles q = warp, warp + 8, ...: a tile's epilogue inputs, row
    // offsets, columns and values are all issued before any of them is used
    for (int q = warp; q < nt; q += kBlock / 32) {
      const Tile t = tl[q];
      load_in(t, E0);
      if (pending) {
        tile_load(a.At.row_ptr, a.plan.icol, a.plan.ival, t, L0);
        tile_sums(a.At.col, a.At.val, yg, t, L0, rs);
      }
      finish(t, E0);
    }
  }
}

template <class T, int kCtas>
__global__ void __launch_bounds__(kBlock, kCtas) primal_step_kernel(PrimalArgs<T> a) {
  __shared__ PrimalShared<T> sm;
  __shared__ union {   // the tiles are done with when the sums begin (cta_sums' first barrier)
    Tile tl[kTilesPerCtaMax];
    double red[kBlock];
  } ph;
  Tile* const tl = ph.tl;
  double* const red = ph.red;
  const int b = a.plan.cta_map ? a.plan.cta_map[blockIdx.x] : (int)blockIdx.x;
  // programmatic dependent launch: stage the constant tile descriptors, wait for the previous
  // kernel, and only then let the next (dual) kernel's CTAs launch: once all of ours have
  // passed this point, the state the previous dual kernel wrote is complete, so the dual
  // kernel may read it before its own wait (this kernel never writes it)
  const int nt = stage_tiles(a.plan.tiles, a.plan.cta_tile_begin[b], a.plan.cta_tile_begin[b + 1], tl);
  pdl_wait();
  pdl_launch_dependents();
  const StepState* st = a.st + a.plan.cta_inst[b];
  const int pending = st->pending_commit;
  const bool commit_only = a.mode == kStepCommitOnly;
  if (commit_only ? !pending || !st->eval_active : st->done != 0) return;
  const PrimalScalars<T> sc{pending != 0, (T)st->commit_weight, (T)st->tto, st->parity ? a.y1 : a.y0};
  T acc = T(0);
  primal_work(a, sc, sm, tl, nt, commit_only, acc);
  if (commit_only) return;
  const T v[1] = {acc};
  __shared__ double o[1];
  cta_sums<1>(v, o, red);
  if (threadIdx.x == 0) a.part_p[b] = o[0];
}

// The chunk is finished: what its evaluation, already queued behind it, needs of the state.
__device__ __forceinline__ void end_chunk(StepState& s) {
  s.done = 1;
  s.eval_active = 1;
  // the average, or the current point (src/primal_dual_hybrid_gradient_gpu.jl:635-642)
  s.eval_current = s.numerical_error || s.count_primal == 0 || s.count_dual == 0 ? 1 : 0;
  if (!s.eval_current) {
    s.rcp_w_primal = 1.0 / s.sum_w_primal;
    s.rcp_w_dual = 1.0 / s.sum_w_dual;
  }
}

// Decision of take_step! for one attempt on the instance's state, by one thread: its chain of
// dependent FP64 operations, the division above all, is the attempt's serial tail, so comparisons
// run on the integer pipe. f1 / f2 are the step-size factors
// (1 - (k+1)^-r), (1 + (k+1)^-g) for the attempt counter after this attempt; movement is
// 0.5 omega ||dx||^2 + 0.5 / omega ||dy||^2. error: the numerical error of :384-390
// (terminate at the next evaluation; the step size is left as it is).
struct StepVerdict {
  double limit, next;   // the step-size limit and the next step size
  bool accept, error;
};
__device__ __forceinline__ StepVerdict step_verdict(const StepState& s, double f1, double f2, double inter_signed,
                                                    double movement) {
  const long long bi = __double_as_longlong(inter_signed) & 0x7fffffffffffffffLL;
  const bool interacts = !s.constant_step && bi > 0 && bi <= 0x7ff0000000000000LL;   // |inter| > 0, not NaN
  const double tau = s.tau;
  StepVerdict v;
  v.limit = __longlong_as_double(0x7ff0000000000000LL);
  if (interacts) v.limit = movement / __longlong_as_double(bi);
  v.error = interacts && (__double_as_longlong(movement) << 1) == 0;
  // positive operands and no NaN: order of the bits; else the comparisons as written
  const long long bl = __double_as_longlong(v.limit), bt = __double_as_longlong(tau);
  const bool plain = bl >= 0 && bl <= 0x7ff0000000000000LL && bt >= 0 && bt <= 0x7ff0000000000000LL;
  v.accept = !v.error && (s.constant_step || (plain ? bt <= bl : tau <= v.limit));
  v.next = tau;
  if (!s.constant_step) {
    const double first = f1 * v.limit, second = f2 * tau;
    const long long b1 = __double_as_longlong(first), b2 = __double_as_longlong(second);
    const bool both = b1 >= 0 && b1 <= 0x7ff0000000000000LL && b2 >= 0 && b2 <= 0x7ff0000000000000LL;
    v.next = both ? __longlong_as_double(b1 < b2 ? b1 : b2) : jmin(first, second);
  }
  return v;
}
// The verdict entered into the state.
__device__ __forceinline__ void step_account(StepState& s, const StepVerdict& v) {
  s.total_iters += s.constant_step ? 0 : 1;
  s.kkt_passes += 1.0;
  s.attempts_in_chunk += 1;
  const bool ends = v.error || s.accepted_in_chunk + (v.accept ? 1 : 0) >= s.target_in_chunk ||
                    s.attempts_in_chunk >= s.max_attempts_in_chunk;
  if (ends || s.attempts_in_chunk == s.launch_attempts) s.launch_ns = global_ns() - s.launch_start_ns;
  if (v.error) {
    s.numerical_error = 1;
    s.pending_commit = 0;
    end_chunk(s);
    return;
  }
  s.tau = v.next;
  s.last_limit = v.limit;
  s.pending_commit = v.accept ? 1 : 0;
  if (v.accept) {
    s.parity ^= 1;
    s.commit_weight = s.iter_start_tau;
    s.count_primal += 1;
    s.count_dual += 1;
    s.sum_w_primal += s.iter_start_tau;
    s.sum_w_dual += s.iter_start_tau;
    s.accepted += 1;
    s.accepted_in_chunk += 1;
    s.iter_start_tau = v.next;
  } else {
    s.rejected += 1;
  }
  if (ends) end_chunk(s);
}

// Step-size factors of the attempt that the state (in L2 or shared memory) stands before (take_step!,
// :405-407): the host table while it lasts, else the same formula on the device.
__device__ __forceinline__ void step_factors(const StepState* st, double (&f)[2]) {
  const long long k = *(volatile const long long*)&st->total_iters + (*(volatile const int*)&st->constant_step ? 0 : 1);
  if (st->pow_table && k < st->pow_table_len) {
    f[0] = __ldcg(st->pow_table + 2 * k);
    f[1] = __ldcg(st->pow_table + 2 * k + 1);
  } else {
    const double k1 = (double)(k + 1);
    f[0] = 1.0 - 1.0 / pow(k1, st->reduction_exponent);
    f[1] = 1.0 + 1.0 / pow(k1, st->growth_exponent);
  }
}

// One lane's epilogue inputs for its row of a tile of A (issued with the tile's matrix loads).
template <class T>
struct DualIn {
  T y;
  T kx;
  T b;
  T sy;
  T sk;
};

// The dual kernel's FP64 tiles stop their segmented scan at the longest lane span of a
// crossing row (tile_sums); FP32 adds are cheap and keep the full scan.
template <class T>
constexpr bool kSpanScan = sizeof(T) == 8;

// What a dual pass takes from its instance's state.
template <class T>
struct DualScalars {
  bool pending;
  T w;
  T od;            // primal_weight * step_size
  const T* ycur;
  T* ynew;
  const T* kxcur;
  T* kxnew;
};

// Row i's epilogue inputs.
template <class T>
__device__ __forceinline__ void dual_load(const DualArgs<T>& a, const DualScalars<T>& sc, int i, DualIn<T>& e) {
  e.y = lds(sc.ycur + i);
  e.kx = lds(sc.kxcur + i);
  e.b = lds(a.b + i);
  if (sc.pending) {
    e.sy = lds(a.sy + i);
    e.sk = lds(a.skx + i);
  }
}
// Row i's pending sums and its candidate y^ (returned) from the row sum rsum, with kdx and d = dy.
template <class T>
__device__ __forceinline__ T dual_row(const DualArgs<T>& a, const DualScalars<T>& sc, int i, bool ineq, T rsum,
                                         const DualIn<T>& e, T& kdx, T& d) {
  const T y = e.y, kx = e.kx;
  if (sc.pending) {
    sts(a.sy + i, e.sy + y * sc.w);
    sts(a.skx + i, e.sk + kx * sc.w);
  }
  kdx = a.direct ? rsum - kx : rsum;
  T v = y + sc.od * ((e.b - T(2) * kdx) - kx);   // (:247), extrapolation coefficient 1
  if (ineq) v = imax(v, T(0));                   // (:254)
  d = v - y;
  const T out = y + d;                           // y += dy (:306)
  sc.ynew[i] = out;                              // gathered by the next primal kernel
  sts(sc.kxnew + i, a.direct ? rsum : kx + kdx); // Kx += K dx (:304)
  return out;
}

// Shared memory of a CTA's dual work.
template <class T>
struct DualShared {
  T rs_all[kBlock / 32][32];
  T wlane[kBlock];
  T ipart[kBlock / 32][kBlock / 32];
  T csum[kDenseSlots<T>];                    // FP64 warp tiles: every row's sum,
  int32_t slot_begin[kTilesPerCtaMax + 1];   // and each tile's first slot in it
};

// One CTA's dual work on its nt staged tiles: the pending commit's y and Kx sums and the next
// candidate of every row. acc_i / acc_d take the thread's share of dy . K dx and ||dy||^2.
template <class T>
__device__ __forceinline__ void dual_work(const DualArgs<T>& a, const DualScalars<T>& sc, DualShared<T>& sm,
                                          const Tile* tl, int nt, T& acc_i, T& acc_d) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  T* rs = sm.rs_all[warp];
  auto load_in = [&](const Tile& t, DualIn<T>& e) {
    e = DualIn<T>{};
    if (lane < t.rows) dual_load(a, sc, t.row_begin + lane, e);
  };
  auto finish = [&](const Tile& t, const DualIn<T>& e) {
    const bool split = t.split >= 0;
    const int i = t.row_begin + lane;
    int rows = t.rows;
    if (split) rows = split_finish(t, a.plan, rs) ? 1 : 0;
    if (lane < rows) {
      T kdx, d;
      dual_row(a, sc, i, i >= t.aux, rs[lane], e, kdx, d);
      if (split) {
        a.part_d_split[2 * t.split] = (double)(kdx * d);
        a.part_d_split[2 * t.split + 1] = (double)(d * d);
        __threadfence();
      } else {
        acc_i = fma(kdx, d, acc_i);
        acc_d = fma(d, d, acc_d);
      }
    }
    __syncwarp();
  };
  TileLoad<T> L0;
  DualIn<T> E0;
  bool interleave = nt == kBlock / 32;
  for (int q = 0; q < nt && interleave; ++q) interleave = tl[q].e_log2 == kWarpLong;
  if (interleave) {
    // kBlock / 32 warp-streamed rows summed together (interleaved_rows_sum); warp w then
    // finishes row w as if it had streamed it
    load_in(tl[warp], E0);
    interleaved_rows_sum(a.A.col, a.A.val, a.dx, tl, sm.ipart, sm.rs_all);
    finish(tl[warp], E0);
  } else if (nt > 0 && tl[0].e_log2 <= group_code(1)) {
    const int W = 1 << group_log2(tl[0].e_log2);
    const int q = warp / W, sub = warp % W;
    const bool has = q < nt;
    Tile t{};
    if (has) t = tl[q];
    if (has && sub == 0) load_in(t, E0);
    group_row_sum(a.A.col, a.A.val, a.dx, t, has, W, sub, sm.wlane, rs);
    if (has && sub == 0) finish(t, E0);
  } else if (kDenseEpilogue<T>) {
    // warp tiles (never split): every row sum into the CTA's slot buffer, then the epilogue
    // with one row per thread, slot by slot (slot = the row's position among the tiles' rows)
    T* csum = sm.csum;
    int32_t* slot_begin = sm.slot_begin;
    if (threadIdx.x == 0) {
      int o = 0;
      for (int q = 0; q < nt; ++q) {
        slot_begin[q] = o;
        o += tl[q].rows;
      }
      slot_begin[nt] = o;
    }
    __syncthreads();
    for (int q = warp; q < nt; q += kBlock / 32) {
      const Tile t = tl[q];
      tile_load(a.A.row_ptr, a.plan.icol, a.plan.ival, t, L0);
      tile_sums<T, kSpanScan<T>>(a.A.col, a.A.val, a.dx, t, L0, rs);
      if (lane < t.rows) csum[slot_begin[q] + lane] = rs[lane];
      __syncwarp();
    }
    __syncthreads();
    const int nslots = slot_begin[nt];
    for (int sl = threadIdx.x; sl < nslots; sl += kBlock) {
      int lo = 0, hi = nt - 1;   // the last tile starting at or before the slot (the non-empty one)
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (slot_begin[mid] <= sl) lo = mid;
        else hi = mid - 1;
      }
      const int i = tl[lo].row_begin + (sl - slot_begin[lo]);
      DualIn<T> e{};
      dual_load(a, sc, i, e);
      T kdx, d;
      dual_row(a, sc, i, i >= tl[lo].aux, csum[sl], e, kdx, d);
      acc_i = fma(kdx, d, acc_i);
      acc_d = fma(d, d, acc_d);
    }
  } else {
    for (int q = warp; q < nt; q += kBlock / 32) {
      const Tile t = tl[q];
      load_in(t, E0);
      tile_load(a.A.row_ptr, a.plan.icol, a.plan.ival, t, L0);
      tile_sums<T, kSpanScan<T>>(a.A.col, a.A.val, a.dx, t, L0, rs);
      finish(t, E0);
    }
  }
}

constexpr int kStateWords = (int)(sizeof(StepState) / 8);
static_assert(sizeof(StepState) % 8 == 0 && kStateWords <= kBlock, "StepState copies");
// The state between L2 and shared memory, one 8-byte word per thread (the caller synchronises).
__device__ __forceinline__ void load_state(const StepState* st, StepState& s) {
  if (threadIdx.x < kStateWords)
    reinterpret_cast<unsigned long long*>(&s)[threadIdx.x] =
        __ldcg(reinterpret_cast<const unsigned long long*>(st) + threadIdx.x);
}
__device__ __forceinline__ void store_state(const StepState& s, StepState* st) {
  if (threadIdx.x < kStateWords)
    reinterpret_cast<unsigned long long*>(st)[threadIdx.x] = reinterpret_cast<const unsigned long long*>(&s)[threadIdx.x];
}

// Plan ranges of an instance: first and end CTA and split row of the dual plan, then of the primal plan.
struct PlanRanges {
  int c0, c1, s0, s1, p0, p1, q0, q1;
};

// What the step decision needs of the instance's sums, in tot (shared): the interaction, ||dy|| and
// 0.5 omega ||dx|| ||dx|| (the primal part of take_step!'s movement, :324-333, evaluated as the
// reference does, the norm squared again). One round of loads for the CTAs' sums of both kernels
// up to 4 x kBlock CTAs, all issued before any is added; split-row slots (rare) follow. The roots
// (580 cycles each) are taken side by side, each by the warp that has its sum.
template <class T>
__device__ __forceinline__ void step_totals(const DualArgs<T>& a, const PlanRanges& g, const StepState& s, double* tot,
                                            double* red) {
  double sd[3] = {0.0, 0.0, 0.0};
  const int count = max(g.c1 - g.c0, g.p1 - g.p0);
  for (int k0 = (int)threadIdx.x; k0 < count; k0 += 4 * kBlock) {
    double ui[4], ud[4], ux[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int k = k0 + j * kBlock;
      const bool in = k < g.c1 - g.c0;
      ui[j] = in ? __ldcg(a.part_d + g.c0 + k) : 0.0;
      ud[j] = in ? __ldcg(a.part_d + a.plan.num_ctas + g.c0 + k) : 0.0;
      ux[j] = k < g.p1 - g.p0 ? __ldcg(a.part_p + g.p0 + k) : 0.0;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (k0 + j * kBlock >= count) break;
      sd[0] += ui[j];
      sd[1] += ud[j];
      sd[2] += ux[j];
    }
  }
  for (int k = g.s0 + (int)threadIdx.x; k < g.s1; k += kBlock) {
    sd[0] += __ldcg(a.part_d_split + 2 * k);
    sd[1] += __ldcg(a.part_d_split + 2 * k + 1);
  }
  for (int k = g.q0 + (int)threadIdx.x; k < g.q1; k += kBlock) sd[2] += __ldcg(a.part_p_split + k);
  cta_sums<3>(sd, tot, red, [&](int q, double sum) {
    if (q == 0) return sum;
    const double norm = sqrt(sum);
    return q == 1 ? norm : __dmul_rn(__dmul_rn(0.5 * s.omega, norm), norm);
  });
}

template <class T, int kCtas>
__global__ void __launch_bounds__(kBlock, kCtas) dual_step_kernel(DualArgs<T> a) {
  __shared__ DualShared<T> sm;
  __shared__ union {   // the tiles are done with when the sums begin (cta_sums' first barrier)
    Tile tl[kTilesPerCtaMax];
    double red[3 * kBlock];
  } ph;
  Tile* const tl = ph.tl;
  double* const red = ph.red;
  __shared__ int is_last;
  __shared__ double tot[3];
  const int b = a.plan.cta_map ? a.plan.cta_map[blockIdx.x] : (int)blockIdx.x;
  pdl_launch_dependents();  // the next primal kernel reads the state only after its wait
  // The state this kernel reads was written by the previous dual kernel, which completed before
  // the primal kernel let this one launch (see there): read it now, from L2 (a line in this SM's
  // L1 may predate it), so the loads overlap the primal kernel's last CTAs. The last CTA of the
  // instance takes the decision on this copy, with the plan ranges read here too: loads of either
  // after the last arrival would be on every attempt's path (FP64, 20,011 x 40,022: 24.8 us an
  // attempt with them there, 22.4 with them here; FP32, 90,007 x 180,014: 35.9 and 30.8).
  __shared__ StepState s;
  __shared__ PlanRanges range;
  const int inst = a.plan.cta_inst[b];
  StepState* stw = a.st_mut + inst;
  load_state(stw, s);
  if (threadIdx.x >= 64 && threadIdx.x < 72) {
    const int k = (int)threadIdx.x - 64, end = k & 1;
    const int32_t* v[4] = {a.plan.inst_cta_begin, a.plan.inst_split_begin, a.p_cta_begin, a.p_split_begin};
    reinterpret_cast<int*>(&range)[k] = v[k >> 1][inst + end];
  }
  const int nt = stage_tiles(a.plan.tiles, a.plan.cta_tile_begin[b], a.plan.cta_tile_begin[b + 1], tl);
  pdl_wait();
  if (s.done) return;
  const int p = s.parity;
  const bool pending = s.pending_commit != 0;
  const DualScalars<T> sc{pending, (T)s.commit_weight, (T)(s.omega * s.tau), p ? a.y1 : a.y0, p ? a.y0 : a.y1,
                          p ? a.kx1 : a.kx0, p ? a.kx0 : a.kx1};
  T acc_i = T(0), acc_d = T(0);
  dual_work(a, sc, sm, tl, nt, acc_i, acc_d);
  const T v[2] = {acc_i, acc_d};
  cta_sums<2>(v, tot, red);
  if (threadIdx.x == 0) {
    a.part_d[b] = tot[0];
    a.part_d[a.plan.num_ctas + b] = tot[1];
    __threadfence();
    const unsigned prev = atomicAdd(&stw->arrive, 1u);
    is_last = (prev == (unsigned)(range.c1 - range.c0 - 1)) ? 1 : 0;
  }
  __syncthreads();
  if (!is_last) return;
  // The instance's last CTA: all CTAs' sums in one round of loads, the step-size factors by a warp
  // that adds none, then thread 0 takes the decision. This tail is on every attempt's path (3-4 us of
  // the 13 us that an attempt of a 203 x 406 LP takes as step kernels): with the primal sum and the
  // decision's inputs formed by the instance's first CTA after its own work, sums by one warp and the
  // state and ranges loaded here it took more than twice as long.
  __shared__ double factors[2];
  if (threadIdx.x == 32 * (kBlock / 32 - 1)) step_factors(&s, factors);
  step_totals(a, range, s, tot, red);
  if (threadIdx.x == 0) {
    s.arrive = 0;
    if (pending) s.primal_spmv += 1;
    step_account(s, step_verdict(s, factors[0], factors[1], tot[0],
                                 __fma_rn(__dmul_rn(s.half_over_omega, tot[1]), tot[1], tot[2])));
    s.tto = s.tau / s.omega;
  }
  __syncthreads();
  store_state(s, stw);
}

// The step kernels are compiled for 2, 3 and 4 resident CTAs per SM, and a launch takes the first that
// holds all of its CTAs at once: a lane's loads in flight and its sums then have up to 128 registers
// instead of 64 (1 per SM, 255 registers, was no faster for 128 CTAs). Per attempt, all with 4 -> as
// chosen: FP64 6,000 x 12,000 (128 dual CTAs) 17.7 -> 15.7 us, 10,000 x 20,000 (212) 18.8 -> 16.3,
// 20,011 x 40,022 (425) 22.1 -> 20.3; FP32 20,000 x 40,000 (204) 16.1 -> 15.9, 40,000 x 80,000 (449)
// 20.6 -> 18.8. One more CTA than fits is a second wave: FP64 22,000 x 44,000 (467) takes 22.3 with 4
// and 25.3 with 3. The lines follow from kSms: on a part with another number of SMs a launch may
// take another variant, with the same results.
template <class T>
using PrimalKernel = void (*)(PrimalArgs<T>);
template <class T>
using DualKernel = void (*)(DualArgs<T>);
template <class T>
inline PrimalKernel<T> primal_kernel(int ctas) {
  static_assert(kPrimalCtasPerSm<T> == 4);
  return ctas <= 2 * kSms ? primal_step_kernel<T, 2> : ctas <= 3 * kSms ? primal_step_kernel<T, 3> : primal_step_kernel<T, 4>;
}
template <class T>
inline DualKernel<T> dual_kernel(int ctas) {
  static_assert(kDualCtasPerSm == 4);
  return ctas <= 2 * kSms ? dual_step_kernel<T, 2> : ctas <= 3 * kSms ? dual_step_kernel<T, 3> : dual_step_kernel<T, 4>;
}

// Launches a step kernel with programmatic dependent launch enabled (see pdl_wait).
template <class Args>
inline void launch_step(void (*kernel)(Args), int grid, cudaStream_t s, const Args& args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kBlock);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  CK(cudaLaunchKernelEx(&cfg, kernel, args));
}

}  // namespace gpdhg
