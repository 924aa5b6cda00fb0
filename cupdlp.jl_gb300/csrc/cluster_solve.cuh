// cluster_solve.cuh — a whole evaluation interval of PDHG step attempts of a small LP on one
// thread-block cluster.
//
// Launched one by one (step_kernels.cuh), an attempt of a small LP is latency: two launches, loads of
// descriptors, state and matrix, and chains of dependent FP64 operations (64 cycles each on GB300),
// around a microsecond of work: 13.4 us for a 203 x 406 and 13.1 for a 1,000 x 2,000 LP in FP64,
// against 7.2 and 7.5 here (launch and staging, 5-6 us an interval, included). Here a cluster
// of up to 16 CTAs keeps the LP on chip for the interval: every CTA holds its share of both
// matrices in shared memory (columns, values and the lanes' row structure, staged once per
// launch) and the whole of the two gathered vectors, x^ / dx and y, into which the CTAs write their
// rows' entries over distributed shared memory. A cluster barrier takes 500 cycles, against 2,200
// for one through L2 (which also rules out the same scheme over the whole GPU: 900-1,300 cycles
// per exchange, and gathers of exchanged words that miss L1). Two barriers per attempt: after the
// primal half (x^ is there) and after the dual half (y and the CTAs' sums are there); every CTA
// then takes the step decision itself.
//
// The work units and every sum's order are those of the step kernels (a CTA here runs the plan CTAs
// b = rank, rank + size, ... of its LP, one tile per warp), so the results are the same bits
// whichever path runs.
//
// A vector needs one buffer: y is gathered in the primal half and written in the dual half, x^ the
// other way round, with a barrier between; a rejected attempt's y is never gathered.
#pragma once

#include "step_kernels.cuh"

namespace gpdhg {

constexpr int kClusterThreads = kBlock + 32;   // a warp per tile, and one that decides
constexpr int kClusterMax = 16;       // CTAs per cluster (above 8: non-portable, GB300 takes 16)
// Plan CTAs per CTA and side, at most. Each round more is a pass of every warp through both halves of
// an attempt: FP64 7.0-7.6 us an attempt with one, 10.1-12.4 with two, 16.1-18.0 with three, against
// 12.5-13.2 as step kernels; FP32 5.1-6.0, 7.3-9.4 and (three) 11.1-13.1, against 11.1-11.7. Random LPs of
// 203 to 5,500 rows with 5 to 20 nonzeros; the room for four rounds cost the others 3-10%.
constexpr int kClusterRounds = 2;
constexpr int kClusterPlanCtas = kClusterMax * kClusterRounds;
constexpr size_t kClusterShared = 200 * 1024;
// Attempts per launch at most (a chunk normally takes its 1 to 64 accepted steps and a few
// rejections): the host launches again while the chunk is not finished.
constexpr int kClusterAttempts = 8192;

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_size() {
  unsigned n;
  asm volatile("mov.u32 %0, %cluster_nctarank;" : "=r"(n));
  return n;
}
// A product kept from being fused with what uses it.
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }

// One side's share of one round: the tiles of a plan CTA, one per warp.
template <class T>
struct ClusterSide {
  T* val;
  unsigned long long* rows;   // 32 per tile: where the sum after each of the lane's elements goes (8
                              // bits): the row that ends there, 33 + lane if it began in an earlier lane, else 32
  int32_t* col;
  unsigned* info;             // 32 per tile: the lane's RunInfo
  Tile* tiles;
  int count;
  int slot0;                  // first slot of the plan's copy staged here
};
constexpr int kClusterTiles = kBlock / 32;
__host__ __device__ constexpr size_t cluster_side_bytes(int slots, int value_bytes) {
  return ((size_t)slots * (value_bytes + 4) + kClusterTiles * (32 * 12 + sizeof(Tile)) + 15) / 16 * 16;
}
template <class T>
__device__ __forceinline__ ClusterSide<T> cluster_side(char* base, int tiles, int slots, int slot0) {
  ClusterSide<T> s;
  s.val = reinterpret_cast<T*>(base);
  s.rows = reinterpret_cast<unsigned long long*>(s.val + slots);
  s.col = reinterpret_cast<int32_t*>(s.rows + 32 * kClusterTiles);
  s.info = reinterpret_cast<unsigned*>(s.col + slots);
  s.tiles = reinterpret_cast<Tile*>(s.info + 32 * kClusterTiles);
  s.count = tiles;
  s.slot0 = slot0;
  return s;
}

// How a lane walks its elements of a tile: bits 0-7 the elements after which a row ends, then
// whether the first of them ends a row that began in an earlier lane (and bits 24-28 that row), whether
// its last row goes on in the next lane, and whether that row began in this lane; the elements it
// holds; and the tile's scan length (how many lanes back a completed row begins, at most).
struct RunInfo {
  static constexpr unsigned kHead = 1u << 8, kTail = 1u << 9, kTailStart = 1u << 10;
  static constexpr int kCountShift = 12, kSpanShift = 16, kRowShift = 24;
};

// Copies a plan CTA's tiles from `tile` on; the caller synchronises.
template <class T>
__device__ __forceinline__ void stage_cluster_side(const ClusterSide<T>& s, const TileView<T>& plan,
                                                   const int32_t* row_ptr, int tile, int slots) {
  const int* src = reinterpret_cast<const int*>(plan.tiles + tile);
  int* dst = reinterpret_cast<int*>(s.tiles);
  for (int k = threadIdx.x; k < s.count * (int)(sizeof(Tile) / 4); k += kClusterThreads) dst[k] = src[k];
  // slots come in multiples of 32 from a multiple of 32, so both copies go in 16-byte pieces
  const int4* vs = reinterpret_cast<const int4*>(plan.ival + s.slot0);
  int4* vd = reinterpret_cast<int4*>(s.val);
  for (int k = threadIdx.x; k < slots * (int)sizeof(T) / 16; k += kClusterThreads) vd[k] = vs[k];
  const int4* cs = reinterpret_cast<const int4*>(plan.icol + s.slot0);
  int4* cd = reinterpret_cast<int4*>(s.col);
  for (int k = threadIdx.x; k < slots / 4; k += kClusterThreads) cd[k] = cs[k];
  const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (q >= s.count) return;
  const Tile& t = plan.tiles[tile + q];
  // lane i holds row i's first element; the rows of the lane's elements by binary search
  const int off = lane <= t.rows ? row_ptr[t.row_begin + lane] - t.nnz_begin : t.nnz;
  const int E = 1 << t.e_log2, kb = lane << t.e_log2, count = min(E, max(0, t.nnz - kb));
  unsigned long long rows = 0;
  unsigned info = (unsigned)count << RunInfo::kCountShift;
  int head_back = 0;
  for (int j = 0; j < E; ++j) {
    const int k = kb + j;
    int lo = 0, hi = t.rows > 0 ? t.rows - 1 : 0;   // the row with off[r] <= k < off[r + 1]
#pragma unroll
    for (int b = 0; b < 5; ++b) {
      const int mid = (lo + hi) >> 1;
      const int v = __shfl_sync(0xffffffffu, off, mid + 1);
      if (lo < hi) {
        if (v > k) hi = mid;
        else lo = mid + 1;
      }
    }
    const int begin = __shfl_sync(0xffffffffu, off, lo), end = __shfl_sync(0xffffffffu, off, lo + 1);
    if (j >= count) continue;
    int to = 32;
    if (k + 1 == end) {
      info |= 1u << j;
      to = lo;
      if (begin < kb) {
        head_back = lane - (begin >> t.e_log2);
        info |= RunInfo::kHead | (unsigned)lo << RunInfo::kRowShift;
        to = 33 + lane;
      }
    }
    rows |= (unsigned long long)to << (8 * j);
    if (k + 1 < end && j == count - 1) info |= RunInfo::kTail | (begin >= kb ? RunInfo::kTailStart : 0u);
  }
  info |= (unsigned)__reduce_max_sync(0xffffffffu, head_back) << RunInfo::kSpanShift;
  s.rows[32 * q + lane] = rows;
  s.info[32 * q + lane] = info;
}

template <class U, int kEMax>
__device__ __forceinline__ void staged_run(const U* base, int e_log2, U* d) {
  constexpr int G = 16 / (int)sizeof(U);
  const int lane = threadIdx.x & 31;
  const int E = 1 << e_log2;
  if (E >= G) {
#pragma unroll
    for (int g = 0; g < kEMax / G; ++g) {
      if (g * G >= E) break;  // uniform over the warp
      *reinterpret_cast<int4*>(d + G * g) = *reinterpret_cast<const int4*>(base + 32 * G * g + G * lane);
    }
  } else {
#pragma unroll
    for (int j = 0; j < (G - 1 < kEMax ? G - 1 : kEMax); ++j) {
      if (j >= E) break;
      d[j] = base[32 * j + lane];
    }
  }
}

// Row sums of the warp's tile q into rs, gathered from x (shared memory): the sums of tile_sums (same
// elements per lane, order and scan), with the walk over rows read from the staged structure and free of
// branches (rs: 65 entries).
template <class T>
__device__ __forceinline__ void staged_tile_sums(const ClusterSide<T>& s, const T* x, const Tile& t, int q, T* rs) {
  constexpr int kEMax = TileTraits<T>::kEMax;
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int E = 1 << t.e_log2;
  int c[kEMax];
  T v[kEMax], xv[kEMax];
  staged_run<int32_t, kEMax>(s.col + (t.data_begin - s.slot0), t.e_log2, c);
  staged_run<T, kEMax>(s.val + (t.data_begin - s.slot0), t.e_log2, v);
  const unsigned info = s.info[32 * q + lane];
  const unsigned long long rows = s.rows[32 * q + lane];
  const int count = (int)(info >> RunInfo::kCountShift) & 15;
  const unsigned to[2] = {(unsigned)rows, (unsigned)(rows >> 32)};
#pragma unroll
  for (int j = 0; j < kEMax; ++j) {
    if (j >= E) break;   // uniform over the warp
    xv[j] = j < count ? x[c[j]] : T(0);
  }
  rs[lane] = T(0);   // rows without elements
  __syncwarp();
  T sum = T(0);
#pragma unroll
  for (int j = 0; j < kEMax; ++j) {
    if (j >= E) break;
    if (j < count) {
      sum = fma(v[j], xv[j], sum);
      rs[to[j >> 2] >> (8 * (j & 3)) & 0xffu] = sum;
    }
    if (info >> j & 1u) sum = T(0);
  }
  const int span = (int)(info >> RunInfo::kSpanShift) & 31;
  if (span > 0) {
    T tail = info & RunInfo::kTail ? sum : T(0);
    int f = !(info & RunInfo::kTail) || (info & RunInfo::kTailStart) ? 1 : 0;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      if (d >= span) break;   // later steps change no value that a completed row reads
      const T up = __shfl_up_sync(full, tail, d);
      const int fu = __shfl_up_sync(full, f, d);
      if (lane >= d) {
        if (!f) tail = up + tail;
        f |= fu;
      }
    }
    const T prev = __shfl_up_sync(full, tail, 1);
    if (info & RunInfo::kHead) rs[info >> RunInfo::kRowShift & 31] = rs[33 + lane] + prev;
  }
  __syncwarp();
}

// Dynamic shared memory of a CTA: both vectors, the rows' terms of its rounds' sums, its tiles.
template <class T>
constexpr int kClusterTerms = sizeof(T) == 8 ? kBlock : kBlock / 32;   // per round and sum
template <class T>
__host__ __device__ constexpr size_t cluster_vector_bytes(int cols, int rows) {
  return ((size_t)cols * sizeof(T) + 15) / 16 * 16 + ((size_t)rows * sizeof(T) + 15) / 16 * 16;
}

// What the attempt under way takes of the state, which the ninth warp keeps up one attempt behind.
struct ClusterStep {
  double w, tto, od;   // commit weight, tau / omega, omega tau
  int pending, parity, done;
};

template <class T>
__global__ void __launch_bounds__(kClusterThreads, 1)
    cluster_kernel(PrimalArgs<T> pa, DualArgs<T> da, const int32_t* p_slot, const int32_t* d_slot, int cols, int rows) {
  extern __shared__ __align__(16) char dynamic[];
  __shared__ T rs_all[kBlock / 32][65];
  __shared__ double part[3][kClusterPlanCtas];   // every plan CTA's sums: dy . K dx, ||dy||^2, ||dx||^2
  __shared__ double total[3], factors[2];
  __shared__ int slot_begin[kClusterRounds][kClusterTiles];
  __shared__ StepState s;
  __shared__ ClusterStep now;
  const int size = (int)cluster_size(), rank = (int)cluster_rank();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  load_state(da.st_mut, s);
  __syncthreads();
  if (s.done) return;   // the whole cluster
  const int np = da.p_cta_begin[1], nd = da.plan.inst_cta_begin[1];   // plan CTAs of both sides
  T* xs = reinterpret_cast<T*>(dynamic);
  T* ys = reinterpret_cast<T*>(dynamic + cluster_vector_bytes<T>(cols, 0));
  char* at = dynamic + cluster_vector_bytes<T>(cols, rows);
  constexpr int kTerms = kClusterTerms<T>;
  double* terms = reinterpret_cast<double*>(at);   // [round][sum][kTerms]
  at += sizeof(double) * kClusterRounds * 3 * kTerms;
  ClusterSide<T> P[kClusterRounds], D[kClusterRounds];
#pragma unroll
  for (int k = 0; k < kClusterRounds; ++k) {
    const int b = rank + k * size;
    P[k].count = D[k].count = 0;
    if (b < np) {
      const int tile = pa.plan.cta_tile_begin[b], slots = p_slot[b + 1] - p_slot[b];
      P[k] = cluster_side<T>(at, pa.plan.cta_tile_begin[b + 1] - tile, slots, p_slot[b]);
      stage_cluster_side(P[k], pa.plan, pa.At.row_ptr, tile, slots);
      at += cluster_side_bytes(slots, sizeof(T));
    }
    if (b < nd) {
      const int tile = da.plan.cta_tile_begin[b], slots = d_slot[b + 1] - d_slot[b];
      D[k] = cluster_side<T>(at, da.plan.cta_tile_begin[b + 1] - tile, slots, d_slot[b]);
      stage_cluster_side(D[k], da.plan, da.A.row_ptr, tile, slots);
      at += cluster_side_bytes(slots, sizeof(T));
    }
  }
  const T* y_now = s.parity ? da.y1 : da.y0;
  for (int i = threadIdx.x; i < rows; i += kClusterThreads) ys[i] = y_now[i];
  for (int i = threadIdx.x; i < kClusterRounds * 3 * kTerms; i += kClusterThreads) terms[i] = 0.0;
  __syncthreads();
  if (threadIdx.x < kClusterRounds) {   // a row's place among the plan CTA's rows
    int at_row = 0;
#pragma unroll
    for (int k = 0; k < kClusterRounds; ++k)
      if (k == (int)threadIdx.x)
        for (int q = 0; q < D[k].count; ++q) {
          slot_begin[k][q] = at_row;
          at_row += D[k].tiles[q].rows;
        }
  }
  T* rs = rs_all[warp % (kBlock / 32)];
  // The ninth warp's first lane takes the decisions. Of one, the others wait for the verdict alone;
  // the state's upkeep and the division for tau / omega run beside the next attempt's sums (7.7 -> 7.4
  // and 7.9 -> 7.7 us an attempt of the LPs above).
  const bool decides = threadIdx.x == kBlock;
  StepVerdict verdict{};
  if (decides) {
    now = ClusterStep{s.commit_weight, s.tto, s.omega * s.tau, s.pending_commit, s.parity, 0};
    step_factors(&s, factors);
  }
  auto account = [&](bool was_pending) {
    if (was_pending) s.primal_spmv += 1;
    step_account(s, verdict);
    s.tto = s.tau / s.omega;
  };
  bool pending_before = false;
  cluster_barrier();   // every CTA runs and has staged: its shared memory may be written
  for (int attempt = 0; attempt < kClusterAttempts; ++attempt) {
    const bool pending = now.pending != 0;
    const int p = now.parity;
    const T w = (T)now.w;
    if (decides && attempt > 0) {
      account(pending_before);
      now.tto = s.tto;
      now.od = s.omega * s.tau;
      step_factors(&s, factors);   // used at the attempt's end
    }
#pragma unroll
    for (int k = 0; k < kClusterRounds; ++k) {
      const bool has = warp < P[k].count;
      Tile t{};
      if (has) t = P[k].tiles[warp];
      const int j = t.row_begin + lane;
      PrimalIn<T> e{};
      if (lane < t.rows) primal_load(pa, pending, false, j, e);
      // waits for the operands: left to their first use, behind the sums, an attempt takes 1.6 us more
      if (has) rs[lane] = e.x;
      T d = T(0), xv = e.x, ktyv = e.dx;
      if (has && pending) {
        staged_tile_sums(P[k], ys, t, warp, rs);
        if (lane < t.rows) {
          ktyv = rs[lane];
          xv = primal_commit(pa, w, j, ktyv, e);
        }
        __syncwarp();
      }
      if (k == 0) named_barrier<1, kClusterThreads>();   // tau / omega is there
      if (!has) continue;
      const T tto = (T)now.tto;
      if (lane < t.rows) {
        T out;
        d = primal_candidate(pa, tto, j, xv, ktyv, e, out);
        for (int r = 0; r < size; ++r) remote_store(remote_address(xs + j, r), out);
      }
      double* term = terms + (3 * k + 2) * kTerms;
      if constexpr (sizeof(T) == 8) {
        term[32 * warp + lane] = mul_rn(d, d);
      } else {
        const T sum = warp_sum(mul_rn(d, d));
        if (lane == 0) term[warp] = (double)sum;
      }
    }
    cluster_barrier();
    {
      const DualScalars<T> sc{pending, w, (T)now.od, p ? da.y1 : da.y0, p ? da.y0 : da.y1,
                              p ? da.kx1 : da.kx0, p ? da.kx0 : da.kx1};
#pragma unroll
      for (int k = 0; k < kClusterRounds; ++k) {
        if (warp >= D[k].count) continue;
        const Tile t = D[k].tiles[warp];
        const int i = t.row_begin + lane;
        DualIn<T> e{};
        if (lane < t.rows) dual_load(da, sc, i, e);
        staged_tile_sums(D[k], xs, t, warp, rs);
        T kdx = T(0), d = T(0);
        if (lane < t.rows) {
          const T out = dual_row(da, sc, i, i >= t.aux, rs[lane], e, kdx, d);
          for (int r = 0; r < size; ++r) remote_store(remote_address(ys + i, r), out);
        }
        __syncwarp();
        double* term = terms + 3 * k * kTerms;
        if constexpr (sizeof(T) == 8) {
          if (lane < t.rows) {
            term[slot_begin[k][warp] + lane] = mul_rn(kdx, d);
            term[kTerms + slot_begin[k][warp] + lane] = mul_rn(d, d);
          }
        } else {
          const T si = warp_sum(mul_rn(kdx, d)), sd = warp_sum(mul_rn(d, d));
          if (lane == 0) {
            term[warp] = (double)si;
            term[kTerms + warp] = (double)sd;
          }
        }
      }
    }
    __syncthreads();
    // the plan CTAs' sums, as cta_sums adds them, one per warp; each to every CTA
    for (int task = warp; task < 3 * kClusterRounds && warp < kBlock / 32; task += kBlock / 32) {
      const int q = task % 3, b = rank + task / 3 * size;
      if (b >= (q == 2 ? np : nd)) continue;
      const double* term = terms + task * kTerms;
      double sum;
      if constexpr (sizeof(T) == 8) {
        sum = term[lane];
#pragma unroll
        for (int v = 1; v < kBlock / 32; ++v) sum += term[32 * v + lane];
        sum = warp_sum(sum);
      } else {
        sum = term[0];
#pragma unroll
        for (int v = 1; v < kBlock / 32; ++v) sum += term[v];
      }
      sum = __shfl_sync(0xffffffffu, sum, 0);
      if (lane < size) remote_store(remote_address(&part[q][b], lane), sum);
    }
    cluster_barrier();
    // the totals, as step_totals adds them, and the decision: the same in every CTA
    if (warp < 3) {
      const int count = warp == 2 ? np : nd;
      double sum = lane < count ? part[warp][lane] : 0.0;
      for (int v = 32 + lane; v < count; v += 32) sum += part[warp][v];
      sum = warp_sum(sum);
      if (lane == 0) {
        if (warp > 0) {
          const double norm = sqrt(sum);
          sum = warp == 1 ? norm : __dmul_rn(__dmul_rn(0.5 * s.omega, norm), norm);
        }
        total[warp] = sum;
      }
    }
    __syncthreads();
    if (decides) {
      verdict = step_verdict(s, factors[0], factors[1], total[0],
                             __fma_rn(__dmul_rn(s.half_over_omega, total[1]), total[1], total[2]));
      pending_before = pending;
      now.pending = verdict.accept ? 1 : 0;
      if (verdict.accept) {
        now.parity = p ^ 1;
        now.w = s.iter_start_tau;
      }
      now.done = verdict.error || s.accepted_in_chunk + now.pending >= s.target_in_chunk ||
                 s.attempts_in_chunk + 1 >= s.max_attempts_in_chunk;
    }
    __syncthreads();
    if (now.done) break;
  }
  if (decides) account(pending_before);
  __syncthreads();
  if (rank == 0) {
    store_state(s, da.st_mut);
  }
}

inline void cluster_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int ctas, int size, size_t shared,
                           cudaStream_t s) {
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(kClusterThreads);
  cfg.dynamicSmemBytes = shared;
  cfg.stream = s;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)size;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
}

// How an LP's intervals run on a cluster: its CTAs (0: they run as graphs of the step kernels).
template <class T>
struct ClusterPlan {
  int size = 0, cols = 0, rows = 0;
  size_t shared = 0;
  DBuf<int32_t> p_slot, d_slot;   // first slot of each plan CTA (CTAs + 1)
};

// First slot of every plan CTA (CTAs + 1).
template <class T>
std::vector<int32_t> cta_slots(const TilePlan<T>& plan) {
  std::vector<int32_t> v;
  v.reserve(plan.cta_tile.size());
  for (int32_t q : plan.cta_tile) v.push_back(plan.tile_slot[(size_t)q]);
  return v;
}

// Fills plan when the lone LP with tile plans p and d qualifies: all tiles summed by one warp each and
// at most one per warp of a plan CTA, at most kClusterRounds plan CTAs per cluster CTA and side, a
// CTA's share within shared memory, and a device that runs such a cluster.
template <class T>
void plan_cluster(ClusterPlan<T>& plan, const TilePlan<T>& p, const TilePlan<T>& d, int n, int m, cudaStream_t s) {
  if (!p.warp_tiles_only || !d.warp_tiles_only || std::max(p.num_ctas, d.num_ctas) > kClusterPlanCtas) return;
  for (const TilePlan<T>* t : {&p, &d})
    for (int b = 0; b < t->num_ctas; ++b)
      if (t->cta_tile[(size_t)b + 1] - t->cta_tile[(size_t)b] > kClusterTiles) return;
  const std::vector<int32_t> ps = cta_slots(p), ds = cta_slots(d);
  const int size = std::min(kClusterMax, std::max(p.num_ctas, d.num_ctas));
  size_t shared = 0;
  for (int r = 0; r < size; ++r) {
    size_t bytes = cluster_vector_bytes<T>(n, m) + sizeof(double) * kClusterRounds * 3 * kClusterTerms<T>;
    for (int b = r; b < p.num_ctas; b += size) bytes += cluster_side_bytes(ps[(size_t)b + 1] - ps[(size_t)b], sizeof(T));
    for (int b = r; b < d.num_ctas; b += size) bytes += cluster_side_bytes(ds[(size_t)b + 1] - ds[(size_t)b], sizeof(T));
    shared = std::max(shared, bytes);
  }
  if (shared > kClusterShared) return;
  CK(cudaFuncSetAttribute(cluster_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClusterShared));
  CK(cudaFuncSetAttribute(cluster_kernel<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cluster_config(cfg, attr, size, size, shared, s);
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, cluster_kernel<T>, &cfg) != cudaSuccess || clusters < 1) {
    cudaGetLastError();
    return;
  }
  plan.size = size;
  plan.shared = shared;
  auto up = [&](auto& buf, const auto* src, size_t count) {
    buf.alloc(count);
    CK(cudaMemcpyAsync(buf.get(), src, sizeof(*src) * count, cudaMemcpyHostToDevice, s));
  };
  up(plan.p_slot, ps.data(), ps.size());
  up(plan.d_slot, ds.data(), ds.size());
  plan.cols = n;
  plan.rows = m;
  CK(cudaStreamSynchronize(s));   // the host arrays die here
}

template <class T>
void launch_cluster(const ClusterPlan<T>& plan, cudaStream_t s, const PrimalArgs<T>& pa, const DualArgs<T>& da) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cluster_config(cfg, attr, plan.size, plan.size, plan.shared, s);
  CK(cudaLaunchKernelEx(&cfg, cluster_kernel<T>, pa, da, (const int32_t*)plan.p_slot.get(),
                        (const int32_t*)plan.d_slot.get(), plan.cols, plan.rows));
}

}  // namespace gpdhg
