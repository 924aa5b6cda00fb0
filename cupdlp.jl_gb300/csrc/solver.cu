// solver.cu — the restarted PDHG loop of optimize() on one GPU.
//
// Host/device split (src/primal_dual_hybrid_gradient_gpu.jl:457-798):
//   * step attempts run as CUDA graphs of [primal_step_kernel, dual_step_kernel] pairs, a
//     small LP's as one cluster_kernel; accept/reject and the step size live on the device
//     (StepState);
//   * evaluations (every termination_evaluation_frequency iterations, the first 10,
//     and on a numerical error) are a graph of FP64 reduction kernels queued behind the
//     steps, so a whole evaluation interval (64 accepted steps) needs one host
//     synchronisation (again after rejected attempts) instead of ~5 per attempt; the host
//     reads ~40 scalars, and the termination test, restart scheme and primal-weight update
//     are the reference's scalar logic there;
//   * with GPDHG_PRECISION_FP32_REFINE the loop runs on FP32 copies of the matrix and
//     iterates until the relative KKT error reaches fp64_handoff_relative_kkt (or stalls),
//     then converts the state to FP64, recomputes K x and K'y exactly, and continues.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <memory>
#include <mutex>
#include <exception>
#include <thread>
#include <limits>
#include <random>
#include <type_traits>
#include <vector>

#include "batch.h"
#include "batch_kernels.cuh"
#include "tiles.h"
#include "eval_kernels.cuh"
#include "host_logic.h"
#include "problem.h"
#include "spmv.cuh"
#include "cluster_solve.cuh"

namespace gpdhg {

void launch_convert_d2f(const double* src, float* dst, long long n, cudaStream_t s) {
  const int grid = std::max(1, std::min(ceil_div(n, kBlock), 4096));
  convert_kernel<double, float><<<grid, kBlock, 0, s>>>(n, src, dst);
  CK_LAUNCH();
}

__global__ void reciprocal_kernel(long long len, const double* src, double* dst) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (long long)gridDim.x * blockDim.x)
    dst[i] = 1.0 / src[i];
}

void launch_reciprocal(const double* src, double* dst, long long n, cudaStream_t s) {
  if (n <= 0) return;
  const int grid = std::max(1, std::min(ceil_div(n, kBlock), 4096));
  reciprocal_kernel<<<grid, kBlock, 0, s>>>(n, src, dst);
  CK_LAUNCH();
}

template <class T>
struct DotF {
  const T* a;
  const T* b;
  struct Params {
    __device__ Params(const StepState*, int) {}
  };
  struct In {
    T a, b;
  };
  __device__ __forceinline__ void load(const Params&, int i, In& v) const { v = In{a[i], b[i]}; }
  __device__ __forceinline__ void apply(const Params&, int, const In& v, double* acc) const {
    acc[0] += (double)v.a * (double)v.b;
  }
};

// Step graphs hold 1, 2, 4, ..., 64 [primal, dual] pairs; a chunk launches the smallest one
// that covers the accepted steps still missing, so finished chunks waste almost no launches.
constexpr int kGraphLevels = 7;
inline int graph_level(int remaining) {
  int lv = 0;
  while (lv + 1 < kGraphLevels && (1 << lv) < remaining) ++lv;
  return lv;
}
// Host table of the step-size factors (1 - (k+1)^-r, 1 + (k+1)^-g) of take_step!
// (:405-407): the device reads it instead of evaluating two FP64 pow() per attempt in one
// thread, and the values are the host libm's, as in the reference's host-side loop.
// The table of an exponent pair is computed once per process (on host threads, each entry
// by the same libm call whatever the thread) and kept for later problems.
void fill_pow_table(std::vector<double>& t, double r, double g) {
  static std::mutex mu;
  static std::vector<std::pair<std::pair<double, double>, std::shared_ptr<const std::vector<double>>>> cache;
  std::shared_ptr<const std::vector<double>> hit;
  {
    std::lock_guard<std::mutex> lock(mu);
    for (auto& e : cache)
      if (e.first.first == r && e.first.second == g) hit = e.second;
  }
  if (!hit) {
    auto v = std::make_shared<std::vector<double>>(2 * kPowTableLen);
    const int T = (int)std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
    std::vector<std::thread> th;
    for (int q = 0; q < T; ++q)
      th.emplace_back([&, q] {
        for (long long k = kPowTableLen * q / T; k < kPowTableLen * (q + 1) / T; ++k) {
          const double k1 = (double)(k + 1);
          (*v)[2 * k] = 1.0 - 1.0 / std::pow(k1, r);
          (*v)[2 * k + 1] = 1.0 + 1.0 / std::pow(k1, g);
        }
      });
    for (auto& x : th) x.join();
    std::lock_guard<std::mutex> lock(mu);
    if (cache.size() >= 8) cache.erase(cache.begin());
    cache.push_back({{r, g}, v});
    hit = v;
  }
  t = *hit;
}

template <class T>
struct Workspace {
  gpdhg_problem* P = nullptr;
  int n = 0, m = 0;
  DBuf<T> l_own, u_own, c_own, b_own;
  const T *l = nullptr, *u = nullptr, *c = nullptr, *b = nullptr;
  DBuf<T> x, dx, kty, sx, ax, agrad, grad, rx, rgrad, tmp_n;
  DBuf<T> y0, y1, kx0, kx1, sy, skx, ay, akx, ry, rkx, tmp_m;
  DBuf<StepState> st_dev;
  PinnedBuf<StepState> st_host;
  DBuf<double> part_p, part_d, red_part_n, red_part_m;
  DBuf<double> rvar, rcon;   // 1 / variable and 1 / constraint rescaling (evaluation divisions)
  PinnedBuf<double> red_host;
  RestartKkt restart_kkt;
  // segmented reductions over [0, n) and [0, m): the same layout a batch uses per instance
  DBuf<SegItem> seg_n, seg_m;
  DBuf<int32_t> seg_n_begin, seg_m_begin;
  int nseg_n = 1, nseg_m = 1;
  ClusterPlan<T> cluster;   // a small LP's intervals run on one cluster instead of as step graphs
  cudaGraphExec_t graphs[kGraphLevels] = {}, evaluation = nullptr;
  // profiled solves (params.profile_kernels): an event between every two step kernels, and the evaluation
  // behind steps that were launched one by one
  std::vector<cudaEvent_t> pev;
  cudaGraphExec_t profiled_evaluation = nullptr;
  // A solution in FP64 and the caller's order on its way to the host: FP32 needs room of its own, laid out
  // with the workspace; FP64 columns take tmp_n, which nothing needs after an evaluation.
  DBuf<double> caller;
  double* caller_buffer() {
    if constexpr (sizeof(T) == sizeof(double)) return tmp_n.get();
    else return caller.get();
  }
  DBuf<double> pow_table;
  double pow_r = -1.0, pow_g = -1.0;
  const int direct = sizeof(T) == sizeof(float) ? 1 : 0;
  // tile plans of A' (primal kernel) and A (dual kernel); the lone LP is a batch of one
  TilePlan<T> plan_p, plan_d;
  DBuf<double> part_p_split, part_d_split;

  explicit Workspace(gpdhg_problem* p) : P(p), n(p->n), m(p->m), st_host(1), red_host(kEvalStride) {
    PhaseTrace tr;
    const size_t N = std::max(n, 1), M = std::max(m, 1);
    cudaStream_t s = P->stream;
    if constexpr (sizeof(T) == sizeof(double)) {
      l = (const T*)P->l.get();
      u = (const T*)P->u.get();
      c = (const T*)P->c.get();
      b = (const T*)P->b.get();
    } else {
      ensure_fp32_values(P);
      l_own.alloc(N); u_own.alloc(N); c_own.alloc(N); b_own.alloc(M);
      launch_convert_d2f(P->l.get(), l_own.get(), n, s);
      launch_convert_d2f(P->u.get(), u_own.get(), n, s);
      launch_convert_d2f(P->c.get(), c_own.get(), n, s);
      if (m) launch_convert_d2f(P->b.get(), b_own.get(), m, s);
      l = l_own.get(); u = u_own.get(); c = c_own.get(); b = b_own.get();
    }
    tr.mark("  ws: FP32 copies");
    // the primal plan (a host pass over the n rows of A') is built on a helper thread while
    // this one allocates the iterate vectors and builds the dual plan
    std::exception_ptr plan_err;
    int device = 0;
    CK(cudaGetDevice(&device));
    std::thread plan_thread([&] {
      try {
        CK(cudaSetDevice(device));   // a new host thread starts on device 0
        build_tile_plan(plan_p, P->At, {0, n}, {}, kPrimalCtasPerSm<T>, kTileSideAt, s);
      } catch (...) {
        plan_err = std::current_exception();
      }
    });
    try {
      for (DBuf<T>* v : {&x, &dx, &kty, &sx, &ax, &agrad, &grad, &rx, &rgrad, &tmp_n}) v->alloc(N);
      for (DBuf<T>* v : {&y0, &y1, &kx0, &kx1, &sy, &skx, &ay, &akx, &ry, &rkx, &tmp_m}) v->alloc(M);
      rvar.alloc(N);
      rcon.alloc(M);
      launch_reciprocal(P->var.get(), rvar.get(), n, s);
      launch_reciprocal(P->con.get(), rcon.get(), m, s);
      st_dev.alloc(1);
      CK(cudaMemsetAsync(st_dev.get(), 0, sizeof(StepState), s));
      tr.mark("  ws: iterate buffers");
      build_tile_plan(plan_d, P->A, {0, m}, {P->neq}, kDualCtasPerSm, kTileSideA, s);
      tr.mark("  ws: dual plan");
    } catch (...) {
      plan_thread.join();
      throw;
    }
    plan_thread.join();
    if (plan_err) std::rethrow_exception(plan_err);
    tr.mark(sizeof(T) == 8 ? "FP64 vectors and plans" : "FP32 vectors and plans");
    part_p.alloc(plan_p.num_ctas);
    part_d.alloc(2 * (size_t)plan_d.num_ctas);
    part_p_split.alloc(std::max(plan_p.num_splits, 1));
    part_d_split.alloc(2 * (size_t)std::max(plan_d.num_splits, 1));
    {
      std::vector<SegItem> it;
      std::vector<int32_t> beg;
      auto upload = [&](DBuf<SegItem>& d, DBuf<int32_t>& db, int len, int& count) {
        build_seg_items({0, len}, it, beg);
        count = (int)it.size();
        d.alloc(it.size());
        db.alloc(beg.size());
        CK(cudaMemcpyAsync(d.get(), it.data(), sizeof(SegItem) * it.size(), cudaMemcpyHostToDevice, s));
        CK(cudaMemcpyAsync(db.get(), beg.data(), sizeof(int32_t) * beg.size(), cudaMemcpyHostToDevice, s));
        CK(cudaStreamSynchronize(s));
      };
      upload(seg_n, seg_n_begin, n, nseg_n);
      upload(seg_m, seg_m_begin, m, nseg_m);
      red_part_n.alloc((size_t)kPassNQ * nseg_n);
      red_part_m.alloc((size_t)kPassMQ * nseg_m);
    }
    if (sizeof(T) == sizeof(float)) caller.alloc(std::max(N, M));
    tr.mark("segments, partials");
    build_graphs();
    tr.mark("step graphs");
  }
  ~Workspace() {
    for (cudaGraphExec_t g : graphs)
      if (g) cudaGraphExecDestroy(g);
    if (evaluation) cudaGraphExecDestroy(evaluation);
    if (profiled_evaluation) cudaGraphExecDestroy(profiled_evaluation);
    for (cudaEvent_t e : pev) cudaEventDestroy(e);
  }

  const T* ycur(int parity) const { return parity ? y1.get() : y0.get(); }
  const T* kxcur(int parity) const { return parity ? kx1.get() : kx0.get(); }

  PrimalArgs<T> primal_args(int mode) {
    return PrimalArgs<T>{P->At.view<T>(), plan_p.view(), c, l, u, x.get(), dx.get(), kty.get(), sx.get(),
                         y0.get(), y1.get(), st_dev.get(), part_p.get(), part_p_split.get(), mode, direct};
  }
  DualArgs<T> dual_args() {
    return DualArgs<T>{P->A.view<T>(), plan_d.view(), plan_p.inst_cta_begin.get(), plan_p.inst_split_begin.get(),
                       dx.get(), b, y0.get(), y1.get(), kx0.get(), kx1.get(), sy.get(), skx.get(), st_dev.get(),
                       part_p.get(), part_p_split.get(), part_d.get(), part_d_split.get(), direct};
  }
  void launch_primal(int mode, cudaStream_t s) { launch_step(primal_kernel<T>(plan_p.num_ctas), plan_p.num_ctas, s, primal_args(mode)); }
  void launch_dual(cudaStream_t s) { launch_step(dual_kernel<T>(plan_d.num_ctas), plan_d.num_ctas, s, dual_args()); }

  // An interval as a graph: the state to the device (unless it is there already), `pairs` step attempts
  // (the cluster kernel's, if the LP runs on one: as many as the interval takes), then its
  // evaluation. pairs 0: the evaluation alone. (Launches of their own stand 4-5 us apart.)
  cudaGraphExec_t capture(int pairs, bool with_state = true) {
    cudaStream_t s = P->stream;
    GraphCapture g(s);
    if (with_state) copy_state(st_host.p, st_dev.get(), 1, s);
    if (pairs && cluster.size) {
      launch_cluster(cluster, s, primal_args(kStepNormal), dual_args());
    } else {
      for (int k = 0; k < pairs; ++k) {
        launch_primal(kStepNormal, s);
        launch_dual(s);
      }
    }
    record_evaluation(g);
    return g.finish();
  }
  void build_graphs() {
    plan_cluster(cluster, plan_p, plan_d, n, m, P->stream);
    evaluation = capture(0);
  }
  // The graph of 2^lv pairs, captured at its first use: a solve needs two or three of the levels (one
  // if it runs on a cluster).
  cudaGraphExec_t step_graph(int lv) {
    if (!graphs[lv]) graphs[lv] = capture(1 << lv);
    return graphs[lv];
  }
  // The same interval with its pairs launched one by one and an event between every two kernels, for
  // per-kernel CUDA-event timing (events recorded as graph nodes cannot be timed).
  void launch_profiled(int pairs) {
    cudaStream_t s = P->stream;
    if (!profiled_evaluation) profiled_evaluation = capture(0, false);
    while ((int)pev.size() < 2 * pairs + 1) {
      cudaEvent_t e = nullptr;
      CK(cudaEventCreate(&e));
      pev.push_back(e);
    }
    copy_state(st_host.p, st_dev.get(), 1, s);
    CK(cudaEventRecord(pev[0], s));
    for (int k = 0; k < pairs; ++k) {
      launch_primal(kStepNormal, s);
      CK(cudaEventRecord(pev[2 * k + 1], s));
      launch_dual(s);
      CK(cudaEventRecord(pev[2 * k + 2], s));
    }
    CK_LAUNCH();
    CK(cudaGraphLaunch(profiled_evaluation, s));
    P->launches += 1 + 2 * pairs + kEvaluationKernels;
  }
  const double* ensure_pow_table(double r, double g) {
    if (pow_table.get() && r == pow_r && g == pow_g) return pow_table.get();
    std::vector<double> t;
    fill_pow_table(t, r, g);
    pow_table.alloc(t.size());
    CK(cudaMemcpyAsync(pow_table.get(), t.data(), sizeof(double) * t.size(), cudaMemcpyHostToDevice, P->stream));
    CK(cudaStreamSynchronize(P->stream));
    pow_r = r;
    pow_g = g;
    return pow_table.get();
  }

  // st: as recorded into an evaluation's graph, whose launch counts its kernels (as for the reductions)
  void spmv(const DeviceMatrix& M, const T* xin, T* yout, const StepState* st = nullptr) {
    if (M.num_items == 0) return;
    spmv_kernel<T><<<M.num_items, kBlock, 0, P->stream>>>(M.view<T>(), xin, yout, nullptr, st);
    CK_LAUNCH();
    if (!st) ++P->launches;
  }

  // one side's pass over its segments into its partials
  template <int Q, unsigned MAXMASK, class F>
  void reduce(bool n_side, const F& f, const StepState* st) {
    launch_reduce<Q, MAXMASK>(n_side ? seg_n.get() : seg_m.get(), st, f, n_side ? red_part_n.get() : red_part_m.get(),
                              n_side ? nseg_n : nseg_m, P->stream);
  }
  SegSide side(bool n_side, int quantities, unsigned maxmask) {
    return SegSide{n_side ? seg_n_begin.get() : seg_m_begin.get(), n_side ? red_part_n.get() : red_part_m.get(),
                   red_host.p + (n_side ? kEvalOutN : 0), n_side ? nseg_n : nseg_m, quantities, maxmask};
  }
  // the partials of both sides reduced (a side without quantities is skipped), into red_host
  void finish_reductions(SegSide a, SegSide b, const StepState* st) {
    seg_finalize_kernel<<<dim3(1, a.quantities + b.quantities), kBlock, 0, P->stream>>>(a, b, st, st ? st_host.p : nullptr);
    CK_LAUNCH();
  }
  // One evaluation, recorded into a graph; it also returns the state: the row pass (the last accepted step's
  // Sigma y and Sigma Kx, the averages y-bar and Kx-bar with their unscaled statistics,
  // src/iteration_stats_utils_gpu.jl:447-502, and restart-scheme ingredients), launched first since it
  // is on the path, and that step's K'y, x and Sigma x beside it; A' y-bar (the reference sums the
  // steps' K'y with the averaging weights instead, src/saddle_point_gpu.jl:176-189; the two agree in
  // exact arithmetic); then the column pass and all sums. It stands right behind the steps of its
  // interval, whose last decision sets what it needs (end_chunk); behind steps that end short of the
  // interval's goal it does nothing. (Launched by the host after reading the state, an interval took 12
  // us more, two round trips instead of one.)
  static constexpr int kEvaluationKernels = 5;
  void record_evaluation(GraphCapture& g) {
    cudaStream_t s = P->stream;
    CK(cudaEventRecord(g.fork, s));
    reduce<kPassMQ, kEvalMMax>(
        false,
        EvalPassM<T>{P->con.get(), rcon.get(), P->ob.get(), b, y0.get(), y1.get(), kx0.get(), kx1.get(), ry.get(),
                     rkx.get(), sy.get(), skx.get(), ay.get(), akx.get(), P->neq, nullptr},
        st_dev.get());
    CK(cudaStreamWaitEvent(g.side, g.fork, 0));
    primal_kernel<T>(plan_p.num_ctas)<<<plan_p.num_ctas, kBlock, 0, g.side>>>(primal_args(kStepCommitOnly));
    CK_LAUNCH();
    CK(cudaEventRecord(g.join, g.side));
    spmv(P->At, ay.get(), tmp_n.get(), st_dev.get());
    CK(cudaStreamWaitEvent(s, g.join, 0));
    reduce<kPassNQ, kEvalNMax>(
        true,
        EvalPassN<T>{P->var.get(), rvar.get(), P->ol.get(), P->ou.get(), P->oc.get(), l, u, c, x.get(), sx.get(),
                     tmp_n.get(), kty.get(), rx.get(), rgrad.get(), ax.get(), agrad.get(), grad.get()},
        st_dev.get());
    finish_reductions(side(false, kPassMQ, kEvalMMax), side(true, kPassNQ, kEvalNMax), st_dev.get());
  }
  void launch_restart(cudaStream_t s) {
    const RestartArgs<T> a{st_dev.get(), nullptr, nullptr, n, m, c, ax.get(), agrad.get(), ay.get(), akx.get(),
                           x.get(), kty.get(), grad.get(), sx.get(), rx.get(), rgrad.get(), y0.get(), y1.get(),
                           kx0.get(), kx1.get(), sy.get(), skx.get(), ry.get(), rkx.get()};
    restart_kernel<T><<<grid_for(std::max(n, m)), kBlock, 0, s>>>(a);
    CK_LAUNCH();
    ++P->launches;
  }

  double dot(const T* a, const T* b2, long long len) {
    const bool n_side = len == n;
    reduce<1, 0u>(n_side, DotF<T>{a, b2}, nullptr);
    finish_reductions(side(n_side, 1, 0u), SegSide{}, nullptr);
    P->launches += 2;
    CK(cudaStreamSynchronize(P->stream));
    return red_host.p[n_side ? kEvalOutN : 0];
  }

  int grid_for(long long len) const { return std::max(1, std::min(ceil_div(len, kBlock), 4096)); }
};

}  // namespace gpdhg

void gpdhg::WorkspaceDeleter::operator()(Workspace<double>* w) const { delete w; }
void gpdhg::WorkspaceDeleter::operator()(Workspace<float>* w) const { delete w; }

gpdhg_problem::~gpdhg_problem() {
  ws64.reset();
  ws32.reset();
  if (stream) cudaStreamDestroy(stream);
}

namespace gpdhg {

namespace {

using Clock = std::chrono::steady_clock;

// Host scalar state of the loop that is not part of StepState.
struct LoopState {
  long long iteration = 0;   // the reference's `iteration` (accepted steps + 1)
  double basic_time = 0.0;   // time_spent_doing_basic_algorithm
  Clock::time_point t0;
  RestartMemory restart;      // CuRestartInfo scalars
  double step_loop_sec = 0.0;
  double primal_kernel_sec = 0.0, dual_kernel_sec = 0.0;
  long long kernel_launches = 0;
  long long launches_at_start = 0;
  int precision = GPDHG_PRECISION_FP64;
  int handoff_iteration = -1;
  double best_rel_kkt = std::numeric_limits<double>::infinity();
  int evals_without_progress = 0;
  double elapsed() const { return std::chrono::duration<double>(Clock::now() - t0).count(); }
};

// The loop in one precision. Returns true when it terminated, false on an FP64 hand-off
// request (state left in W for the caller to convert).
template <class T>
bool run_phase(gpdhg_problem* P, Workspace<T>& W, const gpdhg_params& prm, LoopState& L, gpdhg_result* res,
               double* primal_out, double* dual_out, bool allow_handoff) {
  cudaStream_t s = P->stream;
  StepState& st = *W.st_host.p;
  const long long freq = std::max(1, prm.termination_evaluation_frequency);
  const long long it_limit = prm.iteration_limit;
  const int n = P->n, m = P->m;
  InstanceInfo qi;
  qi.obj_const = P->obj_const;
  qi.linf_c = P->linf_c; qi.linf_b = P->linf_b; qi.l2_c = P->l2_c; qi.l2_b = P->l2_b;

  // The state to the device. The mirror stays untouched until the stream has passed the copy: the
  // host edits it only after synchronising with the work that follows.
  auto push_state_async = [&]() {
    copy_state(W.st_host.p, W.st_dev.get(), 1, s);
    ++P->launches;
  };

  auto launch_evaluation = [&]() {
    CK(cudaGraphLaunch(W.evaluation, s));
    P->launches += 1 + W.kEvaluationKernels;
  };
  bool evaluated = false;   // an evaluation of this iteration ran behind its steps

  while (true) {
    const long long it = L.iteration;
    if (eval_due(it, freq, it_limit, st.numerical_error != 0)) {
      if (!evaluated) {   // not behind steps: at the start, and again in FP64 after a hand-off
        // the average, or the current point (src/primal_dual_hybrid_gradient_gpu.jl:635-642)
        st.eval_active = 1;
        st.eval_current = (st.numerical_error || st.count_primal == 0 || st.count_dual == 0) ? 1 : 0;
        st.eval_restart = W.restart_kkt.valid ? 0 : 1;
        st.rcp_w_primal = st.eval_current ? 0.0 : 1.0 / st.sum_w_primal;
        st.rcp_w_dual = st.eval_current ? 0.0 : 1.0 / st.sum_w_dual;
        launch_evaluation();
        CK(cudaStreamSynchronize(s));
      }
      evaluated = false;
      st.kkt_passes += 2.0;  // KKT_PASSES_PER_TERMINATION_EVALUATION
      st.done = 0;
      st.restart = kNoRestart;
      st.pending_commit = 0;
      const double* em = W.red_host.p;               // kM_*, then the rows' KKT ingredients
      const double* en = W.red_host.p + kEvalOutN;   // kN_*, then the columns'
      double kn[kKktNQ], km[kKktMQ];
      std::memcpy(kn, en + kEvalNQ, sizeof(kn));
      std::memcpy(km, em + kEvalMQ, sizeof(km));
      W.restart_kkt.keep_or_fill(kn, km);
      gpdhg_iteration_stats stats;
      std::memset(&stats, 0, sizeof(stats));
      assemble_stats(qi, prm, en, em, stats);
      stats.iteration_number = (int32_t)(it - 1);
      stats.cumulative_kkt_matrix_passes = st.kkt_passes;
      stats.cumulative_time_sec = L.elapsed();
      stats.step_size = st.tau;
      stats.primal_weight = st.omega;
      stats.precision = L.precision;
      stats.time_spent_doing_basic_algorithm = L.basic_time;
      int reason = check_termination(prm, qi, stats);
      if (st.numerical_error && reason == 0) reason = GPDHG_TERMINATION_REASON_NUMERICAL_ERROR;
      if (it < 10 && (reason == GPDHG_TERMINATION_REASON_PRIMAL_INFEASIBLE ||
                      reason == GPDHG_TERMINATION_REASON_DUAL_INFEASIBLE))
        reason = 0;
      bool pushed = false;
      if (prm.record_iteration_stats || reason != 0) {
        P->history.push_back(stats);
        pushed = true;
      }
      if (reason != 0) {
        // copy the scaled average to the host (:713-720)
        auto fetch = [&](const T* dsrc, const int32_t* perm, double* hdst, int len) {
          if (!hdst || len == 0) return;
          const double* src = reinterpret_cast<const double*>(dsrc);
          if (sizeof(T) == 4 || perm) {
            caller_values_kernel<T><<<W.grid_for(len), kBlock, 0, s>>>(len, dsrc, perm, W.caller_buffer());
            CK_LAUNCH();
            ++P->launches;
            src = W.caller_buffer();
          }
          CK(cudaMemcpyAsync(hdst, src, sizeof(double) * len, cudaMemcpyDeviceToHost, s));
        };
        fetch(W.ax.get(), P->col_perm_dev.get(), primal_out, n);
        fetch(W.ay.get(), nullptr, dual_out, m);
        CK(cudaStreamSynchronize(s));
        std::memset(res, 0, sizeof(*res));
        res->termination_reason = reason;
        res->iteration_count = (int32_t)(it - 1);
        res->total_number_iterations = st.total_iters;
        res->cumulative_kkt_matrix_passes = st.kkt_passes;
        res->solve_time_sec = L.elapsed();
        res->num_iteration_stats = (int32_t)P->history.size();
        res->fp64_handoff_iteration = L.handoff_iteration;
        res->last_iteration_stats = stats;
        res->step_loop_device_sec = L.step_loop_sec;
        res->accepted_steps = st.accepted;
        res->rejected_steps = st.rejected;
        res->primal_kernel_sec = L.primal_kernel_sec;
        res->dual_kernel_sec = L.dual_kernel_sec;
        res->primal_kernel_launches = L.kernel_launches;
        res->primal_spmv_launches = st.primal_spmv;
        res->kernels_launched = P->launches - L.launches_at_start;
        P->last_precision = (sizeof(T) == sizeof(double)) ? GPDHG_PRECISION_FP64 : GPDHG_PRECISION_FP32;
        return true;
      }
      // FP64 hand-off check (FP32_REFINE)
      if (allow_handoff) {
        const double rk = relative_kkt(stats, prm.optimality_norm);
        if (rk < 0.5 * L.best_rel_kkt) {
          L.best_rel_kkt = rk;
          L.evals_without_progress = 0;
        } else {
          L.evals_without_progress++;
        }
        if (rk <= prm.fp64_handoff_relative_kkt ||
            (prm.fp64_handoff_stall_evaluations > 0 && L.evals_without_progress >= prm.fp64_handoff_stall_evaluations)) {
          // leave the evaluation to be repeated by the FP64 phase at the same iteration
          st.kkt_passes -= 2.0;
          if (pushed) P->history.pop_back();
          return false;
        }
      }
      // run_restart_scheme, src/saddle_point_gpu.jl:479-622 (buffer_primal_gradient was
      // refreshed by the column pass)
      int restart_used = GPDHG_RESTART_CHOICE_NO_RESTART;
      if (st.count_primal > 0 && st.count_dual > 0) {
        const RestartDecision dec =
            decide_restart(prm, qi, st.count_primal, st.tau, st.omega, it - 1, kn, km, L.restart);
        if (dec.restart_used != GPDHG_RESTART_CHOICE_NO_RESTART) {
          // the vectors follow in restart_kernel, after the state that it reads
          st.restart = dec.reset_to_average ? kRestartToAverage : kRestartFromCurrent;
          W.restart_kkt.valid = false;  // the restart point moves
          st.count_primal = st.count_dual = 0;
          st.sum_w_primal = st.sum_w_dual = 0.0;
          st.omega = dec.new_omega;
          restart_used = dec.restart_used;
        }
      }
      if (pushed) P->history.back().restart_used = restart_used;
    }

    // take_step! calls until the next evaluation
    const long long target = next_eval_after(it, freq, it_limit) - it;
    st.done = 0;
    st.target_in_chunk = (int)std::min<long long>(target, 1 << 30);
    st.accepted_in_chunk = 0;
    st.attempts_in_chunk = 0;
    st.max_attempts_in_chunk = 1 << 30;
    st.iter_start_tau = st.tau;
    st.half_over_omega = 0.5 / st.omega;
    st.tto = st.tau / st.omega;
    st.arrive = 0;
    st.eval_active = 0;
    st.eval_restart = W.restart_kkt.valid ? 0 : 1;
    const bool prof = prm.profile_kernels != 0, on_cluster = W.cluster.size && !prof;
    auto next_level = [&]() {   // of the next launch's step attempts
      const int lv = graph_level(st.target_in_chunk - st.accepted_in_chunk);
      st.launch_attempts = st.attempts_in_chunk + (on_cluster ? kClusterAttempts : 1 << lv);
      return lv;
    };
    int lv = next_level();
    if (st.restart != kNoRestart) {   // it reads the state ahead of the interval's graph
      push_state_async();
      W.launch_restart(s);
    }
    long long launches = 0;
    const auto tb = Clock::now();
    while (true) {
      const int attempts_before = st.attempts_in_chunk;
      if (prof) {
        W.launch_profiled(1 << lv);
      } else {
        CK(cudaGraphLaunch(W.step_graph(on_cluster ? 0 : lv), s));
        P->launches += 1 + (on_cluster ? 1 : 2 * (1 << lv)) + W.kEvaluationKernels;
      }
      CK(cudaStreamSynchronize(s));
      L.step_loop_sec += 1e-9 * (double)st.launch_ns;
      if (prof) {
        const std::vector<cudaEvent_t>& ev = W.pev;
        const int did = st.attempts_in_chunk - attempts_before;
        for (int k = 0; k < did; ++k) {
          float a = 0.f, b2 = 0.f;
          CK(cudaEventElapsedTime(&a, ev[2 * k], ev[2 * k + 1]));
          CK(cudaEventElapsedTime(&b2, ev[2 * k + 1], ev[2 * k + 2]));
          L.primal_kernel_sec += 1e-3 * a;
          L.dual_kernel_sec += 1e-3 * b2;
        }
        L.kernel_launches += did;
      }
      if (st.done) break;
      // every launch runs an attempt at least; 10^6 launches without the chunk's
      // accepted steps means the step size never settles
      if (++launches > 1000000) throw Error(GPDHG_ERR_INTERNAL, "step chunk did not finish");
      lv = next_level();
    }
    evaluated = true;
    // wall clock of the steps, as the reference takes it: the evaluation's part is not theirs
    L.basic_time += std::chrono::duration<double>(Clock::now() - tb).count() - W.red_host.p[kEvalSpan];
    L.iteration += st.accepted_in_chunk + (st.numerical_error ? 1 : 0);
  }
}

// Initial state of optimize() (:494-611) in workspace W.
template <class T>
void init_state(gpdhg_problem* P, Workspace<T>& W, const gpdhg_params& prm, LoopState& L) {
  cudaStream_t s = P->stream;
  const int n = P->n, m = P->m;
  for (DBuf<T>* v : {&W.x, &W.kty, &W.sx, &W.dx, &W.ax, &W.agrad})
    CK(cudaMemsetAsync(v->get(), 0, sizeof(T) * v->n, s));
  for (DBuf<T>* v : {&W.y0, &W.y1, &W.kx0, &W.kx1, &W.sy, &W.skx, &W.ay, &W.akx})
    CK(cudaMemsetAsync(v->get(), 0, sizeof(T) * v->n, s));
  if (!P->warm_x.empty() || !P->warm_y.empty()) {
    auto upload = [&](const std::vector<double>& h, T* d, int len) {
      if (h.empty() || len == 0) return;
      std::vector<T> tmp(h.begin(), h.end());
      CK(cudaMemcpyAsync(d, tmp.data(), sizeof(T) * len, cudaMemcpyHostToDevice, s));
      CK(cudaStreamSynchronize(s));
    };
    upload(P->warm_x, W.x.get(), n);
    upload(P->warm_y, W.y0.get(), m);
    W.spmv(P->A, W.x.get(), W.kx0.get());
    W.spmv(P->At, W.y0.get(), W.kty.get());
  }
  const int gn = W.grid_for(n);
  grad_kernel<T><<<gn, kBlock, 0, s>>>(n, W.c, W.kty.get(), W.grad.get());
  CK_LAUNCH();
  ++P->launches;
  StepState& st = *W.st_host.p;
  std::memset(&st, 0, sizeof(st));
  st.reduction_exponent = prm.reduction_exponent;
  st.growth_exponent = prm.growth_exponent;
  st.pow_table = W.ensure_pow_table(prm.reduction_exponent, prm.growth_exponent);
  st.pow_table_len = kPowTableLen;
  if (prm.step_size_policy == GPDHG_STEPSIZE_ADAPTIVE) {
    st.kkt_passes += 0.5;
    // 1 / norm(A, Inf): entrywise max (:571). An empty matrix (the reference fails before
    // this point) gets tau_0 = 1, since 1/0 would make every averaging weight infinite.
    st.tau = P->amax > 0.0 ? 1.0 / P->amax : 1.0;
  } else {
    // estimate_maximum_singular_value (:139-172) with 0.001 failure probability, 0.2 error
    const double rel = 0.2, eps = 1.0 - (1.0 - rel) * (1.0 - rel);
    auto fail = [&](long long k) {
      if (k < 2 || eps <= 0.0) return 1.0;
      return std::min(0.824, 0.354 / std::sqrt(eps * (k - 1))) * std::sqrt((double)n) * std::pow(1.0 - eps, (double)k - 0.5);
    };
    std::mt19937_64 rng(1);
    std::normal_distribution<double> nd;
    std::vector<T> hx(n);
    for (auto& v : hx) v = (T)nd(rng);
    CK(cudaMemcpyAsync(W.tmp_n.get(), hx.data(), sizeof(T) * n, cudaMemcpyHostToDevice, s));
    CK(cudaStreamSynchronize(s));
    long long k = 0;
    std::vector<T> h(n);
    while (fail(k) > 0.001) {
      const double nx = std::sqrt(W.dot(W.tmp_n.get(), W.tmp_n.get(), n));
      // on the products' own stream, which waits for no other: a plain copy of pageable memory returns
      // before its transfer ends
      CK(cudaMemcpyAsync(h.data(), W.tmp_n.get(), sizeof(T) * n, cudaMemcpyDeviceToHost, s));
      CK(cudaStreamSynchronize(s));
      for (auto& v : h) v = (T)((double)v / nx);
      CK(cudaMemcpyAsync(W.tmp_n.get(), h.data(), sizeof(T) * n, cudaMemcpyHostToDevice, s));
      CK(cudaStreamSynchronize(s));
      W.spmv(P->A, W.tmp_n.get(), W.tmp_m.get());
      W.spmv(P->At, W.tmp_m.get(), W.dx.get());
      CK(cudaMemcpyAsync(W.tmp_n.get(), W.dx.get(), sizeof(T) * n, cudaMemcpyDeviceToDevice, s));
      ++k;
    }
    W.spmv(P->A, W.tmp_n.get(), W.tmp_m.get());
    W.spmv(P->At, W.tmp_m.get(), W.dx.get());
    const double xz = W.dot(W.tmp_n.get(), W.dx.get(), n);
    const double xx = W.dot(W.tmp_n.get(), W.tmp_n.get(), n);
    const double smax = std::sqrt(xz / xx);
    st.tau = (1.0 - rel) / smax;
    st.kkt_passes += (double)k;
    st.constant_step = 1;
    CK(cudaMemsetAsync(W.dx.get(), 0, sizeof(T) * n, s));
  }
  if (prm.scale_invariant_initial_primal_weight) {
    const double rhs = std::sqrt(1.0) * P->norm2_b_scaled, obj = std::sqrt(1.0) * P->norm2_c_scaled;
    st.omega = (obj > 0.0 && rhs > 0.0) ? prm.primal_importance * (obj / rhs) : prm.primal_importance;
  } else {
    st.omega = prm.primal_importance;
  }
  st.iter_start_tau = st.tau;
  // create_last_restart_info
  W.restart_kkt.valid = false;
  CK(cudaMemcpyAsync(W.rx.get(), W.x.get(), sizeof(T) * n, cudaMemcpyDeviceToDevice, s));
  CK(cudaMemcpyAsync(W.rgrad.get(), W.grad.get(), sizeof(T) * n, cudaMemcpyDeviceToDevice, s));
  if (m) {
    CK(cudaMemcpyAsync(W.ry.get(), W.y0.get(), sizeof(T) * m, cudaMemcpyDeviceToDevice, s));
    CK(cudaMemcpyAsync(W.rkx.get(), W.kx0.get(), sizeof(T) * m, cudaMemcpyDeviceToDevice, s));
  }
  CK(cudaStreamSynchronize(s));
  L.iteration = 1;
  L.t0 = Clock::now();
}

// FP32 -> FP64 hand-off: every vector converted, K x and K'y recomputed in FP64.
void handoff_to_fp64(gpdhg_problem* P, Workspace<float>& F, Workspace<double>& D) {
  cudaStream_t s = P->stream;
  auto conv = [&](const DBuf<float>& a, DBuf<double>& b) {
    const long long len = (long long)a.n;
    convert_kernel<float, double><<<std::max(1, std::min(ceil_div(len, kBlock), 4096)), kBlock, 0, s>>>(len, a.get(), b.get());
    CK_LAUNCH();
    ++P->launches;
  };
  conv(F.x, D.x); conv(F.dx, D.dx); conv(F.sx, D.sx); conv(F.ax, D.ax);
  conv(F.agrad, D.agrad); conv(F.grad, D.grad); conv(F.rx, D.rx); conv(F.rgrad, D.rgrad);
  conv(F.y0, D.y0); conv(F.y1, D.y1); conv(F.sy, D.sy); conv(F.skx, D.skx); conv(F.ay, D.ay);
  conv(F.akx, D.akx); conv(F.ry, D.ry); conv(F.rkx, D.rkx);
  StepState st = *F.st_host.p;
  const int n = P->n, m = P->m;
  // exact FP64 products of the current point
  D.spmv(P->A, D.x.get(), st.parity ? D.kx1.get() : D.kx0.get());
  D.spmv(P->At, st.parity ? D.y1.get() : D.y0.get(), D.kty.get());
  // The FP64 phase restarts its averages at the handed-over point: FP32-accumulated
  // sums (and the K x-bar they imply) are only consistent to ~1e-7 and would feed a
  // phantom residual to the dual update after a restart to the average.
  CK(cudaMemsetAsync(D.sx.get(), 0, sizeof(double) * D.sx.n, s));
  CK(cudaMemsetAsync(D.sy.get(), 0, sizeof(double) * D.sy.n, s));
  CK(cudaMemsetAsync(D.skx.get(), 0, sizeof(double) * D.skx.n, s));
  st.count_primal = st.count_dual = 0;
  st.sum_w_primal = st.sum_w_dual = 0.0;
  st.pending_commit = 0;
  st.pow_table = D.ensure_pow_table(st.reduction_exponent, st.growth_exponent);
  grad_kernel<double><<<D.grid_for(n), kBlock, 0, s>>>(n, D.c, D.kty.get(), D.grad.get());
  CK_LAUNCH();
  ++P->launches;
  D.restart_kkt.valid = false;
  CK(cudaMemcpyAsync(D.rx.get(), D.x.get(), sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
  CK(cudaMemcpyAsync(D.rgrad.get(), D.grad.get(), sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
  if (m) {
    CK(cudaMemcpyAsync(D.ry.get(), st.parity ? D.y1.get() : D.y0.get(), sizeof(double) * m, cudaMemcpyDeviceToDevice, s));
    CK(cudaMemcpyAsync(D.rkx.get(), st.parity ? D.kx1.get() : D.kx0.get(), sizeof(double) * m,
                       cudaMemcpyDeviceToDevice, s));
  }
  *D.st_host.p = st;
  CK(cudaStreamSynchronize(s));
}

}  // namespace

void solve(gpdhg_problem* P, const gpdhg_params& prm, gpdhg_result* res, double* primal_out, double* dual_out) {
  P->history.clear();
  LoopState L;
  L.launches_at_start = P->launches;
  const int prec = prm.precision;
  if (prec == GPDHG_PRECISION_FP64) {
    if (!P->ws64) P->ws64.reset(new Workspace<double>(P));
    L.precision = GPDHG_PRECISION_FP64;
    init_state(P, *P->ws64, prm, L);
    run_phase(P, *P->ws64, prm, L, res, primal_out, dual_out, false);
    return;
  }
  if (!P->ws32) P->ws32.reset(new Workspace<float>(P));
  L.precision = GPDHG_PRECISION_FP32;
  init_state(P, *P->ws32, prm, L);
  const bool refine = prec == GPDHG_PRECISION_FP32_REFINE;
  if (run_phase(P, *P->ws32, prm, L, res, primal_out, dual_out, refine)) return;
  if (!P->ws64) P->ws64.reset(new Workspace<double>(P));
  handoff_to_fp64(P, *P->ws32, *P->ws64);
  L.precision = GPDHG_PRECISION_FP64;
  L.handoff_iteration = (int)(L.iteration - 1);
  run_phase(P, *P->ws64, prm, L, res, primal_out, dual_out, false);
}

void current_iterate(const gpdhg_problem* P, double* x, double* y) {
  cudaStream_t s = P->stream;
  auto get = [&](auto& W) {
    const int p = W.st_host.p->parity;
    if constexpr (std::is_same_v<std::decay_t<decltype(*W.x.get())>, double>) {
      if (x) CK(cudaMemcpyAsync(x, W.x.get(), sizeof(double) * P->n, cudaMemcpyDeviceToHost, s));
      if (y && P->m) CK(cudaMemcpyAsync(y, W.ycur(p), sizeof(double) * P->m, cudaMemcpyDeviceToHost, s));
      CK(cudaStreamSynchronize(s));
    } else {
      std::vector<float> tx(P->n), ty(std::max(P->m, 1));
      CK(cudaMemcpyAsync(tx.data(), W.x.get(), sizeof(float) * P->n, cudaMemcpyDeviceToHost, s));
      if (P->m) CK(cudaMemcpyAsync(ty.data(), W.ycur(p), sizeof(float) * P->m, cudaMemcpyDeviceToHost, s));
      CK(cudaStreamSynchronize(s));
      if (x) for (int j = 0; j < P->n; ++j) x[j] = tx[j];
      if (y) for (int i = 0; i < P->m; ++i) y[i] = ty[i];
    }
  };
  if (P->last_precision == GPDHG_PRECISION_FP64 && P->ws64) get(*P->ws64);
  else if (P->last_precision == GPDHG_PRECISION_FP32 && P->ws32) get(*P->ws32);
  else throw Error(GPDHG_ERR_INVALID_ARGUMENT, "no solve has completed on this problem");
}

}  // namespace gpdhg
