// eval_kernels.cuh — FP64 reductions for termination checks and restart scoring.
//
// The reference computes each statistic with its own broadcast kernel and a host
// round trip per norm, and allocates temporaries for concatenated norms
// (src/iteration_stats_utils_gpu.jl:23-372, src/saddle_point_gpu.jl:250-278). Here every
// statistic of one evaluation is accumulated in FP64 in a single pass per side (n columns,
// m rows) over fixed segments (batch_kernels.cuh), into per-segment partials that one
// finalize CTA per instance and quantity reduces in a fixed order, into the host's memory.
// Comparisons, maxima and sign tests run on the integer pipe (bit patterns), so the FP64
// pipe only does the arithmetic itself.
#pragma once

#include "common.cuh"

namespace gpdhg {

// A double's bits and back through a move the compiler does not look into: given a plain bit cast
// it recognises masks of the sign bit as |v| and -v, and range tests as FP64 comparisons, and emits
// FP64-pipe instructions for them (7 of the 14 that a column of gpdhg_convergence_noalloc took).
__device__ __forceinline__ unsigned long long bits_of(double v) {
  unsigned long long b;
  asm("mov.b64 %0, %1;" : "=l"(b) : "d"(v));
  return b;
}
__device__ __forceinline__ double of_bits(unsigned long long b) {
  double v;
  asm("mov.b64 %0, %1;" : "=d"(v) : "l"(b));
  return v;
}
constexpr unsigned long long kSignBit = 0x8000000000000000ULL;
constexpr unsigned long long kInfBits = 0x7ff0000000000000ULL;

// The evaluation's max-quantities are all magnitudes (|v|, or a positive part): their
// NaN-propagating maximum is the integer maximum of the bit patterns with the sign cleared
// (+0 < ... < +inf < NaN), done on the integer pipe instead of GB300's narrow FP64 pipe.
__device__ __forceinline__ double nan_max(double a, double b) {
  const unsigned long long ua = bits_of(a) & ~kSignBit, ub = bits_of(b) & ~kSignBit;
  return of_bits(ua > ub ? ua : ub);
}

__device__ __forceinline__ bool bits_nan(double v) { return (bits_of(v) & ~kSignBit) > kInfBits; }
__device__ __forceinline__ bool bits_zero(double v) { return (bits_of(v) << 1) == 0; }
__device__ __forceinline__ bool bits_negative(double v) { return (long long)bits_of(v) < 0; }
__device__ __forceinline__ bool bits_finite(double v) { return (bits_of(v) & kInfBits) != kInfBits; }
__device__ __forceinline__ double negate_bits(double v) { return of_bits(bits_of(v) ^ kSignBit); }

// Julia's max(v, 0) (NaN-propagating), by sign and NaN tests on the bits.
__device__ __forceinline__ double pos_part(double v) {
  const unsigned long long b = bits_of(v);
  return of_bits((long long)b > 0 || bits_nan(v) ? b : 0);  // +x (x != 0) and NaN kept; -x, -0, +0 -> +0
}

// (double)v. A float's conversion runs on the FP64 pipe; the exponent is re-biased on the integer
// pipe instead (a subnormal is first made normal by an exact FP32 product with 2^24).
__device__ __forceinline__ double widen(double v) { return v; }
__device__ __forceinline__ double widen(float v) {
  unsigned mag = __float_as_uint(v) & 0x7fffffffu, bias = 0x38000000u;
  if (mag < 0x00800000u) {
    mag = __float_as_uint(__uint_as_float(mag) * 16777216.0f);
    bias = mag ? 0x38000000u - (24u << 20) : 0u;
  } else if (mag >= 0x7f800000u) {
    bias = 0x70000000u;   // infinite and NaN: to the top exponent
  }
  const unsigned hi = (__float_as_uint(v) & 0x80000000u) | ((mag >> 3) + bias);
  return of_bits((unsigned long long)hi << 32 | (unsigned)(mag << 29));
}
// Sums skipped by a warp in which p holds nowhere: c += a b with one rounding, and with the product
// rounded first. (Written as a plain condition, a predicated instruction or a vote around the C
// expression, the arithmetic is moved out and done for every element; a volatile one stays behind
// the vote.)
__device__ __forceinline__ void fma_if(bool p, double a, double b, double& c) {
  if (!__any_sync(__activemask(), p)) return;
  a = of_bits(p ? bits_of(a) : 0ULL);
  b = of_bits(p ? bits_of(b) : 0ULL);
  asm volatile("fma.rn.f64 %0, %1, %2, %0;" : "+d"(c) : "d"(a), "d"(b));
}
__device__ __forceinline__ void add_product_if(bool p, double a, double b, double& c) {
  if (!__any_sync(__activemask(), p)) return;
  a = of_bits(p ? bits_of(a) : 0ULL);
  b = of_bits(p ? bits_of(b) : 0ULL);
  asm volatile("{\n\t.reg .f64 t;\n\tmul.rn.f64 t, %1, %2;\n\tadd.rn.f64 %0, %0, t;\n\t}" : "+d"(c) : "d"(a), "d"(b));
}

__device__ __forceinline__ double warp_nan_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = nan_max(v, __shfl_down_sync(0xffffffffu, v, o));
  return v;
}

__device__ __forceinline__ double block_nan_max(double v, double* sh) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  v = warp_nan_max(v);
  __syncthreads();
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  double r = 0.0;
  if (wid == 0) {
    r = (lane < (int)(blockDim.x >> 5)) ? sh[lane] : 0.0;
    r = warp_nan_max(r);
  }
  return r;
}

// Q per-thread accumulators reduced over the CTA in a fixed order. The values go through
// shared memory (sh: kRedChunk x kBlock doubles, kRedChunk quantities at a time); warp w
// reduces quantities w, w + 8, ... of a chunk: lane l combines entry l of every warp in warp
// order, then a shuffle tree finishes (12 warp-wide FP64 adds per summed quantity, where a
// shuffle tree in every warp takes 40; maxima run on the integer pipe). Bit q of MAXMASK
// selects max (else sum). A quantity's order does not depend on Q. The result for q is
// valid in thread q (res: Q doubles).
constexpr int kRedChunk = 16;
template <int Q, unsigned MAXMASK>
__device__ __forceinline__ double block_reduce_q(const double* acc, double* sh, double* res) {
  static_assert(Q <= 32, "MAXMASK holds 32 quantities");
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
#pragma unroll
  for (int q0 = 0; q0 < Q; q0 += kRedChunk) {
    if (q0 > 0) __syncthreads();  // the previous chunk's readers are done with sh
#pragma unroll
    for (int q = q0; q < Q && q < q0 + kRedChunk; ++q) sh[(q - q0) * kBlock + t] = acc[q];
    __syncthreads();
    for (int q = q0 + wid; q < Q && q < q0 + kRedChunk; q += kBlock / 32) {
      const bool is_max = (MAXMASK >> q) & 1u;
      const double* c = sh + (q - q0) * kBlock + lane;
      double v = c[0];
#pragma unroll
      for (int w = 1; w < kBlock / 32; ++w) v = is_max ? nan_max(v, c[w * 32]) : v + c[w * 32];
      v = is_max ? warp_nan_max(v) : warp_sum(v);
      if (lane == 0) res[q] = v;
    }
  }
  __syncthreads();
  return t < Q ? res[t] : 0.0;
}

// a / b from r = 1 / b (correctly rounded, computed once per divisor): the product a r
// corrected once with the exact residual a - q b (Markstein's correction step, P. Markstein,
// "IA-64 and Elementary Functions", 2000), three FP64 operations instead of a division. It
// returns the correctly rounded quotient for normal operands (a CPU check of 5e7 random
// pairs over a 2^200 range found no difference from a / b); zero and non-finite products
// are returned as they are, which keeps the quotient's sign and infinities.
__device__ __forceinline__ double div_rcp(double a, double b, double r) {
  const double q = a * r;
  if (!bits_finite(q) || bits_zero(q)) return q;
  const double e = fma(-q, b, a);
  return fma(e, r, q);
}

// The statistics below are written so that the FP64 pipe (2 lanes per SM and cycle: a warp-wide
// FP64 instruction takes it for 16 cycles) only sees operations whose result is not known from the
// operands' bits. Measured on the transportation LP (1M columns, FP64): 79 FP64 operations per
// column when written plainly, the negations and absolute values among them (both compile to
// FP64 additions), the pipe 81% busy.

// Squared and largest violation of l <= x <= u: (l - x)+ and (x - u)+
// (src/iteration_stats_utils_gpu.jl:71-90). A projected iterate, or an average of some, violates
// its bounds by rounding at most, so the arithmetic sits behind a comparison of order keys; it
// also runs for non-finite operands, which then propagate as in the plain form.
__device__ __forceinline__ long long bits_key(double v) {   // order_key without a bit cast
  const long long b = (long long)bits_of(v);
  return b ^ (long long)((unsigned long long)(b >> 63) >> 1);
}
// kFused: the square is added with one rounding, else rounded first.
template <bool kFused>
__device__ __forceinline__ void add_violation(double x, double l, double u, double& sq, double& mx) {
  const long long k = bits_key(x);
  const bool below = k < bits_key(l), above = bits_key(u) < k;
  const bool plain = !bits_finite(x) || bits_nan(l) || bits_nan(u) || (below && above);
  if (!(below || above || plain)) return;
  if (plain) {
    const double lv = pos_part(l - x), uv = pos_part(x - u);
    sq = __dadd_rn(sq, __fma_rn(lv, lv, __dmul_rn(uv, uv)));
    mx = nan_max(mx, nan_max(lv, uv));
  } else {
    const double v = of_bits(bits_of(below ? l : x)) - of_bits(bits_of(below ? x : u));
    sq = kFused ? fma(v, v, sq) : __dadd_rn(sq, __dmul_rn(v, v));
    mx = nan_max(mx, v);
  }
}
__device__ __forceinline__ void add_square(double v, double& sq) {
  fma_if(!bits_zero(v), v, v, sq);
}

// Reduced cost of gradient g: max(g, 0) isfinite(l) + min(g, 0) isfinite(u)
// (src/iteration_stats_utils_gpu.jl:168) is g itself or 0, so it and the dual residual g - rc are
// selections (NaN where the plain form is: g NaN, or infinite and kept).
__device__ __forceinline__ bool keeps_cost(double g, bool fl, bool fu) {
  if (bits_nan(g)) return fl || fu;
  return !bits_zero(g) && (bits_negative(g) ? fu : fl);
}
__device__ __forceinline__ double cost_residual(double g, bool kept) {
  return of_bits(!kept ? bits_of(g) : bits_finite(g) ? 0ULL : kInfBits | 1ULL << 51);
}
// Adds the dual objective's term of a kept reduced cost (:120-126): l rc for rc > 0, u rc for
// rc < 0, nothing for NaN; a zero bound adds nothing to a finite rc.
template <bool kFused>
__device__ __forceinline__ void add_bound_term(double g, bool kept, double l, double u, double& sum) {
  const double bound = of_bits(bits_negative(g) ? bits_of(u) : bits_of(l));
  const bool counts = kept && !bits_nan(g) && (!bits_zero(bound) || !bits_finite(g));
  if constexpr (kFused) fma_if(counts, bound, g, sum);
  else add_product_if(counts, bound, g, sum);
}
// The constraint violation b - Kx, or its positive part on an inequality row (:26-45).
__device__ __forceinline__ double row_violation(double d, bool ineq) {
  return of_bits(bits_of(ineq ? pos_part(d) : d));
}
// (-y)+ of an inequality row's dual (:198-211): a bit flip of a negative (or NaN) y
__device__ __forceinline__ double dual_violation(double y, bool ineq) {
  return of_bits(ineq && (bits_negative(y) || bits_nan(y)) && !bits_zero(y) ? bits_of(y) ^ kSignBit : 0ULL);
}

// One evaluation's quantities. Columns: the unscaled statistics of the average (kN_*), then at
// kEvalNQ the weighted-KKT ingredients (src/saddle_point_gpu.jl:250-278) of the current, average
// and last-restart points (4 each: bound violation, c'x, dual residual, bound terms) and
// ||avg - last restart||^2. Rows: kM_*, then 3 per point (violation, dual violation, b'y) and the
// distance.
enum EvalNQ {
  kN_LuSq = 0, kN_LuMax, kN_Cx, kN_XMax, kN_XSq, kN_RcvSq, kN_RcvMax, kN_Contrib,
  kN_RayLuMax, kN_RayRcvMax, kN_RayContrib, kN_RayRcMax, kEvalNQ
};
constexpr unsigned kEvalNMax = (1u << kN_LuMax) | (1u << kN_XMax) | (1u << kN_RcvMax) | (1u << kN_RayLuMax) |
                               (1u << kN_RayRcvMax) | (1u << kN_RayRcMax);
enum EvalMQ { kM_CvSq = 0, kM_CvMax, kM_DrSq, kM_DrMax, kM_By, kM_YMax, kM_YSq, kM_RayCvMax, kEvalMQ };
constexpr unsigned kEvalMMax = (1u << kM_CvMax) | (1u << kM_DrMax) | (1u << kM_YMax) | (1u << kM_RayCvMax);
constexpr int kKktNQ = 13;
constexpr int kKktMQ = 10;
constexpr int kPassNQ = kEvalNQ + kKktNQ;
constexpr int kPassMQ = kEvalMQ + kKktMQ;

// What an instance's passes need of its StepState, read once per CTA.
template <class T>
struct EvalParams {
  double wx, wy, rwx, rwy;
  T commit_weight;
  bool parity, pending, current, restart;
  __device__ __forceinline__ EvalParams(const StepState* st, int inst) {
    const StepState& s = st[inst];
    wx = s.sum_w_primal;
    wy = s.sum_w_dual;
    rwx = s.rcp_w_primal;
    rwy = s.rcp_w_dual;
    commit_weight = (T)s.commit_weight;
    parity = s.parity != 0;
    pending = s.pending_commit != 0;
    current = s.eval_current != 0;
    restart = s.eval_restart != 0;
  }
};

// The row pass of an evaluation (optimize(), src/primal_dual_hybrid_gradient_gpu.jl:633-760): the
// commit of the last accepted step's Sigma y and Sigma Kx, the average y and Kx
// (compute_average!, src/saddle_point_gpu.jl:226-240; the current point when there is no average),
// the unscaled statistics and the KKT ingredients. The instance's weights, buffer parity and
// what to do come from its StepState. The last restart point's ingredients depend on that
// point alone, so they are formed only when it moved (eval_restart).
template <class T>
struct EvalPassM {
  using Params = EvalParams<T>;
  const double* con;   // constraint_rescaling (E)
  const double* rcon;  // 1 / E
  const double* ob;
  const T* b;
  const T* y0; const T* y1; const T* kx0; const T* kx1;
  const T* ry; const T* rkx;
  T* sy;
  T* skx;
  T* ay;         // the average, written
  T* akx;
  int neq;
  const uint8_t* ineq_flag;  // per-row '>=' flag (packed batches); NULL: rows >= neq
  __device__ __forceinline__ void point(T yv, T kv, double b, bool ineq, double* a) const {
    const double y = widen(yv);
    add_square(row_violation(b - widen(kv), ineq), a[0]);
    add_square(dual_violation(y, ineq), a[1]);
    a[2] = fma(b, y, a[2]);
  }
  // A row's operands, loaded apart from their use so that a caller can load ahead.
  struct In {
    T yc, kc, sy, skx, b, ry, rkx;
    double con, rcon, ob;
    bool ineq;
  };
  __device__ __forceinline__ void load(const Params& s, int i, In& v) const {
    v.yc = (s.parity ? y1 : y0)[i];
    v.kc = (s.parity ? kx1 : kx0)[i];
    v.ineq = ineq_flag ? ineq_flag[i] != 0 : i >= neq;
    if (!s.current) {
      v.sy = sy[i];
      v.skx = skx[i];
    }
    v.con = con[i];
    v.rcon = rcon[i];
    v.ob = ob[i];
    v.b = this->b[i];
    v.ry = ry[i];
    if (s.restart) v.rkx = rkx[i];
  }
  __device__ __forceinline__ void apply(const Params& s, int i, const In& v, double* a) const {
    const T yc = v.yc, kc = v.kc;
    const bool ineq = v.ineq;
    T ya = yc, ka = kc;
    if (!s.current) {
      T vy = v.sy, vk = v.skx;
      if (s.pending) {
        vy = fma(yc, s.commit_weight, vy);
        vk = fma(kc, s.commit_weight, vk);
        sy[i] = vy;
        skx[i] = vk;
      }
      ya = (T)div_rcp(widen(vy), s.wy, s.rwy);
      ka = (T)div_rcp(widen(vk), s.wx, s.rwx);
    }
    ay[i] = ya;
    akx[i] = ka;
    {
      const double y = div_rcp(widen(ya), v.con, v.rcon);   // :474-475
      const double kx = widen(ka) * v.con;                  // :476-477
      const double b = v.ob;
      const double cv = row_violation(b - kx, ineq);
      add_square(cv, a[kM_CvSq]);
      a[kM_CvMax] = nan_max(a[kM_CvMax], cv);
      const double dr = dual_violation(y, ineq);
      add_square(dr, a[kM_DrSq]);
      a[kM_DrMax] = nan_max(a[kM_DrMax], dr);
      a[kM_By] = fma(b, y, a[kM_By]);
      a[kM_YMax] = nan_max(a[kM_YMax], y);
      a[kM_YSq] = fma(y, y, a[kM_YSq]);
      // ray: right-hand side 0 (:338)
      a[kM_RayCvMax] = nan_max(a[kM_RayCvMax], row_violation(negate_bits(kx), ineq));
    }
    double* k = a + kEvalMQ;
    const double b = widen(v.b);
    point(yc, kc, b, ineq, k);
    point(ya, ka, b, ineq, k + 3);
    if (s.restart) point(v.ry, v.rkx, b, ineq, k + 6);
    const double d = widen(ya) - widen(v.ry);
    k[9] = fma(d, d, k[9]);
  }
};

// The column pass: the average x, its gradient c - A' y-bar (aty, formed after the row pass;
// the current point takes the gradient buffer as it stood), buffer_primal_gradient = c - K'y
// (:742), the statistics and the KKT ingredients.
template <class T>
struct EvalPassN {
  using Params = EvalParams<T>;
  const double* var;   // variable_rescaling (D)
  const double* rvar;  // 1 / D
  const double* ol; const double* ou; const double* oc;
  const T* l; const T* u; const T* c;
  const T* x; const T* sx; const T* aty; const T* kty;
  const T* rx; const T* rgrad;
  T* ax;         // the average, written
  T* agrad;
  T* grad;
  __device__ __forceinline__ void point(T xv, T gv, double l, double u, double c, bool fl, bool fu, double* a) const {
    const double x = widen(xv), g = widen(gv);
    double unused = 0.0;
    add_violation<false>(x, l, u, a[0], unused);
    a[1] = fma(c, x, a[1]);
    const bool kept = keeps_cost(g, fl, fu);
    add_square(cost_residual(g, kept), a[2]);
    add_bound_term<false>(g, kept, l, u, a[3]);
  }
  // A column's operands, loaded apart from their use so that a caller can load ahead.
  struct In {
    T c, x, sx, g, kty, l, u, rx, rgrad;   // g: A' y-bar, or the gradient as it stood
    double var, rvar, ol, ou, oc;
  };
  __device__ __forceinline__ void load(const Params& s, int j, In& v) const {
    v.c = c[j];
    v.x = x[j];
    if (s.current) {
      v.g = grad[j];
    } else {
      v.sx = sx[j];
      v.g = aty[j];
    }
    v.kty = kty[j];
    v.var = var[j];
    v.rvar = rvar[j];
    v.ol = ol[j];
    v.ou = ou[j];
    v.oc = oc[j];
    v.l = l[j];
    v.u = u[j];
    v.rx = rx[j];
    if (s.restart) v.rgrad = rgrad[j];
  }
  __device__ __forceinline__ void apply(const Params& s, int j, const In& v, double* a) const {
    const T cs = v.c, xc = v.x;
    T xa = xc, ga = v.g;
    if (!s.current) {
      xa = (T)div_rcp(widen(v.sx), s.wx, s.rwx);
      ga = cs - v.g;
    }
    ax[j] = xa;
    agrad[j] = ga;
    const T gc = cs - v.kty;
    grad[j] = gc;
    {
      const double x = div_rcp(widen(xa), v.var, v.rvar);   // :470-471
      const double g = widen(ga) * v.var;                   // :472-473
      const double l = v.ol, u = v.ou, c = v.oc;
      const bool fl = bits_finite(l), fu = bits_finite(u);
      add_violation<true>(x, l, u, a[kN_LuSq], a[kN_LuMax]);
      a[kN_Cx] = fma(c, x, a[kN_Cx]);
      a[kN_XMax] = nan_max(a[kN_XMax], x);
      a[kN_XSq] = fma(x, x, a[kN_XSq]);
      const bool kept = keeps_cost(g, fl, fu);
      const double rcv = cost_residual(g, kept);
      add_square(rcv, a[kN_RcvSq]);
      a[kN_RcvMax] = nan_max(a[kN_RcvMax], rcv);
      add_bound_term<true>(g, kept, l, u, a[kN_Contrib]);
      // primal ray, before division by ||x||_inf: bounds 0 where finite (:335-336)
      const bool xnan = bits_nan(x);
      if (xnan ? fl || fu : (bits_negative(x) ? fl : fu)) a[kN_RayLuMax] = nan_max(a[kN_RayLuMax], x);
      // dual ray: objective set to zero, gradient - c (:346-354)
      const double gr = g - c;
      const bool keptr = keeps_cost(gr, fl, fu);
      a[kN_RayRcvMax] = nan_max(a[kN_RayRcvMax], cost_residual(gr, keptr));
      add_bound_term<true>(gr, keptr, l, u, a[kN_RayContrib]);
      if (keptr) a[kN_RayRcMax] = nan_max(a[kN_RayRcMax], gr);
    }
    double* k = a + kEvalNQ;
    const double l = widen(v.l), u = widen(v.u), c = widen(cs);
    const bool fl = bits_finite(l), fu = bits_finite(u);
    point(xc, gc, l, u, c, fl, fu, k);
    point(xa, ga, l, u, c, fl, fu, k + 4);
    if (s.restart) point(v.rx, v.rgrad, l, u, c, fl, fu, k + 8);
    const double d = widen(xa) - widen(v.rx);
    k[12] = fma(d, d, k[12]);
  }
};

// ---- small vector kernels --------------------------------------------------------

template <class T>
__global__ void grad_kernel(int n, const T* c, const T* kty, T* grad) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) grad[j] = c[j] - kty[j];
}

template <class S, class D>
__global__ void convert_kernel(long long len, const S* src, D* dst) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (long long)gridDim.x * blockDim.x)
    dst[i] = (D)src[i];
}

// A solution as the caller reads it: FP64, entry k at the caller's position perm[k] (NULL: k). On
// the host, widening and permuting 2M columns took 3 ms of a solve's end.
template <class T>
__global__ void caller_values_kernel(int len, const T* __restrict__ src, const int32_t* __restrict__ perm,
                                     double* __restrict__ dst) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < len; k += gridDim.x * blockDim.x)
    dst[perm ? perm[k] : k] = (double)src[k];
}

}  // namespace gpdhg
