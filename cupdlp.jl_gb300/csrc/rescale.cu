// rescale.cu — rescale_problem (src/preprocess.jl:619-675) on the GPU, for
// gpdhg_problem_create_unscaled: Ruiz L-inf iterations (:398-463), the optional L2-norm
// rescaling, and Pock-Chambolle (:494-525), each applied in place to both CSR copies of A,
// to l, u, c, b, and accumulated into the constraint / variable rescaling vectors.
//
// Every operation follows the host restatement (cupdlp/preprocess.py) in kind and order:
// maxima, square roots and divisions are correctly rounded on both sides, a scaled entry is
// ((1 / E_i) a_ij) (1 / D_j) in both CSR copies, c ./= D, bounds .*= D, b ./= E, and the
// cumulative vectors are multiplied in the reference's order, so Ruiz scaling is bitwise the
// host's. Row sums (Pock-Chambolle, L2) add in a fixed order, which differs from
// the host's sequential order by rounding only.
#include <algorithm>
#include <cmath>
#include <vector>

#include "problem.h"

namespace gpdhg {

namespace {

enum RowOp : int { kRowAbsMax = 0, kRowPowSum = 1, kRowScaledSq = 2 };

// max of magnitudes on the integer pipe (an FP64 maximum runs on GB300's narrow FP64 pipe)
__device__ __forceinline__ double magnitude_max(double a, double b) {
  return __longlong_as_double(max(__double_as_longlong(a), __double_as_longlong(b)));
}
__device__ __forceinline__ double magnitude(double v) {
  return __longlong_as_double(__double_as_longlong(v) & 0x7fffffffffffffffLL);
}
// One row (entries [b, e) of val) reduced by `lanes` consecutive lanes of the warp, lane i of them
// first taking entries i, i + lanes, ...; valid in lane 0 of them. Summing, an entry's place is its
// position modulo 32 and the places are added by halves, so a row of at most `lanes` entries has
// the same sum with any number of lanes (the places beyond its end add zeros).
template <int kOp>
__device__ __forceinline__ double reduce_row(const double* __restrict__ val, int b, int e, int i, int lanes,
                                             double alpha, double inv) {
  double acc = 0.0;
  for (int k = b + i; k < e; k += lanes) {
    if constexpr (kOp == kRowAbsMax) acc = magnitude_max(acc, magnitude(val[k]));
    else if constexpr (kOp == kRowPowSum) acc += pow(magnitude(val[k]), alpha);
    else {
      const double t = val[k] * inv;
      acc += t * t;
    }
  }
  for (int o = lanes >> 1; o > 0; o >>= 1) {
    const double v = __shfl_down_sync(0xffffffffu, acc, o);
    acc = kOp == kRowAbsMax ? magnitude_max(acc, v) : acc + v;
  }
  return acc;
}

// Calls row(r, b, e, i, lanes, own) for the rows of a CSR matrix: 32 / lanes rows side by side per
// warp where they have at most `lanes` entries, then each longer one by the whole warp. (A warp
// per row leaves 30 lanes idle on a transportation LP's A', where pow's hundred-odd FP64
// instructions took 5.8 ms.)
// Every lane of the warp makes every call; own: the row is the lane's.
template <class Row>
__device__ __forceinline__ void for_rows(int nrows, const int32_t* __restrict__ rp, int lanes, Row row) {
  const int lane = threadIdx.x & 31, i = lane & (lanes - 1), per_warp = 32 / lanes;
  const long long warps = (long long)gridDim.x * (kBlock / 32);
  for (long long r0 = ((long long)blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5)) * per_warp; r0 < nrows;
       r0 += warps * per_warp) {
    const long long r = r0 + lane / lanes;
    const int b = r < nrows ? rp[r] : 0, e = r < nrows ? rp[r + 1] : 0;
    const bool longer = e - b > lanes;
    row((int)r, b, longer ? b : e, i, lanes, r < nrows && !longer);
    for (unsigned todo = __ballot_sync(0xffffffffu, longer && i == 0); todo; todo &= todo - 1) {
      const int from = __ffs(todo) - 1;
      row((int)(r0 + from / lanes), __shfl_sync(0xffffffffu, b, from), __shfl_sync(0xffffffffu, e, from), lane, 32,
          true);
    }
  }
}

template <int kOp>
__global__ void __launch_bounds__(kBlock) row_reduce_kernel(int nrows, int lanes, const int32_t* __restrict__ rp,
                                                            const double* __restrict__ val, double alpha,
                                                            const double* __restrict__ sf, double* out) {
  for_rows(nrows, rp, lanes, [&](int r, int b, int e, int i, int width, bool own) {
    const double inv = kOp == kRowScaledSq && own ? 1.0 / sf[r] : 0.0;
    const double v = reduce_row<kOp>(val, b, e, i, width, alpha, inv);
    if (own && i == 0) out[r] = v;
  });
}

// a_ij <- ((1 / E_i) a_ij) (1 / D_j) in a CSR whose rows are A's rows (transposed = 0) or
// A's columns (transposed = 1), and the scaled rows' max |a| into row_max (the next Ruiz pass's).
__global__ void __launch_bounds__(kBlock) scale_matrix_kernel(int nrows, int lanes, const int32_t* __restrict__ rp,
                                                              const int32_t* __restrict__ col, double* __restrict__ val,
                                                              const double* __restrict__ inv_con,
                                                              const double* __restrict__ inv_var, int transposed,
                                                              double* __restrict__ row_max) {
  for_rows(nrows, rp, lanes, [&](int r, int b, int e, int i, int width, bool own) {
    const double mine = own ? (transposed ? inv_var[r] : inv_con[r]) : 0.0;
    const double* other = transposed ? inv_con : inv_var;
    double acc = 0.0;
    for (int k = b + i; k < e; k += width) {
      const double o = other[col[k]];
      const double v = transposed ? (o * val[k]) * mine : (mine * val[k]) * o;
      val[k] = v;
      acc = magnitude_max(acc, magnitude(v));
    }
    for (int o = width >> 1; o > 0; o >>= 1) acc = magnitude_max(acc, __shfl_down_sync(0xffffffffu, acc, o));
    if (own && i == 0) row_max[r] = acc;
  });
}

enum FactorOp : int { kFactorSqrt = 0, kFactorL2 = 1 };

// Per entry: f = sqrt(x) (Ruiz, Pock-Chambolle) or f = sqrt(sf * sqrt(x)) (L2); f == 0 -> 1;
// cum *= f; inv = 1 / f; and the vectors it scales: c ./= f, l .*= f, u .*= f (columns), b ./= f (rows).
__device__ __forceinline__ void apply_factor(int i, int op, const double* x, const double* sf, double* inv, double* cum,
                                             double* quotient, double* product_l, double* product_u) {
  double v;
  if (op == kFactorSqrt) {
    v = sqrt(x[i]);
  } else {
    const double s = sf[i] == 0.0 ? 1.0 : sf[i];
    double norm = s * sqrt(x[i]);
    if (norm == 0.0) norm = 1.0;
    v = sqrt(norm);
  }
  if (v == 0.0) v = 1.0;
  inv[i] = 1.0 / v;
  cum[i] *= v;
  quotient[i] = quotient[i] / v;
  if (product_l) {
    product_u[i] = product_u[i] * v;
    product_l[i] = product_l[i] * v;
  }
}
struct FactorSide {
  const double* x;
  const double* sf;
  double* inv;
  double* cum;
};
__global__ void factor_kernel(int n, int m, int op, FactorSide col, FactorSide row, double* c, double* l, double* u,
                              double* b) {
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    apply_factor(i, op, col.x, col.sf, col.inv, col.cum, c, l, u);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += stride)
    apply_factor(i, op, row.x, row.sf, row.inv, row.cum, b, nullptr, nullptr);
}

// sf == 0 -> 1 (the L2 pre-scale of an empty row or column).
__global__ void unit_if_zero_kernel(long long len, double* x) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (long long)gridDim.x * blockDim.x)
    if (x[i] == 0.0) x[i] = 1.0;
}

__global__ void fill_kernel(long long len, double v, double* x) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (long long)gridDim.x * blockDim.x)
    x[i] = v;
}

// total *= cum
__global__ void accumulate_kernel(long long len, const double* __restrict__ cum, double* total) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (long long)gridDim.x * blockDim.x)
    total[i] *= cum[i];
}

// out = max of len magnitudes (one CTA: the row maxima of the scaled matrix)
__global__ void __launch_bounds__(1024) max_kernel(int len, const double* __restrict__ x, double* out) {
  __shared__ double part[32];
  double acc = 0.0;
  for (int i = threadIdx.x; i < len; i += 1024) acc = magnitude_max(acc, x[i]);
  for (int o = 16; o > 0; o >>= 1) acc = magnitude_max(acc, __shfl_down_sync(0xffffffffu, acc, o));
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    acc = part[threadIdx.x];
    for (int o = 16; o > 0; o >>= 1) acc = magnitude_max(acc, __shfl_down_sync(0xffffffffu, acc, o));
    if (threadIdx.x == 0) *out = acc;
  }
}

int grid_of(long long work, int per_block) {
  return (int)std::max<long long>(1, std::min<long long>((work + per_block - 1) / per_block, 8192));
}
// Lanes per row: the power of two from 2 to 32 next above the average row.
int lanes_of(long long nnz, int rows) {
  int lanes = 2;
  while (lanes < 32 && (long long)lanes * rows < nnz) lanes *= 2;
  return lanes;
}

}  // namespace

// Each stage's launches per pass: the factors with the vectors they scale, and each CSR copy scaled
// with its rows' new maxima (the next pass's input). Plainly (maxima, factors, matrix and vectors
// in launches of their own, a warp per row, FP64 maxima) the transportation LP (1M columns,
// 2M nonzeros) took 16.3 ms.
void rescale_on_device(gpdhg_problem* p, const gpdhg_params& prm) {
  cudaStream_t s = p->stream;
  const int n = p->n, m = p->m;
  const size_t N = std::max(n, 1), M = std::max(m, 1);
  DBuf<double> rx(N), cx(M), rsf(N), csf(M), iv(N), ic(M), cum_v(N), cum_c(M), amax(1);
  const int ln = lanes_of(p->nnz, n), lm = lanes_of(p->nnz, std::max(m, 1));
  const int gw_n = grid_of(n, kBlock / ln), gw_m = grid_of(m, kBlock / lm);
  const int ge_n = grid_of(n, kBlock), ge_m = grid_of(m, kBlock);
  bool have_max = false;   // rx / cx hold the row maxima of the matrix as it stands
  // p->var / p->con start at ones (problem_init with no rescaling vectors)
  auto apply = [&](int op) {
    factor_kernel<<<std::max(ge_n, ge_m), kBlock, 0, s>>>(
        n, m, op, FactorSide{rx.get(), rsf.get(), iv.get(), cum_v.get()},
        FactorSide{cx.get(), csf.get(), ic.get(), cum_c.get()}, p->c.get(), p->l.get(), p->u.get(), p->b.get());
    if (m) scale_matrix_kernel<<<gw_m, kBlock, 0, s>>>(m, lm, p->A.row_ptr.get(), p->A.col.get(), p->A.val64.get(),
                                                       ic.get(), iv.get(), 0, cx.get());
    scale_matrix_kernel<<<gw_n, kBlock, 0, s>>>(n, ln, p->At.row_ptr.get(), p->At.col.get(), p->At.val64.get(),
                                                ic.get(), iv.get(), 1, rx.get());
    CK_LAUNCH();
    have_max = true;
  };
  auto maxima = [&](DBuf<double>& cols, DBuf<double>& rows) {
    row_reduce_kernel<kRowAbsMax><<<gw_n, kBlock, 0, s>>>(n, ln, p->At.row_ptr.get(), p->At.val64.get(), 0.0, nullptr,
                                                          cols.get());
    if (m) row_reduce_kernel<kRowAbsMax><<<gw_m, kBlock, 0, s>>>(m, lm, p->A.row_ptr.get(), p->A.val64.get(), 0.0,
                                                                 nullptr, rows.get());
    CK_LAUNCH();
  };
  auto reset_cum = [&]() {
    fill_kernel<<<ge_n, kBlock, 0, s>>>(n, 1.0, cum_v.get());
    if (m) fill_kernel<<<ge_m, kBlock, 0, s>>>(m, 1.0, cum_c.get());
    CK_LAUNCH();
  };
  // total *= cum (the reference multiplies each stage's cumulative vector in)
  auto stage_total = [&]() {
    accumulate_kernel<<<ge_n, kBlock, 0, s>>>(n, cum_v.get(), p->var.get());
    if (m) accumulate_kernel<<<ge_m, kBlock, 0, s>>>(m, cum_c.get(), p->con.get());
    CK_LAUNCH();
  };
  // ruiz_rescaling with p = Inf (:398-463): D_j = sqrt(max_i |a_ij|), E_i = sqrt(max_j |a_ij|)
  if (prm.l_inf_ruiz_iterations > 0) {
    reset_cum();
    maxima(rx, cx);
    for (int it = 0; it < prm.l_inf_ruiz_iterations; ++it) apply(kFactorSqrt);
    stage_total();
  }
  // l2_norm_rescaling: rows and columns scaled by sqrt of their 2-norms
  if (prm.l2_norm_rescaling) {
    reset_cum();
    maxima(rsf, csf);
    unit_if_zero_kernel<<<ge_n, kBlock, 0, s>>>(n, rsf.get());
    if (m) unit_if_zero_kernel<<<ge_m, kBlock, 0, s>>>(m, csf.get());
    row_reduce_kernel<kRowScaledSq><<<gw_n, kBlock, 0, s>>>(n, ln, p->At.row_ptr.get(), p->At.val64.get(), 0.0,
                                                            rsf.get(), rx.get());
    if (m) row_reduce_kernel<kRowScaledSq><<<gw_m, kBlock, 0, s>>>(m, lm, p->A.row_ptr.get(), p->A.val64.get(), 0.0,
                                                                   csf.get(), cx.get());
    CK_LAUNCH();
    apply(kFactorL2);
    stage_total();
  }
  // pock_chambolle_rescaling (:494-525): D_j = sqrt(sum_i |a_ij|^(2-alpha)), E_i = sqrt(sum_j |a_ij|^alpha)
  if (!std::isnan(prm.pock_chambolle_alpha)) {
    const double alpha = prm.pock_chambolle_alpha;
    if (!(alpha >= 0.0 && alpha <= 2.0))
      throw Error(GPDHG_ERR_INVALID_ARGUMENT, "pock_chambolle_alpha must lie in [0, 2]");
    reset_cum();
    row_reduce_kernel<kRowPowSum><<<gw_n, kBlock, 0, s>>>(n, ln, p->At.row_ptr.get(), p->At.val64.get(), 2.0 - alpha,
                                                          nullptr, rx.get());
    if (m) row_reduce_kernel<kRowPowSum><<<gw_m, kBlock, 0, s>>>(m, lm, p->A.row_ptr.get(), p->A.val64.get(), alpha,
                                                                 nullptr, cx.get());
    CK_LAUNCH();
    apply(kFactorSqrt);
    stage_total();
  }
  // host scalars of the scaled problem, as problem_init derives them from a scaled descriptor:
  // tau_0 = 1 / max|a_ij| (:571) from the column maxima, and the norms of
  // select_initial_primal_weight, summed in order on the host
  if (!have_max) maxima(rx, cx);
  max_kernel<<<1, 1024, 0, s>>>(n, rx.get(), amax.get());
  CK_LAUNCH();
  std::vector<double> hc(N), hb(M);
  double largest = 0.0;
  CK(cudaMemcpyAsync(&largest, amax.get(), sizeof(double), cudaMemcpyDeviceToHost, s));
  CK(cudaMemcpyAsync(hc.data(), p->c.get(), sizeof(double) * n, cudaMemcpyDeviceToHost, s));
  if (m) CK(cudaMemcpyAsync(hb.data(), p->b.get(), sizeof(double) * m, cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  double sc = 0.0, sb = 0.0;
  for (int j = 0; j < n; ++j) sc += hc[j] * hc[j];
  for (int i = 0; i < m; ++i) sb += hb[i] * hb[i];
  p->amax = largest;
  p->norm2_c_scaled = std::sqrt(sc);
  p->norm2_b_scaled = m ? std::sqrt(sb) : 0.0;
}

void get_rescaling(const gpdhg_problem* p, double* con, double* var) {
  if (con && p->m)
    CK(cudaMemcpyAsync(con, p->con.get(), sizeof(double) * p->m, cudaMemcpyDeviceToHost, p->stream));
  if (var) CK(cudaMemcpyAsync(var, p->var.get(), sizeof(double) * p->n, cudaMemcpyDeviceToHost, p->stream));
  CK(cudaStreamSynchronize(p->stream));
}

}  // namespace gpdhg
