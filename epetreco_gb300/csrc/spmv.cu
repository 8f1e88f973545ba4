// spmv.cu -- CSR/CSC matrix-vector products and the MLEM element-wise ops.
//
// Replaces cusparseScsrmv (csrmv.hpp:25-36; called at reco.cu:236-249 and
// backprojection.cu:136-138) and the thrust transforms of mlemOperations.hpp.
// The products are HBM-bound streams over (value, column) pairs: a group of
// G lanes owns one row, each lane keeps four independent accumulators so
// that eight loads per lane are in flight, and the matrix streams are read
// with evict-first hints so the gathered vector stays cache-resident.  The
// transpose reads the column-major copy (scatter-free, deterministic).
// Epilogues fuse the MLEM steps: the forward product writes e = y / (A x)
// and the Poisson log-likelihood terms; the transpose writes
// x*c/s (s == 0 -> 1) and the image sum, both reduced in fp64 with a fixed
// order (deterministic).
#include <algorithm>
#include <cstdlib>

#include "common.cuh"
#include "internal.h"
#include "rows.cuh"
#include "spmv.cuh"

namespace epet {

// Generic row kernel: out = Epi(row, dot) over tiles of kSpmvThreads / G
// rows; a grid smaller than the tile count strides over the tiles.  With
// partial, Epi's fp64 values are summed per tile into partial[tile].
template <int G, int U, bool VEC, class Epi>
__global__ void __launch_bounds__(kSpmvThreads)
k_rows(const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
       const float* __restrict__ val, const float* __restrict__ x, int64_t nrows, Epi epi,
       double* __restrict__ partial) {
  constexpr int RPT = kSpmvThreads / G;
  __shared__ double red[kSpmvThreads / 32];
  const int lg = threadIdx.x % G;
  const int64_t ntiles = (nrows + RPT - 1) / RPT;
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t row = tile * RPT + threadIdx.x / G;
    double part = 0.0;
    if (row < nrows) {
      const float d =
          row_dot<G, U, VEC>(idx, val, x, ptr[row], ptr[row + 1], lg, group_mask<G>());
      if (lg == 0) part = epi(row, d);
    }
    if (partial) block_sum_to(part, red, partial + tile);
  }
}

// The same with every value 1 (out = Epi(row, sum of x over the row's
// indices)): the grouped layout's per-column sums over its slots.
template <int G, int U, bool VEC, class Epi>
__global__ void __launch_bounds__(kSpmvThreads)
k_sums(const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
       const float* __restrict__ x, int64_t nrows, Epi epi, double* __restrict__ partial) {
  constexpr int RPT = kSpmvThreads / G;
  __shared__ double red[kSpmvThreads / 32];
  const int lg = threadIdx.x % G;
  const int64_t ntiles = (nrows + RPT - 1) / RPT;
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t row = tile * RPT + threadIdx.x / G;
    double part = 0.0;
    if (row < nrows) {
      const float d = row_sum<G, U, VEC>(idx, x, ptr[row], ptr[row + 1], lg, group_mask<G>());
      if (lg == 0) part = epi(row, d);
    }
    if (partial) block_sum_to(part, red, partial + tile);
  }
}

// y0, y1 = alpha A x + beta y for two vectors stored pairwise.
template <int G, int U, bool VEC>
__global__ void __launch_bounds__(kSpmvThreads)
k_rows_pair(const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
            const float* __restrict__ val, const float2* __restrict__ x, int64_t nrows,
            float alpha, float beta, float* __restrict__ y0, float* __restrict__ y1) {
  constexpr int RPT = kSpmvThreads / G;
  const int lg = threadIdx.x % G;
  const int64_t ntiles = (nrows + RPT - 1) / RPT;
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t row = tile * RPT + threadIdx.x / G;
    if (row >= nrows) continue;
    float2 d;
    if constexpr (VEC)
      d = group_dot2_vec<G, U>(idx, val, x, ptr[row], ptr[row + 1], lg, group_mask<G>());
    else
      d = group_dot2_scalar<G>(idx, val, x, ptr[row], ptr[row + 1], lg, group_mask<G>());
    if (lg == 0) {
      y0[row] = beta == 0.f ? alpha * d.x : alpha * d.x + beta * y0[row];
      y1[row] = beta == 0.f ? alpha * d.y : alpha * d.y + beta * y1[row];
    }
  }
}

// Fixed-order sum of the block partials.
__global__ void k_sum_partials(const double* __restrict__ p, int64_t n, double* out) {
  __shared__ double red[32];
  double s = 0.0;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) s += p[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x / 32); w++) t += red[w];
    *out = t;
  }
}

struct EpiAxpby {  // y = alpha*d + beta*y
  float alpha, beta;
  float* y;
  __device__ double operator()(int64_t r, float d) const {
    y[r] = beta == 0.f ? alpha * d : alpha * d + beta * y[r];
    return 0.0;
  }
};

int pick_group(double avg_len) {
  if (avg_len >= 48) return 32;
  if (avg_len >= 24) return 16;
  if (avg_len >= 12) return 8;
  return 4;
}

RowPlan default_plan(double avg_len) {
  RowPlan p;
  p.G = pick_group(avg_len);
  p.U = 2;
  p.grid = 0;
  return p;
}

template <class Epi>
epet_status launch_rows(const RowPlan& plan, const int64_t* ptr, const int32_t* idx,
                        const float* val, const float* x, int64_t nrows, Epi epi,
                        double* partial, cudaStream_t st) {
  if (nrows <= 0) return EPET_OK;
  const int64_t nt = plan_tiles(plan, nrows);
  const unsigned grid = (unsigned)(plan.grid > 0 ? std::min<int64_t>(nt, plan.grid) : nt);
  // 16-byte loads only when both streams start on a 16-byte boundary
  dispatch_plan(plan, aligned16(idx, val), [&](auto g, auto u, auto v) {
    k_rows<decltype(g)::value, decltype(u)::value, decltype(v)::value, Epi>
        <<<grid, kSpmvThreads, 0, st>>>(ptr, idx, val, x, nrows, epi, partial);
  });
  EPET_LAUNCHED();
  return EPET_OK;
}

template <class Epi>
epet_status launch_sums(const RowPlan& plan, const int64_t* ptr, const int32_t* idx,
                        const float* x, int64_t nrows, Epi epi, double* partial,
                        cudaStream_t st) {
  if (nrows <= 0) return EPET_OK;
  const int64_t nt = plan_tiles(plan, nrows);
  const unsigned grid = (unsigned)(plan.grid > 0 ? std::min<int64_t>(nt, plan.grid) : nt);
  dispatch_plan(plan, aligned16(idx, idx), [&](auto g, auto u, auto v) {
    k_sums<decltype(g)::value, decltype(u)::value, decltype(v)::value, Epi>
        <<<grid, kSpmvThreads, 0, st>>>(ptr, idx, x, nrows, epi, partial);
  });
  EPET_LAUNCHED();
  return EPET_OK;
}
template epet_status launch_sums<EpiMlemUpdate>(const RowPlan&, const int64_t*, const int32_t*,
                                                const float*, int64_t, EpiMlemUpdate, double*,
                                                cudaStream_t);
template epet_status launch_sums<EpiKeep>(const RowPlan&, const int64_t*, const int32_t*,
                                          const float*, int64_t, EpiKeep, double*, cudaStream_t);

template epet_status launch_rows<EpiMlemForward>(const RowPlan&, const int64_t*, const int32_t*,
                                                 const float*, const float*, int64_t,
                                                 EpiMlemForward, double*, cudaStream_t);
template epet_status launch_rows<EpiMlemUpdate>(const RowPlan&, const int64_t*, const int32_t*,
                                                const float*, const float*, int64_t,
                                                EpiMlemUpdate, double*, cudaStream_t);
template epet_status launch_rows<EpiKeep>(const RowPlan&, const int64_t*, const int32_t*,
                                           const float*, const float*, int64_t, EpiKeep,
                                           double*, cudaStream_t);

epet_status launch_sum_partials(const double* p, int64_t n, double* out, cudaStream_t st) {
  k_sum_partials<<<1, 1024, 0, st>>>(p, n, out);
  EPET_LAUNCHED();
  return EPET_OK;
}

// Transpose by scatter (no CSC): y[col] += alpha * v * x[row].
__global__ void k_csr_scatter_t(const int64_t* __restrict__ ptr, const int32_t* __restrict__ col,
                                const float* __restrict__ val, const float* __restrict__ x,
                                int64_t m, float alpha, float* __restrict__ y) {
  const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= m) return;
  const float xr = alpha * x[row];
  if (xr == 0.f) return;
  for (int64_t k = ptr[row] + lane; k < ptr[row + 1]; k += 32)
    atomicAdd(&y[col[k]], val[k] * xr);
}

__global__ void k_scale_vec(float* y, int64_t n, float beta) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = beta == 0.f ? 0.f : beta * y[i];
}

// ------------------------------------------------------ element-wise ops
__global__ void k_divides(float* r, const float* a, const float* b, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) r[i] = fdiv(a[i], b[i]);
}
__global__ void k_divides_multiplies(float* r, const float* a, const float* b, const float* c,
                                     int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    float dvs = c[i];
    dvs = fadd(dvs, (float)(dvs == 0.f));
    r[i] = fdiv(fmul(a[i], b[i]), dvs);
  }
}
__global__ void k_scales(float* x, float alpha, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] = fmul(alpha, x[i]);
}
__global__ void k_sum_f64_part(const float* __restrict__ x, int64_t n,
                               double* __restrict__ partial) {
  __shared__ double red[8];
  double s = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    s += (double)x[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x / 32); w++) t += red[w];
    partial[blockIdx.x] = t;
  }
}

// x = xnew * float(1/sum)  (reco.cu:277-281: scales(x, val_t(1./norm)))
__global__ void k_normalise(const float* __restrict__ xnew, const double* __restrict__ sum,
                            int64_t n, float* __restrict__ x) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] = fmul((float)(1.0 / *sum), xnew[i]);
}

epet_status launch_normalise(const float* xnew, const double* sum, int64_t n, float* x,
                             cudaStream_t st) {
  k_normalise<<<ceil_div(n, 256), 256, 0, st>>>(xnew, sum, n, x);
  EPET_LAUNCHED();
  return EPET_OK;
}

// x = xnew * float(1/sum) with sum = the fixed-order sum of nb partials
// (every block reduces them in the same order, so all see the same value).
__global__ void k_normalise_parts(const float* __restrict__ xnew,
                                  const double* __restrict__ part, int nb, int64_t n,
                                  float* __restrict__ x) {
  __shared__ double red[8];
  __shared__ double tot;
  double s = 0.0;
  for (int i = threadIdx.x; i < nb; i += blockDim.x) s += part[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x / 32); w++) t += red[w];
    tot = t;
  }
  __syncthreads();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] = fmul((float)(1.0 / tot), xnew[i]);
}

int sum_blocks(int64_t n) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(ceil_div(n, 4096), 1024));
}

epet_status launch_sum_normalise(const float* xnew, int64_t n, double* part, float* x,
                                 cudaStream_t st) {
  const int nb = sum_blocks(n);
  k_sum_f64_part<<<nb, 256, 0, st>>>(xnew, n, part);
  EPET_LAUNCHED();
  k_normalise_parts<<<ceil_div(n, 256), 256, 0, st>>>(xnew, part, nb, n, x);
  EPET_LAUNCHED();
  return EPET_OK;
}

__global__ void k_loglik_part(const float* __restrict__ y, const float* __restrict__ yb,
                              int64_t m, double* __restrict__ partial) {
  __shared__ double red[8];
  double s = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double d = (double)yb[i];
    if (d > 0.0) s += (double)y[i] * log(d) - d;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x / 32); w++) t += red[w];
    partial[blockIdx.x] = t;
  }
}

epet_status poisson_loglik(const float* y, const float* ybar, int64_t m, double* partial,
                           int nblocks, double* out, cudaStream_t st) {
  k_loglik_part<<<nblocks, 256, 0, st>>>(y, ybar, m, partial);
  EPET_LAUNCHED();
  return launch_sum_partials(partial, nblocks, out, st);
}

epet_status sum_f64(const float* x, int64_t n, double* partial, int nblocks, double* out,
                    cudaStream_t st) {
  k_sum_f64_part<<<nblocks, 256, 0, st>>>(x, n, partial);
  EPET_LAUNCHED();
  return launch_sum_partials(partial, nblocks, out, st);
}

// Launch plan of a drop-in product (epet_csrmv): the autotuner's, timed once
// per matrix shape and process into a scratch output (so y = alpha A x +
// beta y is only computed once, by the caller's launch); the heuristic plan
// while the stream is being captured (no timing then) unless one is cached,
// and always with EPET_AUTOTUNE=0 in the environment (results then depend on
// the inputs alone).
static epet_status dropin_plan(int kind, const int64_t* ptr, const int32_t* idx,
                               const float* val, const float* x, int64_t nrows, int64_t nnz,
                               int64_t ncols, cudaStream_t st, RowPlan* out) {
  const double avg = nrows ? (double)nnz / nrows : 0.0;
  *out = default_plan(avg);
  static const bool off = [] {
    const char* e = getenv("EPET_AUTOTUNE");
    return e && e[0] == '0';
  }();
  if (off || nrows <= 0 || nnz <= 0) return EPET_OK;
  if (tune_lookup(kind, nrows, nnz, ncols, out)) return EPET_OK;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  EPET_CUDA(cudaStreamIsCapturing(st, &cs));
  if (cs != cudaStreamCaptureStatusNone) return EPET_OK;
  float* scratch = nullptr;
  EPET_CUDA(dev_alloc((void**)&scratch, nrows * 4, st));
  epet_status rc = tune_rows(
      kind, nrows, nnz, ncols, avg,
      [&](const RowPlan& pl) {
        return launch_rows(pl, ptr, idx, val, x, nrows, EpiAxpby{1.f, 0.f, scratch}, nullptr, st);
      },
      st, out);
  dev_free(scratch, st);
  return rc;
}

}  // namespace epet

using namespace epet;

extern "C" {

epet_status epet_csrmv(int trans, const epet_csr* a, const epet_csc* csc, float alpha,
                       const float* x_d, float beta, float* y_d, epet_stream_t stream) {
  if (!a) return set_error(EPET_ERR_INVALID, "bad arguments");
  const int64_t out_len = trans ? a->n : a->m, in_len = trans ? a->m : a->n;
  if ((out_len > 0 && !y_d) || (in_len > 0 && !x_d))
    return set_error(EPET_ERR_INVALID, "bad arguments");
  if (out_len == 0) return EPET_OK;
  cudaStream_t st = (cudaStream_t)stream;
  if (!trans) {
    RowPlan pl;
    EPET_CHECK(dropin_plan(2, a->row_ptr, a->col, a->val, x_d, a->m, a->nnz, a->n, st, &pl));
    return launch_rows(pl, a->row_ptr, a->col, a->val, x_d, a->m, EpiAxpby{alpha, beta, y_d},
                       nullptr, st);
  }
  if (csc) {
    RowPlan pl;
    EPET_CHECK(dropin_plan(3, csc->col_ptr, csc->row, csc->val, x_d, csc->n, csc->nnz, csc->m,
                           st, &pl));
    return launch_rows(pl, csc->col_ptr, csc->row, csc->val, x_d, csc->n,
                       EpiAxpby{alpha, beta, y_d}, nullptr, st);
  }
  if (beta != 1.f) {
    k_scale_vec<<<ceil_div(a->n, 256), 256, 0, st>>>(y_d, a->n, beta);
    EPET_LAUNCHED();
  }
  if (a->m > 0) {
    k_csr_scatter_t<<<ceil_div(a->m * 32, 256), 256, 0, st>>>(a->row_ptr, a->col, a->val, x_d,
                                                               a->m, alpha, y_d);
    EPET_LAUNCHED();
  }
  return EPET_OK;
}

epet_status epet_csrmv2(int trans, const epet_csr* a, const epet_csc* csc, float alpha,
                        const float* x_d, float beta, float* y0_d, float* y1_d,
                        epet_stream_t stream) {
  if (!a || (trans && !csc)) return set_error(EPET_ERR_INVALID, "bad arguments");
  const int64_t out_len = trans ? a->n : a->m, in_len = trans ? a->m : a->n;
  if ((out_len > 0 && (!y0_d || !y1_d)) || (in_len > 0 && !x_d) ||
      (reinterpret_cast<uintptr_t>(x_d) & 7) != 0)
    return set_error(EPET_ERR_INVALID, "bad arguments");
  const int64_t* ptr = trans ? csc->col_ptr : a->row_ptr;
  const int32_t* idx = trans ? csc->row : a->col;
  const float* val = trans ? csc->val : a->val;
  const int64_t nrows = trans ? csc->n : a->m, ncols = trans ? csc->m : a->n;
  if (nrows <= 0) return EPET_OK;
  cudaStream_t st = (cudaStream_t)stream;
  RowPlan pl;  // (tuned on the first elements of x_d as one vector)
  EPET_CHECK(dropin_plan(trans ? 3 : 2, ptr, idx, val, x_d, nrows, trans ? csc->nnz : a->nnz, ncols,
                         st, &pl));
  const int64_t nt = plan_tiles(pl, nrows);
  const unsigned grid = (unsigned)(pl.grid > 0 ? std::min<int64_t>(nt, pl.grid) : nt);
  dispatch_plan(pl, aligned16(idx, val), [&](auto g, auto u, auto v) {
    k_rows_pair<decltype(g)::value, decltype(u)::value, decltype(v)::value>
        <<<grid, kSpmvThreads, 0, st>>>(ptr, idx, val, reinterpret_cast<const float2*>(x_d), nrows,
                                        alpha, beta, y0_d, y1_d);
  });
  EPET_LAUNCHED();
  return EPET_OK;
}

epet_status epet_divides(float* r_d, const float* a_d, const float* b_d, int64_t n,
                         epet_stream_t stream) {
  if (n < 0 || (n > 0 && (!r_d || !a_d || !b_d)))
    return set_error(EPET_ERR_INVALID, "bad arguments");
  if (n == 0) return EPET_OK;
  k_divides<<<ceil_div(n, 256), 256, 0, (cudaStream_t)stream>>>(r_d, a_d, b_d, n);
  EPET_LAUNCHED();
  return EPET_OK;
}

epet_status epet_divides_multiplies(float* r_d, const float* a_d, const float* b_d,
                                    const float* c_d, int64_t n, epet_stream_t stream) {
  if (n < 0 || (n > 0 && (!r_d || !a_d || !b_d || !c_d)))
    return set_error(EPET_ERR_INVALID, "bad arguments");
  if (n == 0) return EPET_OK;
  k_divides_multiplies<<<ceil_div(n, 256), 256, 0, (cudaStream_t)stream>>>(r_d, a_d, b_d, c_d,
                                                                            n);
  EPET_LAUNCHED();
  return EPET_OK;
}

epet_status epet_scales(float* x_d, float alpha, int64_t n, epet_stream_t stream) {
  if (n < 0 || (n > 0 && !x_d)) return set_error(EPET_ERR_INVALID, "bad arguments");
  if (n == 0) return EPET_OK;
  k_scales<<<ceil_div(n, 256), 256, 0, (cudaStream_t)stream>>>(x_d, alpha, n);
  EPET_LAUNCHED();
  return EPET_OK;
}

epet_status epet_sum_f64(const float* x_d, int64_t n, double* out_d, epet_stream_t stream) {
  if (n < 0 || !out_d || (n > 0 && !x_d)) return set_error(EPET_ERR_INVALID, "bad arguments");
  cudaStream_t st = (cudaStream_t)stream;
  const int nb = (int)std::max<int64_t>(1, std::min<int64_t>(ceil_div(n, 256), 1024));
  double* part = nullptr;
  EPET_CUDA(dev_alloc((void**)&part, nb * 8, st));
  epet_status rc = sum_f64(x_d, n, part, nb, out_d, st);
  dev_free(part, st);
  return rc;
}

}  // extern "C"
