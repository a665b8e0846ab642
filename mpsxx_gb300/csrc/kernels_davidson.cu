// Vector algebra of one Davidson problem, fused around its reductions.  The basis is kept
// as it was orthonormalised (no rotation to Ritz vectors): one product of the new vector
// with every H_eff * trial gives the subspace matrix's new row, and one pass over the basis
// gives residual, its norm, the preconditioned correction and its projections.
//
// Bound by latency at small n and by the FP64 pipe at large n (2.1 FMA per clock and SM,
// about 3 m + 15 operations per element and iteration): a launch is at most 304 CTAs of 128
// threads whose sums are added in a fixed order by the last CTA to arrive, so that no second
// kernel is needed, and launches are chained.  Sums the host reads are written to mapped host
// memory as well.  An iteration took 25 launches with rotations and separate reductions on
// n / 2048 CTAs: 45 us per dot product at n = 16 k, now 4 us.
#include <cuda_runtime.h>

#include "kernels.hpp"
#include "launch.hpp"

namespace mpsxx {

namespace {

constexpr int DT = 128;            // threads
constexpr int NVMAX = kMaxDot + 2;  // sums of one launch
constexpr int PER = 8;             // threads that add one sum
static_assert(NVMAX * PER <= DT, "a sum's threads");

// acc[0..nv) summed over all threads of the grid into out (and host) in a fixed order.
__device__ void grid_sums(const double (&acc)[NVMAX], int nv, const DvReduce& rd) {
  __shared__ double s[NVMAX][DT + 1];
  __shared__ bool last;
  const int t = threadIdx.x, v = t / PER, sub = t % PER;
#pragma unroll
  for (int i = 0; i < NVMAX; ++i)
    if (i < nv) s[i][t] = acc[i];
  __syncthreads();
  double x = 0.0;
  if (v < nv)
    for (int k = sub; k < DT; k += PER) x += s[v][k];
  for (int o = PER / 2; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o, PER);
  if (v < nv && sub == 0) rd.partial[blockIdx.x * NVMAX + v] = x;
  __threadfence();
  __syncthreads();
  if (t == 0) last = atomicAdd(rd.ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  x = 0.0;
  if (v < nv)
    for (int b = sub; b < (int)gridDim.x; b += PER) x += __ldcg(rd.partial + b * NVMAX + v);
  for (int o = PER / 2; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o, PER);
  if (v < nv && sub == 0) {
    rd.out[v] = x;
    if (rd.host != nullptr) {
      *const_cast<volatile double*>(rd.host + v) = x;
      __threadfence_system();
    }
  }
  if (t == 0) *rd.ticket = 0;
}

// out[j] = x . Y_j, j < m
__global__ void __launch_bounds__(DT) dv_dots_kernel(const double* __restrict__ x, const double* __restrict__ Y, int m,
                                                     int64_t n, DvReduce rd) {
  chain_wait();
  chain_next();
  double acc[NVMAX] = {};
  for (int64_t e = blockIdx.x * (int64_t)DT + threadIdx.x; e < n; e += (int64_t)gridDim.x * DT) {
    const double a = x[e];
#pragma unroll
    for (int j = 0; j < kMaxDot; ++j)
      if (j < m) acc[j] = fma(a, Y[j * n + e], acc[j]);
  }
  grid_sums(acc, m, rd);
}

// With t = sum_i r_i T_i, s = sum_i r_i S_i: res = s - e t, c = res / (e - diag);
// out = [|res|^2, |c|^2, T_i . c]
__global__ void __launch_bounds__(DT) dv_residual_kernel(const double* __restrict__ T, const double* __restrict__ S,
                                                         const double* __restrict__ diag, int m, int64_t n, DvCoef r,
                                                         double e, double* __restrict__ c, DvReduce rd) {
  chain_wait();
  chain_next();
  double acc[NVMAX] = {};
  for (int64_t i = blockIdx.x * (int64_t)DT + threadIdx.x; i < n; i += (int64_t)gridDim.x * DT) {
    double tv[kMaxDot], t = 0.0, s = 0.0;
#pragma unroll
    for (int j = 0; j < kMaxDot; ++j)
      if (j < m) {
        tv[j] = T[j * n + i];
        t = fma(r.v[j], tv[j], t);
        s = fma(r.v[j], S[j * n + i], s);
      }
    const double res = fma(-e, t, s);
    double den = e - diag[i];
    if (fabs(den) < 1.0e-8) den = 1.0e-8;
    const double cv = res / den;
    c[i] = cv;
    acc[0] = fma(res, res, acc[0]);
    acc[1] = fma(cv, cv, acc[1]);
#pragma unroll
    for (int j = 0; j < kMaxDot; ++j)
      if (j < m) acc[2 + j] = fma(tv[j], cv, acc[2 + j]);
  }
  grid_sums(acc, m + 2, rd);
}

// One pass of classical Gram-Schmidt: c <- f (c - sum_i p_i T_i) with f = 1 / sqrt(in[1]) in
// the first pass (p = in[2..]), 1 in the second (p = in[0..]).  out: the projections T_i . c
// of the new c (first pass), |c|^2 (second pass).
__global__ void __launch_bounds__(DT) dv_project_kernel(const double* __restrict__ T, int m, int64_t n,
                                                        double* __restrict__ c, const double* __restrict__ in, int second,
                                                        DvReduce rd) {
  chain_wait();
  chain_next();
  double acc[NVMAX] = {}, p[kMaxDot];
  const double f = second ? 1.0 : 1.0 / sqrt(in[1]);
#pragma unroll
  for (int j = 0; j < kMaxDot; ++j) p[j] = j < m ? (second ? in[j] : f * in[2 + j]) : 0.0;
  for (int64_t i = blockIdx.x * (int64_t)DT + threadIdx.x; i < n; i += (int64_t)gridDim.x * DT) {
    double tv[kMaxDot], v = f * c[i];
#pragma unroll
    for (int j = 0; j < kMaxDot; ++j)
      if (j < m) {
        tv[j] = T[j * n + i];
        v = fma(-p[j], tv[j], v);
      }
    c[i] = v;
    if (second) {
      acc[0] = fma(v, v, acc[0]);
    } else {
#pragma unroll
      for (int j = 0; j < kMaxDot; ++j)
        if (j < m) acc[j] = fma(tv[j], v, acc[j]);
    }
  }
  grid_sums(acc, second ? 1 : m, rd);
}

// t = x / sqrt(in[0]) (t may be x); z = 0 (z may be null)
__global__ void __launch_bounds__(DT) dv_scaled_copy_kernel(const double* x, int64_t n, const double* __restrict__ in,
                                                            double* t, double* __restrict__ z) {
  chain_wait();
  chain_next();
  const double f = 1.0 / sqrt(in[0]);
  for (int64_t i = blockIdx.x * (int64_t)DT + threadIdx.x; i < n; i += (int64_t)gridDim.x * DT) {
    t[i] = f * x[i];
    if (z != nullptr) z[i] = 0.0;
  }
}

// out = sum_i r_i T_i (out may be T_0)
__global__ void __launch_bounds__(DT) dv_combine_kernel(const double* T, int m, int64_t n, DvCoef r, double* out) {
  chain_wait();
  chain_next();
  for (int64_t i = blockIdx.x * (int64_t)DT + threadIdx.x; i < n; i += (int64_t)gridDim.x * DT) {
    double t = 0.0;
#pragma unroll
    for (int j = 0; j < kMaxDot; ++j)
      if (j < m) t = fma(r.v[j], T[j * n + i], t);
    out[i] = t;
  }
}

int dv_blocks(int64_t n) {
  const int64_t b = (n + DT - 1) / DT;
  return static_cast<int>(b < 1 ? 1 : b > kMultidotMaxBlocks ? kMultidotMaxBlocks : b);
}

}  // namespace

size_t dv_partial_doubles() { return size_t(kMultidotMaxBlocks) * NVMAX; }

void launch_dv_dots(const double* x, const double* Y, int m, int64_t n, const DvReduce& rd, cudaStream_t st) {
  launch_chained(dv_dots_kernel, dim3(dv_blocks(n)), DT, 0, st, x, Y, m, n, rd);
}

void launch_dv_residual(const double* T, const double* S, const double* diag, int m, int64_t n, const DvCoef& r,
                        double e, double* c, const DvReduce& rd, cudaStream_t st) {
  launch_chained(dv_residual_kernel, dim3(dv_blocks(n)), DT, 0, st, T, S, diag, m, n, r, e, c, rd);
}

void launch_dv_project(const double* T, int m, int64_t n, double* c, const double* in, int second, const DvReduce& rd,
                       cudaStream_t st) {
  launch_chained(dv_project_kernel, dim3(dv_blocks(n)), DT, 0, st, T, m, n, c, in, second, rd);
}

void launch_dv_scaled_copy(const double* x, int64_t n, const double* in, double* t, double* z, cudaStream_t st) {
  launch_chained(dv_scaled_copy_kernel, dim3(dv_blocks(n)), DT, 0, st, x, n, in, t, z);
}

void launch_dv_combine(const double* T, int m, int64_t n, const DvCoef& r, double* out, cudaStream_t st) {
  launch_chained(dv_combine_kernel, dim3(dv_blocks(n)), DT, 0, st, T, m, n, r, out);
}

}  // namespace mpsxx
