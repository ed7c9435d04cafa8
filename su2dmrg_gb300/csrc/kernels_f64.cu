// FP64 kernels of the hot path:
//   * gemm_f64_tiles: the block-sparse contraction engine (one CTA per tile of
//     the work list, gemm_work.hpp), FP64 tensor-core MMA
//     (mma.sync.m8n8k4.f64) fed from global memory through L1;
//   * gemm_f64_dense: dense products with the same tile code;
//   * deterministic BLAS-1 (dot, axpy, scale) for the Lanczos iteration.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <map>
#include <mutex>
#include <type_traits>

#include "gemm_work.hpp"
#include "kernels.hpp"
#include "overlap.cuh"

namespace su2g {
namespace {

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;

__device__ __forceinline__ void dmma_m8n8k4(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// sacc = op(A) B over the steps [step0, step1) of 4 contracted values of one
// segment, for nj 8 x 8 fragments side by side: this lane reads row `row` of
// op(A) and the columns col[j] of B.
//
// Bound by the FP64 pipe: GB300 does about two multiply-adds per clock and SM,
// so one m8n8k4 occupies an SM for 128 clocks while its operands are 512 bytes.
// Every warp therefore reads its fragments straight from global memory (a few
// bytes per clock and SM through L1 and L2): no staging, no barriers, and no
// work for padding beyond a fragment's edge.  Four steps of loads are in
// flight before the MMAs that use them; other warps cover the latency.  At
// D = 2000, 18 terms, an application takes 131.7 ms (1.066 TFLOP/s, 0.97 of
// cuBLAS DGEMM's 1.10); 64 x 64 tiles staged in shared memory took 153 ms, the
// difference being the work done for their padding.
//
// Rows and columns past the block are clamped to it and feed only entries
// that are never stored; values past K are zero in both operands.
template <int FN>
__device__ __forceinline__ void seg_mma(const GemmSeg& g, const Bases& bases, int row, const int (&col)[FN], int nj,
                                        int step0, int step1, int fc, int64_t zero, double (&sacc)[FN][2]) {
  constexpr int U = 4;
#pragma unroll
  for (int j = 0; j < FN; ++j) sacc[j][0] = sacc[j][1] = 0.0;
  const int64_t ks = g.transA ? 1 : g.lda;  // distance of neighbouring k in A
  const int k = step0 * 4 + fc;
  const double* ap = after_wait(resolve(bases, g.a_buf, g.a), zero) + (g.transA ? (int64_t)row * g.lda : row) + k * ks;
  const double* bp[FN];
#pragma unroll
  for (int j = 0; j < FN; ++j) bp[j] = after_wait(resolve(bases, g.b_buf, g.b), zero) + (int64_t)col[j] * g.ldb + k;
  int step = step0;
  const int full = min(step1, g.K / 4);
  for (; step + U <= full; step += U) {
    double a[U], b[U][FN];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      a[u] = ap[4 * u * ks];
#pragma unroll
      for (int j = 0; j < FN; ++j) b[u][j] = j < nj ? bp[j][4 * u] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int j = 0; j < FN; ++j)
        if (j < nj) dmma_m8n8k4(sacc[j], a[u], b[u][j]);
    ap += 4 * U * ks;
#pragma unroll
    for (int j = 0; j < FN; ++j) bp[j] += 4 * U;
  }
  for (; step < step1; ++step) {  // the last steps one by one, the very last perhaps past K
    const bool ok = step * 4 + fc < g.K;
    const double a = ok ? *ap : 0.0;
#pragma unroll
    for (int j = 0; j < FN; ++j) {
      const double b = (ok && j < nj) ? *bp[j] : 0.0;
      if (j < nj) dmma_m8n8k4(sacc[j], a, b);
      bp[j] += 4;
    }
    ap += 4 * ks;
  }
}

template <int FN>
__device__ __forceinline__ void add_scaled(double alpha, const double (&sacc)[FN][2], double (&acc)[FN][2]) {
#pragma unroll
  for (int j = 0; j < FN; ++j) {
    acc[j][0] += alpha * sacc[j][0];
    acc[j][1] += alpha * sacc[j][1];
  }
}

// The sub-tile of t at rows m1.. and columns n1.., C = sum_s alpha_s op(A_s)
// B_s, by WM x WN warps of FN fragments side by side: every segment is
// accumulated on its own, scaled by its alpha and added (the reference scales
// each block product by its recoupling factor before summing,
// tensor_su2_dmrg_src.cpp:997-1004).  Only fragments that hold rows and
// columns of the block are computed.  Every element sums its products in k
// order whatever the tile shape.
template <int FN, int WM, int WN>
__device__ __forceinline__ void sub_tile(const GemmTile& t, int m1, int n1, const GemmSeg* __restrict__ segs,
                                         const Bases& bases, int64_t zero) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wr = warp % WM, wc = warp / WM;
  const int fr = lane >> 2, fc = lane & 3;
  const int mlen = min(WM * 8, t.mlen - m1), nlen = min(WN * FN * 8, t.nlen - n1);
  const int nj = ((nlen + 7) / 8 - wc + WN - 1) / WN;  // fragments are dealt to the warps in turn
  if (wr * 8 >= mlen || nj <= 0) return;
  const int row = t.m0 + m1 + min(wr * 8 + fr, mlen - 1);
  int col[FN];
#pragma unroll
  for (int j = 0; j < FN; ++j) col[j] = t.n0 + n1 + min((wc + WN * j) * 8 + fr, nlen - 1);
  double acc[FN][2] = {};
  for (int s = t.seg0; s < t.seg0 + t.nseg; ++s) {
    const GemmSeg g = segs[s];
    double sacc[FN][2];
    seg_mma<FN>(g, bases, row, col, nj, 0, (g.K + 3) / 4, fc, zero, sacc);
    add_scaled<FN>(g.alpha, sacc, acc);
  }
  double* C = resolve(bases, t.c_buf, t.c);
  const int r = wr * 8 + fr;
  if (r >= mlen) return;
#pragma unroll
  for (int j = 0; j < FN; ++j)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int c = (wc + WN * j) * 8 + 2 * fc + q;
      if (c < nlen) C[(int64_t)(t.m0 + m1 + r) + (int64_t)(t.n0 + n1 + c) * t.ldc] = acc[j][q];
    }
}

// One output tile of one 8 x 8 fragment whose contraction is dealt to the eight
// warps: the steps of all its segments, laid end to end, in eight equal runs.
// The eight partial tiles are summed through shared memory in run order.
__global__ void __launch_bounds__(kThreads, 4) gemm_f64_ksplit(const GemmTile* __restrict__ tiles,
                                                               const GemmSeg* __restrict__ segs, Bases bases) {
  __shared__ double part[kWarps * 64];
  const GemmTile t = tiles[blockIdx.x];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int fr = lane >> 2, fc = lane & 3;
  const int row = t.m0 + min(fr, t.mlen - 1), col[1] = {t.n0 + min(fr, t.nlen - 1)};
  double acc[1][2] = {};
  int total = 0;  // steps of 4 over all segments
  for (int s = lane; s < t.nseg; s += 32) total += (segs[t.seg0 + s].K + 3) / 4;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
  const int lo = (int)((int64_t)total * warp / kWarps), hi = (int)((int64_t)total * (warp + 1) / kWarps);
  const int64_t zero = wait_for_predecessor();
  for (int s0 = 0, base = 0; s0 < t.nseg && base < hi; s0 += 32) {
    const int n = s0 + lane < t.nseg ? (segs[t.seg0 + s0 + lane].K + 3) / 4 : 0;
    int end = n;  // inclusive prefix sum
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, end, o);
      if (lane >= o) end += v;
    }
    end += base;
    unsigned mine = __ballot_sync(0xffffffffu, n > 0 && end > lo && end - n < hi);
    while (mine) {
      const int b = __ffs(mine) - 1;
      mine &= mine - 1;
      const int e1 = __shfl_sync(0xffffffffu, end, b), e0 = e1 - __shfl_sync(0xffffffffu, n, b);
      const GemmSeg g = segs[t.seg0 + s0 + b];
      double sacc[1][2];
      seg_mma<1>(g, bases, row, col, 1, max(lo - e0, 0), min(hi, e1) - e0, fc, zero, sacc);
      add_scaled<1>(g.alpha, sacc, acc);
    }
    base = __shfl_sync(0xffffffffu, end, 31);
  }
  // Not earlier: the next launch's CTAs would take whatever slots are free, four
  // heavy ones on one SM while others idle, instead of spreading (an
  // application at D = 123: 38 us, with nothing overlapped 28, like this 23).
  dependents_may_start();
  part[warp * 64 + lane] = acc[0][0];
  part[warp * 64 + 32 + lane] = acc[0][1];
  __syncthreads();
  if (threadIdx.x < 64) {
    const int e = threadIdx.x, l = e & 31;
    const int r = l >> 2, c = 2 * (l & 3) + (e >> 5);
    if (r < t.mlen && c < t.nlen) {
      double v = 0.0;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) v += part[w * 64 + e];
      resolve(bases, t.c_buf, t.c)[(int64_t)(t.m0 + r) + (int64_t)(t.n0 + c) * t.ldc] = v;
    }
  }
}

// One CTA per whole tile of the work list, 32 x 32 at a time.  (The dependents
// start as the CTAs end, for the reason given above.)
__global__ void __launch_bounds__(kThreads, 4) gemm_f64_tiles(const GemmTile* __restrict__ tiles,
                                                              const GemmSeg* __restrict__ segs, Bases bases) {
  const GemmTile t = tiles[blockIdx.x];
  const int64_t zero = wait_for_predecessor();
  for (int m1 = 0; m1 < t.mlen; m1 += 32)
    for (int n1 = 0; n1 < t.nlen; n1 += 32) sub_tile<2, 4, 2>(t, m1, n1, segs, bases, zero);
}

// One dense product C = op(A) B in tiles of WM x WN FN fragments, the tile at
// (bx, by) and its segment formed from the kernel's arguments (no work list to
// upload): the same tile code, so the same sums in the same order as a
// work-list launch of unsplit tiles.
template <int FN, int WM, int WN>
__device__ __forceinline__ void dense_tile(const DenseGemm& d, int bx, int by) {
  GemmSeg g;
  g.a = (int64_t)((uintptr_t)d.A / 8);
  g.b = (int64_t)((uintptr_t)d.B / 8);
  g.a_len = 0;
  g.b_len = 0;
  g.a_buf = g.b_buf = kBufAbs;
  g.lda = d.lda;
  g.ldb = d.ldb;
  g.K = d.K;
  g.transA = d.transA;
  g.alpha = 1.0;
  GemmTile t;
  t.c = (int64_t)((uintptr_t)d.C / 8);
  t.c_len = 0;
  t.c_buf = kBufAbs;
  t.ldc = d.ldc;
  t.m0 = bx * (WM * 8);
  t.n0 = by * (WN * FN * 8);
  t.mlen = min(WM * 8, d.M - t.m0);
  t.nlen = min(WN * FN * 8, d.N - t.n0);
  t.seg0 = 0;
  t.nseg = 1;
  t.kwork = d.K;
  t.cls = 0;
  t.ksplit = 0;
  sub_tile<FN, WM, WN>(t, 0, 0, &g, Bases{}, 0);
}

// Several products in one launch: a truncation takes three for every sector and
// refinement level, each a few microseconds' work for a few dozen CTAs.
constexpr int kDenseMost = 48;  // 3.3 KB of parameters
struct DenseList {
  DenseGemm job[kDenseMost];
  int first[kDenseMost];  // the job's first tile
};
template <int FN, int WM, int WN>
__global__ void __launch_bounds__(WM * WN * 32) gemm_f64_dense(const __grid_constant__ DenseList list, int njobs) {
  int j = 0;
  while (j + 1 < njobs && list.first[j + 1] <= (int)blockIdx.x) ++j;
  const int tile = blockIdx.x - list.first[j], across = (list.job[j].M + WM * 8 - 1) / (WM * 8);
  dense_tile<FN, WM, WN>(list.job[j], tile % across, tile / across);
}

}  // namespace

// Tiles of 32 x 32 once they fill the SMs three times over, else of 16 x 16
// (the same sums): the operands' traffic is no bound at either size, idle SMs
// are.
cudaError_t launch_gemm_f64_dense_many(const DenseGemm* jobs, int njobs, cudaStream_t stream) {
  auto tiles = [](const DenseGemm& d, int side) {
    return (int64_t)((d.M + side - 1) / side) * ((d.N + side - 1) / side);
  };
  int64_t total = 0;
  for (int j = 0; j < njobs; ++j) total += tiles(jobs[j], 32);
  const int side = total >= 3 * kF64Sms ? 32 : 16;
  for (int j = 0; j < njobs;) {
    DenseList list{};
    int n = 0;
    int64_t first = 0;
    for (; j < njobs && n < kDenseMost; ++j) {
      if (jobs[j].M <= 0 || jobs[j].N <= 0) continue;
      if (n > 0 && first + tiles(jobs[j], side) > INT32_MAX) break;
      list.job[n] = jobs[j];
      list.first[n++] = (int)first;
      first += tiles(jobs[j], side);
    }
    if (n == 0) continue;
    if (side == 32) gemm_f64_dense<2, 4, 2><<<(unsigned)first, 256, 0, stream>>>(list, n);
    else gemm_f64_dense<1, 2, 2><<<(unsigned)first, 128, 0, stream>>>(list, n);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_gemm_f64_dense(bool transA, int M, int N, int K, const double* A, int lda, const double* B,
                                  int ldb, double* C, int ldc, cudaStream_t stream) {
  const DenseGemm d{transA, M, N, K, A, lda, B, ldb, C, ldc};
  return launch_gemm_f64_dense_many(&d, 1, stream);
}

cudaError_t launch_gemm_f64(const GemmTile* tiles, const F64Counts& n, const GemmSeg* segs, const Bases& bases,
                            cudaStream_t stream) {
  cudaError_t e = cudaSuccess;
  if (n.whole > 0) e = launch_overlapped(gemm_f64_tiles, dim3(n.whole), kThreads, 0, 0, stream, tiles, segs, bases);
  if (e == cudaSuccess && n.split > 0)
    e = launch_overlapped(gemm_f64_ksplit, dim3(n.split), kThreads, 0, 0, stream, tiles + n.whole, segs, bases);
  return e;
}

namespace {

// ---------------------------------------------------------------- BLAS-1 --
constexpr int kRedBlocks = 512;  // fixed: the summation order never depends on the device
constexpr int kRedThreads = 256;

// the sum of a block's values, valid in thread 0: sh[t] += sh[t + s] for
// s = 128 .. 1, the last five steps inside warp 0
__device__ __forceinline__ double block_sum(double v, double* sh) {
  const int tid = threadIdx.x;
  __syncthreads();  // sh may still be read from an earlier sum
  sh[tid] = v;
  __syncthreads();
#pragma unroll
  for (int s = kRedThreads / 2; s >= 32; s >>= 1) {
    if (tid < s) sh[tid] = v = v + sh[tid + s];
    __syncthreads();
  }
  if (tid < 32) {
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) v += __shfl_down_sync(0xffffffffu, v, s);
  }
  return v;
}

// a dot product's value from its kRedBlocks partial sums, in every thread
__device__ __forceinline__ double sum_partials(const double* part, double* sh) {
  double v = 0;
#pragma unroll
  for (int i = 0; i < kRedBlocks; i += kRedThreads) v += part[i + threadIdx.x];
  v = block_sum(v, sh);
  if (threadIdx.x == 0) sh[0] = v;
  __syncthreads();
  v = sh[0];
  return v;
}

// Elements of a block's share in order, four in flight: f(i, count) handles
// the elements i, i + stride, ..., count of them (four, or the last one by one).
template <class F>
__device__ __forceinline__ void grid_stride4(int64_t n, F f) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (; i + 3 * stride < n; i += 4 * stride) f(i, stride, std::integral_constant<int, 4>());
  for (; i < n; i += stride) f(i, stride, std::integral_constant<int, 1>());
}

__global__ void __launch_bounds__(kRedThreads) dot_partial(const double* x_in, const double* y_in, int64_t n, double* part) {
  __shared__ double sh[kRedThreads];
  dependents_may_start();
  const int64_t zero = wait_for_predecessor();
  const double *x = after_wait(x_in, zero), *y = after_wait(y_in, zero);
  double v = 0;
  grid_stride4(n, [&](int64_t i, int64_t stride, auto U) {
    double a[U.value], b[U.value];
#pragma unroll
    for (int u = 0; u < U.value; ++u) a[u] = x[i + u * stride], b[u] = y[i + u * stride];
#pragma unroll
    for (int u = 0; u < U.value; ++u) v += a[u] * b[u];
  });
  const double s = block_sum(v, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// x . x and x . y in one pass
__global__ void __launch_bounds__(kRedThreads) dot2_partial(const double* x_in, const double* y_in, int64_t n, double* part) {
  __shared__ double sh[kRedThreads];
  dependents_may_start();
  const int64_t zero = wait_for_predecessor();
  const double *x = after_wait(x_in, zero), *y = after_wait(y_in, zero);
  double v = 0, w = 0;
  grid_stride4(n, [&](int64_t i, int64_t stride, auto U) {
    double a[U.value], b[U.value];
#pragma unroll
    for (int u = 0; u < U.value; ++u) a[u] = x[i + u * stride], b[u] = y[i + u * stride];
#pragma unroll
    for (int u = 0; u < U.value; ++u) v += a[u] * a[u], w += a[u] * b[u];
  });
  const double s = block_sum(v, sh), t = block_sum(w, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = s, part[kRedBlocks + blockIdx.x] = t;
}

// out[b] = the value of the dot product whose partial sums are part[b kRedBlocks ..]
__global__ void __launch_bounds__(kRedThreads) dot_final(const double* part, double* out) {
  __shared__ double sh[kRedThreads];
  dependents_may_start();
  const int64_t zero = wait_for_predecessor();
  const double s = sum_partials(after_wait(part, zero) + blockIdx.x * kRedBlocks, sh);
  if (threadIdx.x == 0) out[blockIdx.x] = s;
}

// One update of the Lanczos recurrence and the reduction the next one needs:
//     c = the dot product whose partial sums are part_in;  *c_out = c
//     y -= c x0;  y -= (*c1) x1 (c1 null: not);  part_out = partial sums of y . z
// (z null: y . y).  Every block sums the 512 partials itself (4 KB from L2, in
// the order of dot_final), so a coefficient costs no launch and no round trip
// of its own.  Bound by launch and L2 latency up to D = 600 or so, then by the
// passes over y, x0 and z.  A step that orthogonalises against m vectors is
// m + 3 launches where a dot product, its final sum and an update apiece were
// 3 m + 7; with the eigenvector's combination below in one launch, a solve on
// a kept plan (five vectors, seven matvecs) takes 547 us instead of 797 at
// D = 123 in FP64 and 2459 instead of 2704 at D = 600 with 7 slices.  (Vectors
// of up to kClMax elements now go through one cluster, further down.)
__global__ void __launch_bounds__(kRedThreads) update_dot_kernel(const double* part_in, double* c_out, const double* x0_in,
                                                                const double* c1_in, const double* x1_in, double* y,
                                                                const double* z_in, int64_t n, double* part_out) {
  __shared__ double sh[kRedThreads];
  dependents_may_start();
  const int64_t zero = wait_for_predecessor();
  const double *x0 = after_wait(x0_in, zero), *c1 = after_wait(c1_in, zero), *x1 = after_wait(x1_in, zero), *z = after_wait(z_in, zero);
  part_in = after_wait(part_in, zero);
  if ((int64_t)blockIdx.x * kRedThreads >= n) {  // no element here
    if (threadIdx.x == 0) part_out[blockIdx.x] = 0.0;
    return;
  }
  const double c = sum_partials(part_in, sh);
  if (blockIdx.x == 0 && threadIdx.x == 0) *c_out = c;
  const double a0 = -c, a1 = c1 ? -*c1 : 0.0;
  double v = 0;
  grid_stride4(n, [&](int64_t i, int64_t stride, auto U) {
    double f[U.value], g[U.value], h[U.value], w[U.value];
#pragma unroll
    for (int u = 0; u < U.value; ++u) {
      const int64_t k = i + u * stride;
      f[u] = y[k];
      g[u] = x0[k];
      h[u] = c1 ? x1[k] : 0.0;
      w[u] = z ? z[k] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U.value; ++u) {
      double t = fma(a0, g[u], f[u]);
      if (c1) t = fma(a1, h[u], t);
      y[i + u * stride] = t;
      v += t * (z ? w[u] : t);
    }
  });
  const double s = block_sum(v, sh);
  if (threadIdx.x == 0) part_out[blockIdx.x] = s;
}

// b = sqrt of the dot product whose partial sums are part_in, x *= 1 / b
// (b_out null: not stored)
__global__ void __launch_bounds__(kRedThreads) normalize_part_kernel(const double* part_in, double* x_in, int64_t n,
                                                                    double* b_out) {
  __shared__ double sh[kRedThreads];
  dependents_may_start();
  const int64_t zero = wait_for_predecessor();
  part_in = after_wait(part_in, zero);
  double* x = after_wait(x_in, zero);
  if ((int64_t)blockIdx.x * kRedThreads >= n) return;
  const double b = sqrt(sum_partials(part_in, sh));
  const double f = 1.0 / b;
  if (b_out && blockIdx.x == 0 && threadIdx.x == 0) *b_out = b;
  grid_stride4(n, [&](int64_t i, int64_t stride, auto U) {
    double t[U.value];
#pragma unroll
    for (int u = 0; u < U.value; ++u) t[u] = x[i + u * stride];
#pragma unroll
    for (int u = 0; u < U.value; ++u) x[i + u * stride] = t[u] * f;
  });
}

// v = z_0 f_0 + z_1 f_1 + ... (f_j = f + j stride), added in that order
// (first: v starts from z_0 f_0, else from v); part: partial sums of v . v
constexpr int kCombineMax = 16;
struct CombineCoefs {
  double z[kCombineMax];
};
__global__ void __launch_bounds__(kRedThreads) combine_vectors_kernel(CombineCoefs c, int m, bool first,
                                                                     const double* f_in, int64_t stride_f, double* v_in,
                                                                     int64_t n, double* part) {
  __shared__ double sh[kRedThreads];
  dependents_may_start();
  const int64_t zero = wait_for_predecessor();
  const double* f = after_wait(f_in, zero);
  double* v = after_wait(v_in, zero);
  double s = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double t = first ? __dmul_rn(c.z[0], f[i]) : fma(c.z[0], f[i], v[i]);
#pragma unroll 4
    for (int j = 1; j < m; ++j) t = fma(c.z[j], f[j * stride_f + i], t);
    v[i] = t;
    s += t * t;
  }
  s = block_sum(s, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// ---- the same steps on one cluster ----
// A vector of a few thousand elements is a microsecond's work, and a launch per
// coefficient (4 to 5 us each, most of it launch, the partial sums' way through
// L2 and the ramps) is all a Lanczos step's tail then costs.  One cluster of
// sixteen CTAs holds the vector in registers and goes through the whole tail:
// the CTAs' sums meet in shared memory (every CTA writes its own to all
// sixteen), the next vector's elements are loaded while they do.  Each
// coefficient takes 1.3 to 2 us instead of 5: a chain of FP64 additions, the
// cluster's barrier (920 clocks) and the FP64 pipe of sixteen SMs, one
// multiply-add a clock each.  A solve on a new plan (five vectors, FP64) takes
// 407 us instead of 455 at D = 123 (6,111 elements), 266 instead of 330 at D =
// 24; 490 instead of 525 at 15,700 elements, but 600 instead of 590 at 17,400.
constexpr int kClCtas = 16, kClThreads = 128, kClMostElems = 8;
constexpr int64_t kClMax = (int64_t)kClCtas * kClThreads * kClMostElems;

struct ClusterSum {
  double part[kClThreads];
  double cta[2][kClCtas];  // by turns: one is read while the other is written
  double all;
};

// The cluster's slice of one thread: E elements, kClThreads apart.  E follows
// the vector's length (by_elems): an FP64 instruction whose lanes are all
// switched off holds the pipe as long as any other.
template <int E>
struct ClusterSlice {
  int64_t base;
  int len;
  __device__ explicit ClusterSlice(int64_t n) {
    const int64_t share = (n + kClCtas - 1) / kClCtas, begin = blockIdx.x * share;
    base = begin + threadIdx.x;
    len = (int)(min(n, begin + share) - begin) - (int)threadIdx.x;
  }
  __device__ bool has(int u) const { return u * kClThreads < len; }
  __device__ void load(const double* x, double (&r)[E]) const {
#pragma unroll
    for (int u = 0; u < E; ++u)
      if (has(u)) r[u] = x[base + u * kClThreads];
  }
  __device__ void store(double* x, const double (&r)[E]) const {
#pragma unroll
    for (int u = 0; u < E; ++u)
      if (has(u)) x[base + u * kClThreads] = r[u];
  }
  // this thread's part of a . b
  __device__ double dot(const double (&a)[E], const double (&b)[E]) const {
    double v = 0.0;
#pragma unroll
    for (int u = 0; u < E; ++u)
      if (has(u)) v = fma(a[u], b[u], v);
    return v;
  }
  __device__ void axpy(double c, const double (&x)[E], double (&y)[E]) const {
#pragma unroll
    for (int u = 0; u < E; ++u)
      if (has(u)) y[u] = fma(c, x[u], y[u]);
  }
  __device__ void scale(double c, double (&y)[E]) const {
#pragma unroll
    for (int u = 0; u < E; ++u)
      if (has(u)) y[u] *= c;
  }
};

// A CTA's shared memory may be written from another one only once it runs:
// every kernel of a cluster arrives here first of all and waits before its first
// cluster_sum, behind the wait for the predecessor and the first loads.
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); }

// The sum of every thread's v over the cluster, in every thread; turn: 0, 1, 0,
// ...  An FP64 addition keeps the SM's pipe busy for 32 clocks whatever its
// lanes hold, so one warp does them all, twelve in a row: with a butterfly in
// every warp (sixteen of them then) a coefficient took 2.9 us.
__device__ __forceinline__ double cluster_sum(double v, ClusterSum& sh, int turn) {
  const int lane = threadIdx.x & 31;
  sh.part[threadIdx.x] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
#pragma unroll
    for (int i = 1; i < kClThreads / 32; ++i) v += sh.part[threadIdx.x + 32 * i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane < kClCtas) {
      uint32_t to;
      asm("mapa.shared::cluster.u32 %0, %1, %2;"
          : "=r"(to)
          : "r"((uint32_t)__cvta_generic_to_shared(&sh.cta[turn][blockIdx.x])), "r"(lane));
      asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(to), "d"(v) : "memory");
    }
    __syncwarp();  // the barrier is a whole warp's
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (threadIdx.x < 32) {
    v = sh.cta[turn][lane & (kClCtas - 1)];
#pragma unroll
    for (int o = kClCtas / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) sh.all = v;
  }
  __syncthreads();
  return sh.all;
}

// launch_lanczos_tail in one launch
template <int E>
__global__ void __launch_bounds__(kClThreads) lanczos_tail_cluster(int m, double* f, int64_t stride_f, int64_t n,
                                                                  double* alpha, double* beta, double* q) {
  __shared__ ClusterSum sh;
  cluster_arrive();
  dependents_may_start();
  const int64_t zero = wait_for_predecessor();
  f = after_wait(f, zero);
  beta = after_wait(beta, zero);
  const ClusterSlice<E> at(n);
  const bool first = blockIdx.x == 0 && threadIdx.x == 0;
  double y[E], x[E], next[E];
  at.load(f + m * stride_f, y);
  at.load(f + (m - 1) * stride_f, x);
  if (m >= 2) at.load(f + (m - 2) * stride_f, next);
  cluster_wait();
  int turn = 0;
  double c = cluster_sum(at.dot(x, y), sh, turn);
  if (first) alpha[m - 1] = c;
  at.axpy(-c, x, y);
  if (m >= 2) {
    at.axpy(-beta[m - 1], next, y);
    at.load(f, x);
    for (int j = 0; j < m; ++j) {
      const double part = at.dot(x, y);
      if (j + 1 < m) at.load(f + (j + 1) * stride_f, next);
      c = cluster_sum(part, sh, turn ^= 1);
      if (first) q[j] = c;
      at.axpy(-c, x, y);
#pragma unroll
      for (int u = 0; u < E; ++u) x[u] = next[u];
    }
  }
  const double b = sqrt(cluster_sum(at.dot(y, y), sh, turn ^= 1)), s = 1.0 / b;
  if (first) beta[m] = b;
  at.scale(s, y);
  at.store(f + m * stride_f, y);
}

// out = x / |x|, *b_out = |x| (null: not stored)
template <int E>
__global__ void __launch_bounds__(kClThreads) unit_cluster(const double* x, double* out, int64_t n, double* b_out) {
  __shared__ ClusterSum sh;
  cluster_arrive();
  dependents_may_start();
  const int64_t zero = wait_for_predecessor();
  x = after_wait(x, zero);
  const ClusterSlice<E> at(n);
  double y[E];
  at.load(x, y);
  cluster_wait();
  const double b = sqrt(cluster_sum(at.dot(y, y), sh, 0)), s = 1.0 / b;
  if (b_out && blockIdx.x == 0 && threadIdx.x == 0) *b_out = b;
  at.scale(s, y);
  at.store(out, y);
}

// out[0] = x . y, or (two) out[0] = x . x and out[1] = x . y
template <int E>
__global__ void __launch_bounds__(kClThreads) dot_cluster(const double* x, const double* y, int64_t n, bool two,
                                                         double* out) {
  __shared__ ClusterSum sh;
  cluster_arrive();
  dependents_may_start();
  const int64_t zero = wait_for_predecessor();
  x = after_wait(x, zero);
  y = after_wait(y, zero);
  const ClusterSlice<E> at(n);
  double a[E], b[E];
  at.load(x, a);
  at.load(y, b);
  cluster_wait();
  const double v = cluster_sum(at.dot(a, b), sh, 0);
  const double w = two ? cluster_sum(at.dot(a, a), sh, 1) : 0.0;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (two) out[0] = w, out[1] = v;
    else out[0] = v;
  }
}

// v = z_0 f_0 + z_1 f_1 + ... (as combine_vectors_kernel), then v /= |v|
template <int E>
__global__ void __launch_bounds__(kClThreads) combine_unit_cluster(CombineCoefs c, int m, const double* f,
                                                                  int64_t stride_f, double* out, int64_t n) {
  __shared__ ClusterSum sh;
  cluster_arrive();
  dependents_may_start();
  const int64_t zero = wait_for_predecessor();
  f = after_wait(f, zero);
  const ClusterSlice<E> at(n);
  double y[E], x[E];
  at.load(f, y);
  at.scale(c.z[0], y);
  for (int j = 1; j < m; ++j) {
    at.load(f + j * stride_f, x);
    at.axpy(c.z[j], x, y);
  }
  cluster_wait();
  const double s = 1.0 / sqrt(cluster_sum(at.dot(y, y), sh, 0));
  at.scale(s, y);
  at.store(out, y);
}

cudaLaunchConfig_t cluster_config(cudaLaunchAttribute* attr, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = kClCtas;
  attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
  cfg.gridDim = dim3(kClCtas);
  cfg.blockDim = dim3(kClThreads);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// clusters of sixteen, beyond the portable eight, are allowed per kernel
template <int E>
bool allow_clusters() {
  const void* kernels[] = {(const void*)lanczos_tail_cluster<E>, (const void*)unit_cluster<E>,
                           (const void*)dot_cluster<E>, (const void*)combine_unit_cluster<E>};
  for (const void* k : kernels) {
    cudaLaunchAttribute attr = {};
    const cudaLaunchConfig_t cfg = cluster_config(&attr, nullptr);
    int most = 0;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&most, k, &cfg) != cudaSuccess || most < 1) {
      cudaGetLastError();
      return false;
    }
  }
  return true;
}

// whether the current device runs them; asked once per device
bool cluster_runs() {
  static std::mutex mu;
  static std::map<int, bool> known;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  std::lock_guard<std::mutex> lock(mu);
  const auto it = known.find(dev);
  if (it != known.end()) return it->second;
  return known[dev] = allow_clusters<1>() && allow_clusters<2>() && allow_clusters<4>() && allow_clusters<8>();
}

template <class... P, class... A>
cudaError_t launch_cluster(cudaStream_t stream, void (*kernel)(P...), A... args) {
  return launch_overlapped(kernel, dim3(kClCtas), kClThreads, 0, kClCtas, stream, args...);
}

// launch(E) with the elements a thread that a vector of n asks for
template <class F>
cudaError_t by_elems(int64_t n, F launch) {
  const int64_t e = (n + kClCtas * kClThreads - 1) / (kClCtas * kClThreads);
  if (e <= 1) return launch(std::integral_constant<int, 1>());
  if (e <= 2) return launch(std::integral_constant<int, 2>());
  if (e <= 4) return launch(std::integral_constant<int, 4>());
  return launch(std::integral_constant<int, kClMostElems>());
}

// Vectors of up to kClMax elements go through one cluster, longer ones through
// the whole chip.
bool on_cluster(int64_t n) { return n > 0 && n <= kClMax && cluster_runs(); }

__global__ void axpy_kernel(double alpha, const double* __restrict__ x, double* __restrict__ y, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    y[i] += alpha * x[i];
}

__global__ void scale_kernel(double alpha, double* __restrict__ x, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    x[i] *= alpha;
}

}  // namespace

int reduction_scratch_doubles() { return kRedBlocks + 1; }
int lanczos_scratch_doubles() { return 2 * kRedBlocks + 2; }

namespace {
cudaError_t launch_dot_partial(const double* x, const double* y, int64_t n, double* scratch, int half,
                               cudaStream_t stream) {
  return launch_overlapped(dot_partial, dim3(kRedBlocks), kRedThreads, 0, 0, stream, x, y, n, scratch + half * kRedBlocks);
}

cudaError_t dot_on_grid(const double* x, const double* y, int64_t n, double* scratch, double* out,
                        cudaStream_t stream) {
  cudaError_t e = launch_dot_partial(x, y, n, scratch, 0, stream);
  if (e != cudaSuccess) return e;
  return launch_overlapped(dot_final, dim3(1), kRedThreads, 0, 0, stream, scratch, out);
}

cudaError_t launch_update_dot(double* scratch, int half, double* c_out, const double* x0, const double* c1,
                              const double* x1, double* y, const double* z, int64_t n, cudaStream_t stream) {
  return launch_overlapped(update_dot_kernel, dim3(kRedBlocks), kRedThreads, 0, 0, stream, scratch + half * kRedBlocks,
                           c_out, x0, c1, x1, y, z, n, scratch + (1 - half) * kRedBlocks);
}

cudaError_t launch_normalize_part(const double* scratch, int half, double* x, int64_t n, double* b_out,
                                  cudaStream_t stream) {
  return launch_overlapped(normalize_part_kernel, dim3(kRedBlocks), kRedThreads, 0, 0, stream,
                           scratch + half * kRedBlocks, x, n, b_out);
}
}  // namespace

cudaError_t launch_dot(const double* x, const double* y, int64_t n, double* scratch, cudaStream_t stream) {
  return dot_on_grid(x, y, n, scratch, scratch + kRedBlocks, stream);
}

cudaError_t launch_dot_to(const double* x, const double* y, int64_t n, double* scratch, double* out,
                          cudaStream_t stream) {
  if (on_cluster(n))
    return by_elems(n, [&](auto E) { return launch_cluster(stream, dot_cluster<E.value>, x, y, n, false, out); });
  return dot_on_grid(x, y, n, scratch, out, stream);
}

cudaError_t launch_unit(const double* x, double* out, int64_t n, double* scratch, double* b_out, cudaStream_t stream) {
  if (on_cluster(n))
    return by_elems(n, [&](auto E) { return launch_cluster(stream, unit_cluster<E.value>, x, out, n, b_out); });
  cudaError_t e = x == out ? cudaSuccess
                           : cudaMemcpyAsync(out, x, n * sizeof(double), cudaMemcpyDeviceToDevice, stream);
  if (e == cudaSuccess) e = launch_dot_partial(out, out, n, scratch, 0, stream);
  if (e == cudaSuccess) e = launch_normalize_part(scratch, 0, out, n, b_out, stream);
  return e;
}

cudaError_t launch_combine_vectors(const double* z, int m, const double* f, int64_t stride_f, double* v, int64_t n,
                                   double* scratch, bool unit, cudaStream_t stream) {
  if (unit && m <= kCombineMax && on_cluster(n)) {
    CombineCoefs c{};
    std::copy(z, z + m, c.z);
    return by_elems(n, [&](auto E) {
      return launch_cluster(stream, combine_unit_cluster<E.value>, c, m, f, stride_f, v, n);
    });
  }
  cudaError_t e = cudaSuccess;
  for (int j0 = 0; j0 < m && e == cudaSuccess; j0 += kCombineMax) {
    CombineCoefs c{};
    const int k = std::min(kCombineMax, m - j0);
    std::copy(z + j0, z + j0 + k, c.z);
    e = launch_overlapped(combine_vectors_kernel, dim3(kRedBlocks), kRedThreads, 0, 0, stream, c, k, j0 == 0,
                          f + j0 * stride_f, stride_f, v, n, scratch);
  }
  return e == cudaSuccess && unit ? launch_normalize_part(scratch, 0, v, n, nullptr, stream) : e;
}

cudaError_t launch_dot2(const double* x, const double* y, int64_t n, double* scratch, cudaStream_t stream) {
  if (on_cluster(n))
    return by_elems(n, [&](auto E) {
      return launch_cluster(stream, dot_cluster<E.value>, x, y, n, true, scratch + 2 * kRedBlocks);
    });
  const cudaError_t e = launch_overlapped(dot2_partial, dim3(kRedBlocks), kRedThreads, 0, 0, stream, x, y, n, scratch);
  if (e != cudaSuccess) return e;
  return launch_overlapped(dot_final, dim3(2), kRedThreads, 0, 0, stream, scratch, scratch + 2 * kRedBlocks);
}

cudaError_t launch_lanczos_tail(int m, double* f, int64_t stride_f, int64_t n, double* alpha, double* beta, double* q,
                                double* scratch, cudaStream_t stream) {
  if (on_cluster(n))
    return by_elems(n, [&](auto E) {
      return launch_cluster(stream, lanczos_tail_cluster<E.value>, m, f, stride_f, n, alpha, beta, q);
    });
  auto ff = [&](int j) { return f + j * stride_f; };
  double* y = ff(m);
  cudaError_t e = launch_dot_partial(ff(m - 1), y, n, scratch, 0, stream);
  int half = 0;
  if (m < 2) {
    if (e == cudaSuccess) e = launch_update_dot(scratch, half, alpha + m - 1, ff(0), nullptr, nullptr, y, nullptr, n, stream);
    half ^= 1;
  } else {
    if (e == cudaSuccess)
      e = launch_update_dot(scratch, half, alpha + m - 1, ff(m - 1), beta + m - 1, ff(m - 2), y, ff(0), n, stream);
    half ^= 1;
    for (int j = 0; j < m && e == cudaSuccess; ++j, half ^= 1)
      e = launch_update_dot(scratch, half, q + j, ff(j), nullptr, nullptr, y, j + 1 < m ? ff(j + 1) : nullptr, n, stream);
  }
  if (e == cudaSuccess) e = launch_normalize_part(scratch, half, y, n, beta + m, stream);
  return e;
}

cudaError_t launch_axpy(double alpha, const double* x, double* y, int64_t n, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  int blocks = (int)((n + 255) / 256);
  if (blocks > 4 * 152 * 4) blocks = 4 * 152 * 4;
  axpy_kernel<<<blocks, 256, 0, stream>>>(alpha, x, y, n);
  return cudaGetLastError();
}

cudaError_t launch_scale(double alpha, double* x, int64_t n, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  int blocks = (int)((n + 255) / 256);
  if (blocks > 4 * 152 * 4) blocks = 4 * 152 * 4;
  scale_kernel<<<blocks, 256, 0, stream>>>(alpha, x, n);
  return cudaGetLastError();
}

}  // namespace su2g
