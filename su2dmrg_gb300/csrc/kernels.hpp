// Launchers of the device kernels (kernels_f64.cu and friends).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "gemm_work.hpp"

namespace su2g {

// records the calling thread's su2g_last_error() text and returns code
int set_last_error(int code, const std::string& msg);

// Device memory from a per-device stream-ordered pool (devmem.cu): usable on
// any stream when dev_alloc returns; dev_free releases it once `after` has
// passed the point of the call (pass the stream of its last use).  Neither
// synchronises the device.
cudaError_t dev_alloc(void** p, size_t bytes);
void dev_free(void* p, cudaStream_t after);
// the same pool, for use on `st` alone
cudaError_t stream_alloc(void** p, size_t bytes, cudaStream_t st);
// dev_alloc + a copy of `bytes` host bytes, complete on return
cudaError_t upload_bytes(const void* host, size_t bytes, void** dptr);
// the calling thread's private non-blocking stream on the current device
cudaError_t setup_stream(cudaStream_t* out);

cudaError_t launch_gemm_f64(const GemmTile* tiles, const F64Counts& n, const GemmSeg* segs, const Bases& bases,
                            cudaStream_t stream);
// one dense product C (M x N, ld ldc) = op(A) B with the same tile code
// (op(A) = A, M x K, or for transA A^T with A stored K x M; B stored K x N),
// the work formed from the arguments
cudaError_t launch_gemm_f64_dense(bool transA, int M, int N, int K, const double* A, int lda, const double* B,
                                  int ldb, double* C, int ldc, cudaStream_t stream);

// several of them in one launch (48 at a time): the same sums
struct DenseGemm {
  bool transA;
  int M, N, K;
  const double* A;
  int lda;
  const double* B;
  int ldb;
  double* C;
  int ldc;
};
cudaError_t launch_gemm_f64_dense_many(const DenseGemm* jobs, int njobs, cudaStream_t stream);

// deterministic dot product: partial sums in scratch[0..reduction_scratch_doubles()-1),
// the result in scratch[reduction_scratch_doubles()-1]
int reduction_scratch_doubles();
cudaError_t launch_dot(const double* x, const double* y, int64_t n, double* scratch, cudaStream_t stream);
cudaError_t launch_axpy(double alpha, const double* x, double* y, int64_t n, cudaStream_t stream);
// The vector work of a Lanczos step with every scalar on the device.  scratch
// holds lanczos_scratch_doubles(): two halves of partial sums and two results.
int lanczos_scratch_doubles();
// *out = x . y
cudaError_t launch_dot_to(const double* x, const double* y, int64_t n, double* scratch, double* out,
                          cudaStream_t stream);
// out = x / |x|, *b_out = |x| (b_out null: not); x and out may be one vector
cudaError_t launch_unit(const double* x, double* out, int64_t n, double* scratch, double* b_out, cudaStream_t stream);
// v = sum_j z[j] (f + j stride_f) for j < m in order (z on the host), then (unit) v /= |v|
cudaError_t launch_combine_vectors(const double* z, int m, const double* f, int64_t stride_f, double* v, int64_t n,
                                   double* scratch, bool unit, cudaStream_t stream);
// x . x and x . y to the two results at the end of scratch
cudaError_t launch_dot2(const double* x, const double* y, int64_t n, double* scratch, cudaStream_t stream);
// every launch of a step after its matvec (lanczos_su2.cpp:136-142, 156-173):
// alpha = f(m-1) . f(m), the three-term update, full reorthogonalisation against
// f(0) .. f(m-1), the norm beta and the division by it; f(j) = f + j stride_f,
// alpha, beta, q: the coefficient arrays
cudaError_t launch_lanczos_tail(int m, double* f, int64_t stride_f, int64_t n, double* alpha, double* beta, double* q,
                                double* scratch, cudaStream_t stream);
cudaError_t launch_scale(double alpha, double* x, int64_t n, cudaStream_t stream);
// y += alpha * (*scale) * x with the scale read on the device (combine.cu)
cudaError_t launch_axpy_dev(double alpha, const double* scale, const double* x, double* y, int64_t n,
                            cudaStream_t stream);

namespace oz {
struct PackJob;
struct OzSeg;
struct OzTile;
struct RedTile;
cudaError_t launch_reduce(const RedTile* reds, int n, const Bases& bases, cudaStream_t stream);
// one-time per-process setup of the GEMM kernel (function attributes, SM count),
// done before any launch is captured into a graph
cudaError_t prepare_ozaki_gemm(int S);
// runs the GEMM's bounded mbarrier wait on a barrier nothing arrives at, with
// `limit` polls; *timed_out_host = 1 when it gave up (the expected outcome)
cudaError_t bounded_wait_selftest(long long limit, int* timed_out_host, cudaStream_t stream);
// CTAs of the persistent GEMM grid on the current device (its SM count); 152
// when no device answers (host-only planning and validation).
int ozaki_persistent_grid();
// kernels of a launch_pack of some units
int pack_launches(bool rows_pass, bool unit_alpha, int max_nkt);
// row-exponent pass (when rows_pass) + digit pass: 1 or 2 kernels, none for nunits == 0;
// unit_alpha: every job's scale is 1 or -1 and none has row maxima; clear[0,
// nclear) = 0 in the first of them
cudaError_t launch_pack(int S, const PackJob* jobs, const int2* units, int nunits, int max_nkt, bool rows_pass,
                        const Bases& bases, uint8_t* packed, int* exps, cudaStream_t stream, bool unit_alpha = false,
                        int* clear = nullptr, int nclear = 0);
cudaError_t launch_ozaki_gemm(int S, const OzTile* tiles, int ntiles, const OzSeg* segs, const uint8_t* packed,
                              int* exps, const Bases& bases, int* err, cudaStream_t stream);
int gemm_smem_bytes(int S);
}  // namespace oz

}  // namespace su2g
