// Truncation of a two-site vector (tensor_su2::svd, tensor_su2.cpp:1619-1758,
// with the per-sector tensor::svd of tensor.cpp:1472-1700), on the GPU:
//   * per sector, the Gram matrix of the smaller side and its FP64
//     eigendecomposition (cuSOLVER syevd in its deterministic mode,
//     eigenvalues ascending like dsyev), then the reference's refinement:
//     while more than one eigenvalue
//     lies below 0.1 of the largest of the current subspace, re-diagonalise
//     the original Gram matrix projected on that subspace (from the basis at
//     hand by a few products where that converges, else by another
//     eigendecomposition);
//   * the other factor by one more product, singular values = sqrt of the
//     eigenvalues above 1e-100 of the largest, columns scaled by s^(p1-1) and
//     s^p2 (or the mirror for wide blocks);
//   * every product (Gram matrices, the refinement's projections and
//     rotations, the other factor) runs on the library's FP64 tile engine,
//     whose sums have a fixed order: the result of a truncation does not
//     depend on what else shares the GPU (a library GEMM picks its internal
//     implementation by the concurrent load, and near a cut in the rounding
//     noise that changes which multiplets are kept);
//   * the sectors go through these steps together, a launch a step for all of
//     them; their first eigendecompositions run on a stream, cuSOLVER handle and
//     host thread each;
//   * on the host: all kept singular values sorted by the Shell sort of
//     sort2.f (dsort2, whose handling of equal values decides ties), the
//     largest max_dcut multiplets kept (no (2j+1) weighting), and the
//     singular values reported kept-then-discarded as the reference writes
//     them.
#include <cuda_runtime.h>
#include <cusolverDn.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <deque>
#include <cmath>
#include <cstring>
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "heff_plan.hpp"
#include "kernels.hpp"
#include "su2_meta.hpp"
#include "svd_levels.hpp"
#include "su2g.h"

namespace {

int fail(int code, const std::string& msg) { return su2g::set_last_error(code, msg); }

// Every sector's part of a step is one entry of a list in the kernel's
// parameters (JobList): a step is one launch, whatever the sectors.
constexpr int kJobMost = 60;
template <class J>
struct JobList {
  J job[kJobMost];
  int first[kJobMost];  // the job's first CTA
};
// kernel(list, njobs) with ctas(job) CTAs for each job
template <class J, class C, class... A>
cudaError_t launch_jobs(void (*kernel)(JobList<J>, int, A...), const std::vector<J>& jobs, C ctas, int threads,
                        size_t smem, cudaStream_t st, A... args) {
  static_assert(sizeof(JobList<J>) <= 4000, "kernel parameters");
  for (size_t j = 0; j < jobs.size();) {
    JobList<J> list;
    int n = 0, first = 0;
    for (; j < jobs.size() && n < kJobMost; ++j) {
      const int c = ctas(jobs[j]);
      if (c <= 0) continue;
      list.job[n] = jobs[j];
      list.first[n++] = first;
      first += c;
    }
    if (n == 0) continue;
    kernel<<<first, threads, smem, st>>>(list, n, args...);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
// this CTA's job, and in *cta its number within it
template <class J>
__device__ __forceinline__ const J& my_job(const JobList<J>& list, int n, int* cta) {
  int j = 0;
  while (j + 1 < n && list.first[j + 1] <= (int)blockIdx.x) ++j;
  *cta = blockIdx.x - list.first[j];
  return list.job[j];
}

struct ScaleJob {  // columns c0 .. c0 + ncol of a (ld rows) times f
  double* a;
  int rows, c0, ncol;
  const double* f;
};
__global__ void scale_columns(const __grid_constant__ JobList<ScaleJob> list, int n) {
  int c;
  const ScaleJob& j = my_job(list, n, &c);
  double* col = j.a + (int64_t)(j.c0 + c) * j.rows;
  const double f = j.f[c];
  for (int r = threadIdx.x; r < j.rows; r += blockDim.x) col[r] *= f;
}

struct CopyJob {
  double* dst;
  const double* src;
  int64_t len;
};
constexpr int kCopyTile = 1024;
__global__ void copy_arrays(const __grid_constant__ JobList<CopyJob> list, int n) {
  int c;
  const CopyJob& j = my_job(list, n, &c);
  const int64_t end = min(j.len, (int64_t)(c + 1) * kCopyTile);
  for (int64_t i = (int64_t)c * kCopyTile + threadIdx.x; i < end; i += blockDim.x) j.dst[i] = j.src[i];
}

// A matrix (n x n, ld n) as the leading block of one of size N for a batch of
// equal sizes: beyond it a diagonal below every eigenvalue, of the matrix's own
// scale, so that the padding comes first and its rows stay zero in the others'
// eigenvectors.  And the vectors back.  A level in the rounding noise has
// negative eigenvalues, often larger than every entry of its diagonal: the bound
// lies an eighth beyond the largest column sum of magnitudes.
struct PadJob {
  double* mat;
  int n;
  double* box;
};
__global__ void pad_matrix(const __grid_constant__ JobList<PadJob> list, int njobs, int N) {
  __shared__ double smax[8];
  int c;
  const PadJob& j = my_job(list, njobs, &c);
  double mx = 0;  // every CTA finds it: 128 columns at most
  for (int q = threadIdx.x >> 5; q < j.n; q += 8) {
    double sum = 0;
    for (int i = threadIdx.x & 31; i < j.n; i += 32) sum += fabs(j.mat[(int64_t)q * j.n + i]);
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    mx = fmax(mx, sum);
  }
  if ((threadIdx.x & 31) == 0) smax[threadIdx.x >> 5] = mx;
  __syncthreads();
  for (int w = 0; w < 8; ++w) mx = fmax(mx, smax[w]);
  const double below = mx > 0 ? -1.125 * mx : -1.0;
  double* col = j.box + (int64_t)c * N;  // one column a CTA
  for (int r = threadIdx.x; r < N; r += blockDim.x)
    col[r] = r < j.n && c < j.n ? j.mat[(int64_t)c * j.n + r] : r == c ? below : 0.0;
}
__global__ void unpad_vectors(const __grid_constant__ JobList<PadJob> list, int njobs, int N) {
  int c;
  const PadJob& j = my_job(list, njobs, &c);
  const double* col = j.box + (int64_t)(N - j.n + c) * N;
  for (int r = threadIdx.x; r < j.n; r += blockDim.x) j.mat[(int64_t)c * j.n + r] = col[r];
}

// out (cols x rows) = in^T, 32 x 32 tiles through shared memory
__global__ void transpose_kernel(const double* __restrict__ in, int rows, int cols, double* __restrict__ out) {
  __shared__ double t[32][33];
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  for (int j = threadIdx.y; j < 32; j += 8) {
    const int r = r0 + threadIdx.x, c = c0 + j;
    if (r < rows && c < cols) t[j][threadIdx.x] = in[(int64_t)c * rows + r];
  }
  __syncthreads();
  for (int j = threadIdx.y; j < 32; j += 8) {
    const int c = c0 + threadIdx.x, r = r0 + j;
    if (r < rows && c < cols) out[(int64_t)r * cols + c] = t[threadIdx.x][j];
  }
}

// The eigenvector sign rule of su2g::canonical_column_signs (tridiag.hpp)
// on the device: one CTA per column of the n x n matrix z.
// The largest magnitude and the first index above 1e-4 of it are exact
// reductions (max, min), so the choice does not depend on the order.
struct SignJob {
  double* z;
  int n;
};
__global__ void __launch_bounds__(256) canonical_signs_kernel(const __grid_constant__ JobList<SignJob> list, int n) {
  __shared__ double smax[8];
  __shared__ int sfirst[8];
  int c;
  const SignJob& job = my_job(list, n, &c);
  const int rows = job.n;
  double* col = job.z + (int64_t)c * rows;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double mx = 0;
  for (int i = threadIdx.x; i < rows; i += blockDim.x) mx = fmax(mx, fabs(col[i]));
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) smax[wid] = mx;
  __syncthreads();
  mx = smax[0];
  for (int w = 1; w < 8; ++w) mx = fmax(mx, smax[w]);
  int first = rows;
  for (int i = threadIdx.x; i < rows; i += blockDim.x)
    if (fabs(col[i]) > 1e-4 * mx) {
      first = i;
      break;
    }
  for (int o = 16; o > 0; o >>= 1) first = min(first, __shfl_xor_sync(0xffffffffu, first, o));
  if (lane == 0) sfirst[wid] = first;
  __syncthreads();
  first = sfirst[0];
  for (int w = 1; w < 8; ++w) first = min(first, sfirst[w]);
  if (first < rows && col[first] < 0)
    for (int i = threadIdx.x; i < rows; i += blockDim.x) col[i] = -col[i];
}

// ---- refinement levels without an eigendecomposition ----
// A level's matrix M (n x n, the Gram matrix projected on the level's subspace)
// is nearly diagonal already: the basis came from an eigendecomposition, whose
// rounding is all that is left off the diagonal.  What the level must resolve
// are the eigenvectors of its top decade T (the rest is projected again and
// resolved on later levels), and those follow from M by the quadratically
// convergent iteration of Ogita & Aishima ("Iterative refinement for symmetric
// eigenvalue decomposition", Japan J. Indust. Appl. Math. 35 (2018)): with
// S = X^T M X and R = I - X^T X,
//     lambda_i = S_ii / (1 - R_ii),
//     X <- X + X E,  E_ij = (S_ij + lambda_j R_ij) / (lambda_j - lambda_i),
//     E_ii = R_ii / 2,
// here with E_ij = R_ij / 2 (orthonormality only) where neither i nor j lies in
// T, or where the coupling is rounding noise of the level and as large as the
// gap (a degenerate pair: any basis of it is as good).  Mostly one step from X =
// I does, which is one launch and no product.  A level of 101 rows takes 0.3 ms
// where cuSOLVER's eigendecomposition takes 4.6 (it is a chain of some hundred
// dependent launches).  With it and the lockstep further down a truncation at D =
// 400 (14 sectors of up to 108 rows, 10 levels) takes 9.0 ms, 47.3 before, and
// those of a sweep of the 8x4 cylinder at D = 400 0.50 s, 2.49 before, with the
// same or smaller residuals and orthonormality errors.
using su2g::kDecade;                    // T: diagonal entries from a tenth of the largest on
using su2g::kStepMax;
constexpr double kStepDone = 1e-8;      // steps up to this leave an error below rounding
constexpr int kRefineMax = 6000;        // the kernel's shared memory (48 KB of eigenvalues)
constexpr double kLevelNoise = 8 * 2.220446049250313e-16;  // of the level's largest entry

// x = I + E from S (the upper triangle counts; ld n) and P = X^T X (null: X =
// I).  info[0]: the largest |E_ij| (as bits), lam[i] the eigenvalue estimates.
// One CTA per column; every CTA finds the decade's first index itself.
struct StepJob {
  const double *S, *P;
  int n;
  double *x, *lam;  // lam: n eigenvalue estimates, then info
};
__global__ void __launch_bounds__(256) refine_step_kernel(const __grid_constant__ JobList<StepJob> list, int njobs) {
  extern __shared__ double d[];  // n eigenvalue estimates
  __shared__ double red[8];
  __shared__ int redi[8];
  int j;
  const StepJob& job = my_job(list, njobs, &j);
  const double* __restrict__ S = job.S;
  const double* __restrict__ P = job.P;
  const int n = job.n, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  double *x = job.x, *lam = job.lam;
  unsigned long long* info = (unsigned long long*)(lam + n);
  double top = 0;
  for (int i = tid; i < n; i += 256) {
    const double v = S[(int64_t)i * n + i] / (P ? P[(int64_t)i * n + i] : 1.0);  // 1 - R_ii = P_ii
    d[i] = v;
    if (j == 0) lam[i] = v;
    top = fmax(top, v);
  }
  for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
  if (lane == 0) red[wid] = top;
  __syncthreads();
  for (int w = 0; w < 8; ++w) top = fmax(top, red[w]);
  int t0 = 0;  // T = [t0, n): after the last entry below a tenth of the largest
  for (int i = tid; i < n; i += 256)
    if (!(d[i] >= kDecade * top)) t0 = i + 1;
  for (int o = 16; o > 0; o >>= 1) t0 = max(t0, __shfl_xor_sync(0xffffffffu, t0, o));
  if (lane == 0) redi[wid] = t0;
  __syncthreads();
  for (int w = 0; w < 8; ++w) t0 = max(t0, redi[w]);
  const double noise = kLevelNoise * top;
  double big = 0;
  for (int i = tid; i < n; i += 256) {
    const int64_t at = i < j ? (int64_t)j * n + i : (int64_t)i * n + j;  // the upper triangle's copy
    const double r = P ? (i == j ? 1.0 : 0.0) - P[at] : 0.0;
    double e = 0.5 * r;
    if (i != j && (i >= t0 || j >= t0)) {
      const double m = S[at] + d[j] * r, gap = d[j] - d[i];
      if (!(fabs(m) <= noise && fabs(m) > kStepMax * fabs(gap))) e = m / gap;
    }
    x[(int64_t)j * n + i] = (i == j ? 1.0 : 0.0) + e;
    big = fmax(big, isfinite(e) ? fabs(e) : 1e300);
  }
  for (int o = 16; o > 0; o >>= 1) big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
  if (lane == 0 && big > 0) atomicMax(info, (unsigned long long)__double_as_longlong(big));
}

// Per-device resources kept across calls: lanes (one stream and one cuSOLVER
// handle each; creating a handle costs milliseconds), lent
// to a call for each sector it processes and returned after it, so calls from
// several host threads (independent solves) run at the same time; and a
// library-private memory pool whose freed blocks stay reserved (stream-ordered
// allocation without device-wide synchronisation, unlike cudaMalloc).
struct Lane {
  cudaStream_t st = nullptr;
  cusolverDnHandle_t sol = nullptr;
  cusolverDnParams_t params = nullptr;
};
struct DeviceRes {
  cudaMemPool_t pool = nullptr;
  std::vector<Lane> free_lanes;
};
std::mutex g_res_mutex;
std::map<int, DeviceRes> g_res;

// Lends n lanes of device dev (creating what is missing) and the pool;
// returns an error message or "".
std::string take_lanes(int dev, int n, std::vector<Lane>* out, cudaMemPool_t* pool) {
  std::lock_guard<std::mutex> lock(g_res_mutex);
  DeviceRes& r = g_res[dev];
  if (!r.pool) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    if (cudaMemPoolCreate(&r.pool, &props) != cudaSuccess) {
      r.pool = nullptr;
      return "cannot create a memory pool";
    }
    uint64_t keep = UINT64_MAX;  // freed blocks stay in the pool
    cudaMemPoolSetAttribute(r.pool, cudaMemPoolAttrReleaseThreshold, &keep);
  }
  *pool = r.pool;
  out->clear();
  while ((int)out->size() < n && !r.free_lanes.empty()) {
    out->push_back(r.free_lanes.back());
    r.free_lanes.pop_back();
  }
  while ((int)out->size() < n) {
    Lane l;
    if (cudaStreamCreateWithFlags(&l.st, cudaStreamNonBlocking) != cudaSuccess) return "cannot create a stream";
    if (cusolverDnCreateParams(&l.params) != CUSOLVER_STATUS_SUCCESS) {
      cudaStreamDestroy(l.st);
      return "cannot create cuSOLVER parameters";
    }
    if (cusolverDnCreate(&l.sol) != CUSOLVER_STATUS_SUCCESS) {
      cusolverDnDestroyParams(l.params);
      cudaStreamDestroy(l.st);
      return "cannot create a cuSOLVER handle";
    }
    cusolverDnSetStream(l.sol, l.st);
    // the eigensolver's deterministic mode: a truncation's result must not
    // depend on what else runs on the GPU
    if (cusolverDnSetDeterministicMode(l.sol, CUSOLVER_DETERMINISTIC_RESULTS) != CUSOLVER_STATUS_SUCCESS) {
      cusolverDnDestroy(l.sol);
      cusolverDnDestroyParams(l.params);
      cudaStreamDestroy(l.st);
      return "cannot set the eigensolver's deterministic mode";
    }
    out->push_back(l);
  }
  return "";
}

void give_lanes(int dev, const std::vector<Lane>& lanes) {
  std::lock_guard<std::mutex> lock(g_res_mutex);
  DeviceRes& r = g_res[dev];
  r.free_lanes.insert(r.free_lanes.end(), lanes.begin(), lanes.end());
}

// Host threads for the eigendecompositions of a call (cuSOLVER launches a long
// chain of kernels from the calling thread).  Kept across calls and grown on
// demand, instead of one thread per sector per call; never joined (the process
// ends with them).
class SectorThreads {
 public:
  static SectorThreads& get() {
    static SectorThreads* t = new SectorThreads();
    return *t;
  }
  // runs body(0..n-1), body(0) on the calling thread, and returns when all are done
  void run(size_t n, const std::function<void(size_t)>& body) {
    if (n == 0) return;
    struct Latch {
      std::mutex mu;
      std::condition_variable cv;
      size_t left;
    } latch;
    latch.left = n - 1;
    {
      std::lock_guard<std::mutex> lock(mu_);
      for (size_t q = 1; q < n; ++q)
        queue_.push_back([&, q] {
          body(q);
          std::lock_guard<std::mutex> l(latch.mu);
          if (--latch.left == 0) latch.cv.notify_all();
        });
      while (idle_ < queue_.size()) {  // a thread per waiting task
        std::thread(&SectorThreads::loop, this).detach();
        ++idle_;
      }
    }
    cv_.notify_all();
    body(0);
    std::unique_lock<std::mutex> l(latch.mu);
    latch.cv.wait(l, [&] { return latch.left == 0; });
  }

 private:
  void loop() {
    for (;;) {
      std::function<void()> task;
      {
        std::unique_lock<std::mutex> lock(mu_);
        cv_.wait(lock, [&] { return !queue_.empty(); });
        task = std::move(queue_.front());
        queue_.pop_front();
        --idle_;
      }
      task();
      std::lock_guard<std::mutex> lock(mu_);
      ++idle_;
    }
  }
  std::mutex mu_;
  std::condition_variable cv_;
  std::deque<std::function<void()>> queue_;
  size_t idle_ = 0;
};

using su2g::small_count;

// One stream's part of a truncation: its allocations (from the pool, on the
// stream; released on `free_st` once the caller's stream has used them) and its
// error state.
struct Ctx {
  cudaStream_t st = nullptr;
  cudaStream_t free_st = nullptr;
  cudaMemPool_t pool = nullptr;
  cusolverDnHandle_t sol = nullptr;
  cusolverDnParams_t params = nullptr;
  std::vector<void*> allocs;
  std::string err;
  int code = SU2G_OK;

  Ctx(const Lane& lane, cudaStream_t free_stream, cudaMemPool_t p)
      : st(lane.st), free_st(free_stream), pool(p), sol(lane.sol), params(lane.params) {}
  Ctx(const Ctx&) = delete;
  Ctx& operator=(const Ctx&) = delete;
  ~Ctx() {
    for (void* p : allocs) cudaFreeAsync(p, free_st);
  }
  bool ok() const { return code == SU2G_OK; }
  void set(int c, const std::string& m) {
    if (code == SU2G_OK) {
      code = c;
      err = m;
    }
  }
  void cuda(cudaError_t e) {
    if (e != cudaSuccess) set(SU2G_ECUDA, std::string("svd: ") + cudaGetErrorString(e));
  }
  void* bytes(size_t n) {
    void* p = nullptr;
    cudaError_t e = cudaMallocFromPoolAsync(&p, std::max<size_t>(n, 8), pool, st);
    if (e != cudaSuccess) {
      set(e == cudaErrorMemoryAllocation ? SU2G_ENOMEM : SU2G_ECUDA, std::string("svd: ") + cudaGetErrorString(e));
      return nullptr;
    }
    allocs.push_back(p);
    return p;
  }
  double* dalloc(int64_t n) { return (double*)bytes((size_t)std::max<int64_t>(n, 1) * sizeof(double)); }
  // products on the library's FP64 tile engine: every element sums its
  // products in a fixed order, whatever else runs on the GPU
  void gemms(const std::vector<su2g::DenseGemm>& jobs) {
    if (ok()) cuda(su2g::launch_gemm_f64_dense_many(jobs.data(), (int)jobs.size(), st));
  }
  template <class J, class C, class... A>
  void launch(void (*kernel)(JobList<J>, int, A...), const std::vector<J>& jobs, C ctas, size_t smem, A... args) {
    if (ok()) cuda(launch_jobs(kernel, jobs, ctas, 256, smem, st, args...));
  }
  void signs(const std::vector<SignJob>& jobs) {
    launch(canonical_signs_kernel, jobs, [](const SignJob& j) { return j.n; }, 0);
  }
  void copies(const std::vector<CopyJob>& jobs) {
    launch(copy_arrays, jobs, [](const CopyJob& j) { return (int)((j.len + kCopyTile - 1) / kCopyTile); }, 0);
  }
  // device -> host, and everything queued so far is done
  void fetch(void* dst, const void* src, size_t n) {
    if (!ok()) return;
    cudaError_t e = cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cuda(e);
  }
  // out (cols x rows) = in^T (in: rows x cols, column-major)
  void transpose(const double* in, int rows, int cols, double* out) {
    if (!ok() || rows == 0 || cols == 0) return;
    const dim3 grid((cols + 31) / 32, (rows + 31) / 32);
    transpose_kernel<<<grid, dim3(32, 8), 0, st>>>(in, rows, cols, out);
    cuda(cudaGetLastError());
  }
  // symmetric eigendecomposition in place (a: n x n, ld n); w: host eigenvalues
  void eigh(double* a, int n, std::vector<double>* w) {
    if (!ok()) return;
    int lwork = 0;
    double* dw = dalloc(n + 1);
    if (!ok()) return;
    if (cusolverDnDsyevd_bufferSize(sol, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, n, a, n, dw, &lwork) !=
        CUSOLVER_STATUS_SUCCESS) {
      set(SU2G_ECUDA, "svd: syevd buffer query failed");
      return;
    }
    double* work = dalloc(lwork);
    if (!ok()) return;
    if (cusolverDnDsyevd(sol, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, n, a, n, dw, work, lwork,
                         (int*)(dw + n)) != CUSOLVER_STATUS_SUCCESS) {
      set(SU2G_ECUDA, "svd: syevd failed");
      return;
    }
    std::vector<double> h(n + 1);
    fetch(h.data(), dw, h.size() * sizeof(double));
    int info = 0;
    std::memcpy(&info, &h[n], sizeof(info));
    if (ok() && info != 0) set(SU2G_ECUDA, "svd: syevd did not converge (info " + std::to_string(info) + ")");
    w->assign(h.begin(), h.begin() + n);
  }
};

// A matrix to decompose in place and where its eigenvalues go.
struct EighJob {
  double* a;
  int n;
  std::vector<double>* w;
};

// cuSOLVER's solver is a chain of small launches (4.8 ms for 108 rows, 0.4 for
// 16).  The decompositions that refinement levels still need go through it
// together, padded to the largest: 14 of up to 54 rows take 1.4 ms.  From 160
// rows on a batch is the slower way (14 of 160: 10.7 ms, of 555: 69, and 15 ms
// for one alone).  The first pass keeps a stream and a host thread for each of
// eight sectors at a time, largest first (a truncation at D = 400, 14 sectors of
// up to 108 rows: 9.1 ms; 11.1 with all 14 at once, whose threads wait for one
// another in CUDA's launch path, 10.6 with six; D = 2000: 95, 97 and 101).  A batch
// would be faster (6.8), but the Gram matrix is known to its rounding only, so the
// directions of its smallest eigenvalues are whatever the solver makes of that,
// and a padded matrix gives other ones: the new tensors move by 7e-10, without
// it by 6e-11.
constexpr size_t kEighLanes = 8;
constexpr int kBatchEigh = 128;

// one sector of the truncation
struct Sector {
  int i = -1;  // leg-0 sector index
  int m = 0, n = 0;
  const double* blk = nullptr;
  bool tall = true;  // the Gram matrix is blk^T blk
  int k = 0;         // its size
  double* A0 = nullptr;
  double* G = nullptr;    // eigenvectors
  std::vector<double> w;  // eigenvalues, ascending
  // refinement: the level's size, the size before it, and the buffers
  int np = 0, npp = 0;
  double *M = nullptr, *V = nullptr;  // the matrix and the basis it was projected from
  double* buf[7] = {};                // k x k each
  double *nextM = nullptr, *x = nullptr, *y = nullptr, *p = nullptr, *q = nullptr;
  double* lam = nullptr;  // device: npp + 1, as StepJob's
  const double* h = nullptr;  // the same on the host
  std::vector<double> ws;     // the level's eigenvalues
  std::vector<int> levels;    // trace: the levels' sizes
  // result
  int dc = 0;           // singular values kept by the sector's own rule
  double* u = nullptr;  // m x dc (ld m), smallest first
  double* v = nullptr;  // n x dc (ld n)
  std::vector<double> s;  // dc values, ascending

  // buffers for the next level: those that M and V do not hold
  void assign() {
    int at = 0;
    auto next = [&] {
      while (buf[at] == M || buf[at] == V) ++at;
      return buf[at++];
    };
    nextM = next();
    x = next();
    y = next();
    p = next();
    q = next();
  }
};

// The sectors of a truncation in lockstep: every step (a product, a
// correction, a copy) is one launch for all of them, and the host reads all
// their eigenvalues back at once.  With a stream and a host thread for each
// sector, ten launches a level and sector fought for CUDA's launch path: nine levels of
// 14 sectors took 5 ms, in lockstep 2.6, half of it the last levels' solver.
class Truncation {
 public:
  // decomposes the jobs on other streams and runs `beside` meanwhile
  using OnLanes = std::function<void(const std::vector<EighJob>&, const std::function<void()>& beside)>;
  Truncation(Ctx& ctx, std::vector<Sector>& sectors, OnLanes lanes)
      : c(ctx), secs(sectors), on_lanes(std::move(lanes)) {}

  // First pass of tensor::svd (n0 = 1): the Gram matrix of every sector's
  // smaller side and its eigendecomposition (tensor.cpp:1484-1490).
  void first_pass() {
    std::vector<su2g::DenseGemm> gram;
    std::vector<CopyJob> keep;
    std::vector<EighJob> eig;
    std::vector<SignJob> signs;
    for (Sector& s : secs) {
      s.tall = s.m >= s.n;
      const int k = s.k = std::min(s.m, s.n), r = std::max(s.m, s.n);
      const int64_t kk = (int64_t)k * k;
      s.A0 = c.dalloc(kk);
      s.G = c.dalloc(kk);
      const double* b = s.blk;
      if (!s.tall) {  // blk blk^T = (blk^T)^T (blk^T)
        double* bt = c.dalloc((int64_t)s.m * s.n);
        if (!c.ok()) return;
        c.transpose(s.blk, s.m, s.n, bt);
        b = bt;
      }
      if (!c.ok()) return;
      gram.push_back({true, k, k, r, b, r, b, r, s.A0, k});
      keep.push_back({s.G, s.A0, kk});
      eig.push_back({s.G, k, &s.w});
      signs.push_back({s.G, k});
    }
    c.gemms(gram);
    c.copies(keep);
    eigh(eig, false);
    c.signs(signs);  // G now holds the eigenvectors
  }

  // The reference's refinement of the small-eigenvalue subspaces
  // (tensor.cpp:1491-1529).  Each refinement re-solves the
  // subspace of eigenvalues below 0.1 of its largest and rotates only those
  // columns, so a subspace whose largest eigenvalue is below 0.1 of lam_cut (the
  // max_dcut-th largest eigenvalue over all sectors, 0 when every multiplet is
  // kept or when the cut is too close to the first pass's rounding error to be
  // placed) holds no multiplet the truncation keeps: refining it further changes
  // neither the kept columns, their values nor the selection, and is skipped
  // (its values, all discarded, stay those of the last refinement).
  void refine(double lam_cut) {
    cut = lam_cut;
    std::vector<Sector*> run, wait;
    int64_t nlam = 0;
    for (Sector& s : secs) {
      s.npp = small_count(s.w, s.k);
      if (s.npp <= 1 || beyond_cut(s.w, s.npp)) continue;
      s.np = s.k;
      s.M = s.A0;
      s.V = s.G;
      for (double*& b : s.buf) b = c.dalloc((int64_t)s.k * s.k);
      nlam += s.k + 1;
      run.push_back(&s);
    }
    lam_dev = c.dalloc(nlam);
    if (!c.ok()) return;
    lam_host.resize(nlam);
    int64_t at = 0;
    for (Sector* s : run) {
      s->lam = lam_dev + at;
      s->h = lam_host.data() + at;
      at += s->k + 1;
    }
    // Sectors whose level needs an eigendecomposition wait until no other can
    // go on without one: they are decomposed together.
    while (c.ok() && !(run.empty() && wait.empty())) {
      if (run.empty()) {
        std::vector<CopyJob> copies;
        std::vector<EighJob> eig;
        for (Sector* s : wait) {
          copies.push_back({s->x, s->nextM, (int64_t)s->npp * s->npp});
          eig.push_back({s->x, s->npp, &s->ws});
        }
        c.copies(copies);
        eigh(eig, true);
        run = finish_level(wait);
        wait.clear();
        continue;
      }
      const std::vector<Sector*> solved = level(run, &wait);
      run = finish_level(solved);
    }
  }

  // The other factors, singular values above 1e-100 of the largest, scaling
  // (tensor.cpp:1530-1567).
  void factors(double p1, double p2, int max_dcut) {
    std::vector<su2g::DenseGemm> gemms;
    std::vector<double> f;
    for (Sector& s : secs) {
      const int m = s.m, n = s.n, k = s.k;
      double *U, *V;
      if (s.tall) {  // V = eigenvectors (n x n), U = blk V (m x n)
        V = s.G;
        U = c.dalloc((int64_t)m * n);
        gemms.push_back({false, m, n, n, s.blk, m, V, n, U, m});
      } else {  // U = eigenvectors (m x m), V = blk^T U (n x m)
        U = s.G;
        V = c.dalloc((int64_t)n * m);
        gemms.push_back({true, n, m, m, s.blk, m, U, m, V, n});
      }
      const double num = s.w[k - 1];
      int dcut = 0;
      if (num > 1.e-100)
        for (int i = k - 1; i >= 0; --i) {
          if (s.w[i] / num > 1.e-100) {
            s.w[i] = std::sqrt(s.w[i]);
            ++dcut;
          } else {
            s.w[i] = 0;
          }
        }
      if (dcut > max_dcut) dcut = max_dcut;
      s.dc = dcut;
      s.u = U;
      s.v = V;
      s.s.assign(s.w.begin() + (k - dcut), s.w.begin() + k);
      for (int side = 0; side < 2; ++side)
        for (double x : s.s) {
          const double down = s.tall ? std::pow(x, p1 - 1.) : std::pow(x, p1);
          const double across = s.tall ? std::pow(x, p2) : std::pow(x, p2 - 1.);
          f.push_back(x > 0 ? (side ? across : down) : 0.0);
        }
    }
    c.gemms(gemms);
    double* df = c.dalloc((int64_t)f.size());
    if (!c.ok()) return;
    if (!f.empty()) c.cuda(cudaMemcpyAsync(df, f.data(), f.size() * sizeof(double), cudaMemcpyHostToDevice, c.st));
    std::vector<ScaleJob> scale;
    int64_t at = 0;
    for (Sector& s : secs) {
      scale.push_back({s.u, s.m, s.k - s.dc, s.dc, df + at});
      scale.push_back({s.v, s.n, s.k - s.dc, s.dc, df + at + s.dc});
      at += 2 * s.dc;
      s.u += (int64_t)s.m * (s.k - s.dc);
      s.v += (int64_t)s.n * (s.k - s.dc);
    }
    c.launch(scale_columns, scale, [](const ScaleJob& j) { return j.ncol; }, 0);
  }

 private:
  bool beyond_cut(const std::vector<double>& w, int n) const { return su2g::beyond_cut(w, n, cut); }

  // eigendecompositions in place, signs as they come: each on a stream and
  // host thread of its own, or (together) the small ones as a batch beside them
  void eigh(const std::vector<EighJob>& jobs, bool together) {
    std::vector<EighJob> small, alone;
    for (const EighJob& j : jobs) (together && j.n <= kBatchEigh ? small : alone).push_back(j);
    if (alone.empty()) {
      batch(small);
    } else if (c.ok()) {
      c.cuda(cudaStreamSynchronize(c.st));  // the matrices are there for the other streams
      if (c.ok()) on_lanes(alone, [&] { batch(small); });
    }
  }
  void batch(const std::vector<EighJob>& small) {
    if (small.size() == 1) {
      c.eigh(small[0].a, small[0].n, small[0].w);
    } else if (!small.empty()) {
      int N = 0;
      for (const EighJob& j : small) N = std::max(N, j.n);
      const int nb = (int)small.size();
      double* box = c.dalloc((int64_t)nb * N * N);
      double* dw = c.dalloc((int64_t)nb * (N + 1));  // eigenvalues, then info
      if (!c.ok()) return;
      int* info = (int*)(dw + (int64_t)nb * N);
      std::vector<PadJob> pads;
      for (int q = 0; q < nb; ++q) pads.push_back({small[q].a, small[q].n, box + (int64_t)q * N * N});
      c.launch(pad_matrix, pads, [&](const PadJob&) { return N; }, 0, N);
      size_t ldev = 0, lhost = 0;
      if (c.ok() && cusolverDnXsyevBatched_bufferSize(c.sol, c.params, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER,
                                                      N, CUDA_R_64F, box, N, CUDA_R_64F, dw, CUDA_R_64F, &ldev, &lhost,
                                                      nb) != CUSOLVER_STATUS_SUCCESS)
        c.set(SU2G_ECUDA, "svd: syev buffer query failed");
      void* work = c.bytes(ldev);
      std::vector<uint8_t> host(lhost);
      if (c.ok() && cusolverDnXsyevBatched(c.sol, c.params, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, N,
                                           CUDA_R_64F, box, N, CUDA_R_64F, dw, CUDA_R_64F, work, ldev, host.data(),
                                           lhost, info, nb) != CUSOLVER_STATUS_SUCCESS)
        c.set(SU2G_ECUDA, "svd: syev failed");
      c.launch(unpad_vectors, pads, [](const PadJob& j) { return j.n; }, 0, N);
      std::vector<double> h((size_t)nb * (N + 1));
      c.fetch(h.data(), dw, h.size() * sizeof(double));
      if (!c.ok()) return;
      const int* hinfo = (const int*)(h.data() + (size_t)nb * N);
      for (int q = 0; q < nb; ++q) {
        if (hinfo[q] != 0)
          c.set(SU2G_ECUDA, "svd: syev did not converge (info " + std::to_string(hinfo[q]) + ")");
        small[q].w->assign(h.begin() + (size_t)q * N + (N - small[q].n), h.begin() + (size_t)(q + 1) * N);
      }
    }
  }

  // One level of every sector of `run`: the Gram matrix projected on the
  // subspace (nextM) and its eigenvectors (x) by refinement of the basis at
  // hand.  Returns the sectors solved; the others, for which couplings are too
  // large for the gaps, the order of the values is not settled, or the
  // subspace left is the last to be looked at (its values are reported as they
  // are), go to `wait`.
  std::vector<Sector*> level(const std::vector<Sector*>& run, std::vector<Sector*>* wait) {
    std::vector<su2g::DenseGemm> g1, g2;
    for (Sector* s : run) {
      const int np = s->np, npp = s->npp;
      s->assign();
      s->levels.push_back(npp);
      g1.push_back({true, npp, np, np, s->V, np, s->M, np, s->y, npp});
      g2.push_back({false, npp, npp, np, s->y, npp, s->V, np, s->nextM, npp});
    }
    c.gemms(g1);
    c.gemms(g2);
    std::vector<Sector*> open, solved;
    for (Sector* s : run) (s->npp <= kRefineMax ? open : *wait).push_back(s);
    for (int it = 0; it < 4 && !open.empty() && c.ok(); ++it) {
      if (it > 0) {
        g1.clear();
        g2.clear();
        for (Sector* s : open) {
          const int n = s->npp;
          g1.push_back({false, n, n, n, s->nextM, n, s->x, n, s->y, n});
          g2.push_back({true, n, n, n, s->x, n, s->y, n, s->q, n});  // S
          g2.push_back({true, n, n, n, s->x, n, s->x, n, s->p, n});  // P
        }
        c.gemms(g1);
        c.gemms(g2);
      }
      std::vector<StepJob> step;
      int most = 0;
      for (Sector* s : open) {
        step.push_back({it > 0 ? s->q : s->nextM, it > 0 ? s->p : nullptr, s->npp, it > 0 ? s->y : s->x, s->lam});
        most = std::max(most, s->npp);
      }
      if (c.ok()) c.cuda(cudaMemsetAsync(lam_dev, 0, lam_host.size() * sizeof(double), c.st));
      c.launch(refine_step_kernel, step, [](const StepJob& j) { return j.n; }, most * sizeof(double));
      c.fetch(lam_host.data(), lam_dev, lam_host.size() * sizeof(double));
      if (!c.ok()) return {};
      std::vector<Sector*> more;
      g1.clear();
      for (Sector* s : open) {
        const int n = s->npp;
        if (!su2g::level_settled(std::vector<double>(s->h, s->h + n), s->h[n], it, cut)) {
          wait->push_back(s);
          continue;
        }
        if (it > 0) {
          g1.push_back({false, n, n, n, s->x, n, s->y, n, s->q, n});
          std::swap(s->x, s->q);
        }
        if (s->h[n] <= kStepDone) {
          s->ws.assign(s->h, s->h + n);
          solved.push_back(s);
        } else {
          more.push_back(s);
        }
      }
      c.gemms(g1);
      open = more;
    }
    wait->insert(wait->end(), open.begin(), open.end());
    return solved;
  }

  // Rotates the solved sectors' columns and goes on to their next levels;
  // returns the sectors that have one.
  std::vector<Sector*> finish_level(const std::vector<Sector*>& solved) {
    std::vector<SignJob> signs;
    std::vector<su2g::DenseGemm> rotate;
    std::vector<CopyJob> copies;
    std::vector<Sector*> next;
    if (!c.ok()) return next;
    for (Sector* s : solved) {
      const int k = s->k, n = s->npp;
      signs.push_back({s->x, n});
      // s->G may still be the basis of the first level: it is not read after this
      rotate.push_back({false, k, n, n, s->G, k, s->x, n, s->y, k});
      copies.push_back({s->G, s->y, (int64_t)k * n});
      std::copy(s->ws.begin(), s->ws.end(), s->w.begin());
      s->V = s->x;
      s->M = s->nextM;
      s->np = n;
      s->npp = small_count(s->ws, n);
      if (s->npp > 1 && !beyond_cut(s->ws, s->npp)) next.push_back(s);
    }
    c.signs(signs);
    c.gemms(rotate);
    c.copies(copies);
    return next;
  }

  Ctx& c;
  std::vector<Sector>& secs;
  OnLanes on_lanes;
  double cut = 0;
  double* lam_dev = nullptr;
  std::vector<double> lam_host;
};

}  // namespace

bool same_sectors(const su2g::Bond& a, const su2g::Bond& b) { return a.angm == b.angm && a.dim == b.dim; }

extern "C" int su2g_svd(const int* psi_desc, const int* psi_flag, const double* psi, const int* tu_desc, double p1,
                        const int* tv_desc, double p2, int max_dcut, int* bond, int bond_cap, double* wout,
                        int wout_cap, int* dout, double* tu, int64_t tu_cap, double* tv, int64_t tv_cap,
                        void* stream) {
  su2g::Struct P, TU, TV;
  std::string e;
  if (!psi_desc || !P.parse(psi_desc, &e)) return fail(SU2G_EINVAL, "svd: psi: " + e);
  if (P.nbond != 2) return fail(SU2G_EINVAL, "svd: psi must have 2 legs");
  if (!tu_desc || !TU.parse(tu_desc, &e) || TU.nbond != 3) return fail(SU2G_EINVAL, "svd: tu: 3-leg desc expected " + e);
  if (!tv_desc || !TV.parse(tv_desc, &e) || TV.nbond != 3) return fail(SU2G_EINVAL, "svd: tv: 3-leg desc expected " + e);
  if (!bond || !wout || !dout || max_dcut < 0) return fail(SU2G_EINVAL, "svd: bad arguments");
  // psi legs are the fused (tu leg 0, tu leg 1) and (tv leg 0, tv leg 1) (tensor_su2.cpp:1628-1634)
  if (!same_sectors(su2g::fuse(TU.legs[0], TU.legs[1]), P.legs[0]) ||
      !same_sectors(su2g::fuse(TV.legs[0], TV.legs[1]), P.legs[1]))
    return fail(SU2G_EINVAL, "svd: psi legs are not the fused legs 0, 1 of tu / tv");
  P.set_layout(psi_flag);
  if (P.total > 0 && !psi) return fail(SU2G_EINVAL, "svd: null psi");
  cudaStream_t cst = (cudaStream_t)stream;
  // SU2G_SVD_TRACE=<file>: one JSON line per call appended there (per sector:
  // m, n, Gram size, host milliseconds of the call's two passes, the sizes of
  // the refinement subspaces), for time breakdowns of whole sweeps
  const char* trace = std::getenv("SU2G_SVD_TRACE");
  if (trace && !*trace) trace = nullptr;
  const auto t_call = std::chrono::steady_clock::now();
  const int n0 = P.legs[0].n(), n1 = P.legs[1].n();
  // sectors in the reference's loop order: leg-0 sector, then the leg-1 sector of equal spin
  struct Job {
    int i, b, m, n;
  };
  std::vector<Job> jobs;
  for (int i = 0; i < n0; ++i)
    for (int j = 0; j < n1; ++j) {
      if (P.legs[0].angm[i] != P.legs[1].angm[j]) continue;
      const int b = i + j * n0;
      if (P.flag[b]) jobs.push_back(Job{i, b, P.legs[0].dim[i], P.legs[1].dim[j]});
    }
  int dev = 0;
  cudaError_t ce = cudaGetDevice(&dev);
  if (ce != cudaSuccess) return fail(SU2G_ECUDA, std::string("svd: ") + cudaGetErrorString(ce));
  // lane 0 for everything the sectors share, the others for decompositions
  std::vector<Lane> lanes;
  cudaMemPool_t pool = nullptr;
  const std::string rerr = take_lanes(dev, 1 + (int)std::min<size_t>(jobs.size(), kEighLanes), &lanes, &pool);
  if (!rerr.empty()) {
    give_lanes(dev, lanes);
    return fail(SU2G_ECUDA, "svd: " + rerr);
  }
  // the lanes go back to the device's free list when the call returns
  struct LaneReturn {
    int dev;
    const std::vector<Lane>& lanes;
    ~LaneReturn() { give_lanes(dev, lanes); }
  } lane_return{dev, lanes};
  std::vector<std::unique_ptr<Ctx>> ctx;
  for (const Lane& l : lanes) ctx.emplace_back(new Ctx(l, cst, pool));
  Ctx& c = *ctx[0];
  std::vector<Sector> secs(jobs.size());
  for (size_t q = 0; q < jobs.size(); ++q) {
    secs[q].i = jobs[q].i;
    secs[q].m = jobs[q].m;
    secs[q].n = jobs[q].n;
    secs[q].blk = psi + P.offset[jobs[q].b];
  }
  // psi is written on the caller's stream
  cudaEvent_t order = nullptr;
  ce = cudaEventCreateWithFlags(&order, cudaEventDisableTiming);
  if (ce == cudaSuccess) ce = cudaEventRecord(order, cst);
  if (ce == cudaSuccess) ce = cudaStreamWaitEvent(c.st, order, 0);
  c.cuda(ce);
  Truncation tr(c, secs, [&](const std::vector<EighJob>& alone, const std::function<void()>& beside) {
    // largest first, each lane taking the next when it is through with one
    std::vector<EighJob> order(alone);
    std::stable_sort(order.begin(), order.end(), [](const EighJob& x, const EighJob& y) { return x.n > y.n; });
    std::atomic<size_t> next{0};
    SectorThreads::get().run(std::min(ctx.size() - 1, alone.size()) + 1, [&](size_t q) {
      if (q == 0) {
        beside();
        return;
      }
      Ctx& mine = *ctx[q];
      mine.cuda(cudaSetDevice(dev));
      for (size_t j = next++; j < order.size(); j = next++) mine.eigh(order[j].a, order[j].n, order[j].w);
    });
    for (size_t q = 1; q < ctx.size(); ++q)
      if (!ctx[q]->ok()) c.set(ctx[q]->code, ctx[q]->err);
  });
  const auto t_eig = std::chrono::steady_clock::now();
  if (c.ok()) tr.first_pass();
  const auto t_refine = std::chrono::steady_clock::now();
  double lam_cut = 0.0, lam_cut_raw = 0.0, noise_floor = 0.0;
  if (c.ok()) {
    // the max_dcut-th largest eigenvalue over all sectors; 0 (refine every
    // subspace, as the reference) when nothing is cut or when the cut lies
    // within 1e3 of the first pass's error k eps lambda_max of some sector,
    // where values near it are not yet known well enough to place them
    std::vector<double> all;
    double floor = 0.0;
    for (const Sector& s : secs) {
      const double top = s.w.empty() ? 0.0 : s.w.back();
      floor = std::max(floor, (double)s.k * 2.3e-16 * top);
      for (double v : s.w)
        if (v > 0 && v / top > 1.e-100) all.push_back(v);
    }
    if (max_dcut > 0 && (int64_t)all.size() > max_dcut) {
      std::nth_element(all.begin(), all.begin() + (max_dcut - 1), all.end(), std::greater<double>());
      lam_cut = lam_cut_raw = all[max_dcut - 1];
      if (lam_cut < 1e3 * floor) lam_cut = 0.0;
    }
    noise_floor = floor;
    tr.refine(lam_cut);
  }
  if (c.ok()) tr.factors(p1, p2, max_dcut);
  if (trace) cudaStreamSynchronize(c.st);
  const auto t_done = std::chrono::steady_clock::now();
  // the caller's stream continues after the sectors' (placement copies, frees)
  if (order) {
    ce = cudaEventRecord(order, c.st);
    if (ce == cudaSuccess) ce = cudaStreamWaitEvent(cst, order, 0);
    cudaEventDestroy(order);
    c.cuda(ce);
  }
  if (!c.ok()) return fail(c.code, c.err);
  // global selection of the max_dcut largest multiplets (tensor_su2.cpp:1686-1695)
  std::vector<double> ws;
  std::vector<int> is;
  for (const Sector& s : secs)
    for (int q = 0; q < s.dc; ++q) {
      ws.push_back(s.s[q]);
      is.push_back(s.i);
    }
  const int n = (int)ws.size();
  su2g::dsort2(n, ws.data(), is.data());
  std::vector<int> dim(n0, 0);
  for (int q = n - 1; q >= std::max(0, n - max_dcut); --q) ++dim[is[q]];
  // the new bond: kept sectors of psi leg 0, direction -1 (tensor_su2.cpp:1733)
  su2g::Bond nb;
  nb.dir = -1;
  for (int i = 0; i < n0; ++i)
    if (dim[i] > 0) {
      nb.angm.push_back(P.legs[0].angm[i]);
      nb.dim.push_back(dim[i]);
    }
  if (bond_cap < 1 + 2 * nb.n()) return fail(SU2G_EINVAL, "svd: bond output too small");
  bond[0] = nb.n();
  for (int q = 0; q < nb.n(); ++q) {
    bond[1 + q] = nb.angm[q];
    bond[1 + nb.n() + q] = nb.dim[q];
  }
  // kept values (per sector, ascending), then the discarded ones (tensor_su2.cpp:1706-1731)
  if (n > wout_cap) return fail(SU2G_EINVAL, "svd: wout too small (" + std::to_string(n) + " values)");
  int total_kept = 0;
  for (int d : dim) total_kept += d;
  int mk = 0, md = total_kept;
  for (const Sector& s : secs) {
    const int d = dim[s.i];
    for (int q = 0; q < d; ++q) wout[mk + q] = s.s[s.dc - d + q];
    for (int q = 0; q < s.dc - d; ++q) wout[md + q] = s.s[q];
    mk += d;
    md += s.dc - d;
  }
  *dout = md;
  // tu = fuse(tu legs 0, 1) x kept U, tv likewise with V: row ranges of the
  // kept columns, every legal block present (tensor_su2.cpp:1733-1745)
  for (int side = 0; side < 2; ++side) {
    double* out = side ? tv : tu;
    if (!out) continue;
    const su2g::Struct& T = side ? TV : TU;
    su2g::Struct O;
    O.nbond = 3;
    O.locspin = 0;
    O.legs[0] = T.legs[0];
    O.legs[1] = T.legs[1];
    O.legs[2] = nb;
    O.nten = O.legs[0].n() * O.legs[1].n() * nb.n();
    O.set_layout(nullptr);
    if (O.total > (side ? tv_cap : tu_cap))
      return fail(SU2G_EINVAL, std::string("svd: ") + (side ? "tv" : "tu") + " output too small (" +
                                   std::to_string(O.total) + " doubles)");
    for (int b = 0; b < O.nten; ++b) {
      if (!O.flag[b]) continue;
      int sec[3];
      O.sectors(b, sec);
      const int ang = nb.angm[sec[2]], d = nb.dim[sec[2]];
      const Sector* src = nullptr;
      for (const Sector& s : secs)
        if (P.legs[0].angm[s.i] == ang) src = &s;
      const int r0 = su2g::fused_row(O.legs[0], O.legs[1], ang, sec[0], sec[1]);
      const int rows = O.legs[0].dim[sec[0]] * O.legs[1].dim[sec[1]];
      if (!src || r0 < 0) return fail(SU2G_EINVAL, "svd: internal placement error");
      const int ld = side ? src->n : src->m;
      const double* col0 = (side ? src->v : src->u) + (int64_t)ld * (src->dc - d) + r0;
      const cudaError_t me = cudaMemcpy2DAsync(out + O.offset[b], rows * sizeof(double), col0,
                                               ld * sizeof(double), rows * sizeof(double), d,
                                               cudaMemcpyDeviceToDevice, cst);
      if (me != cudaSuccess) return fail(SU2G_ECUDA, std::string("svd: ") + cudaGetErrorString(me));
    }
  }
  ce = cudaStreamSynchronize(cst);
  if (ce != cudaSuccess) return fail(SU2G_ECUDA, std::string("svd: ") + cudaGetErrorString(ce));
  if (trace) {
    static std::mutex trace_mu;
    std::lock_guard<std::mutex> tl(trace_mu);
    if (FILE* f = std::fopen(trace, "a")) {
      const double ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_call).count();
      std::fprintf(f,
                   "{\"ms\": %.3f, \"max_dcut\": %d, \"lam_cut\": %.6e, \"lam_cut_raw\": %.6e, "
                   "\"noise_floor\": %.6e, \"kept\": %d, \"sectors\": [",
                   ms, max_dcut, lam_cut, lam_cut_raw, noise_floor, total_kept);
      for (size_t q = 0; q < jobs.size(); ++q) {
        std::fprintf(f, "%s{\"m\": %d, \"n\": %d, \"k\": %d, \"ms_eig\": %.3f, \"ms_finish\": %.3f, \"levels\": [",
                     q ? ", " : "", jobs[q].m, jobs[q].n, secs[q].k,
                     std::chrono::duration<double, std::milli>(t_refine - t_eig).count(),
                     std::chrono::duration<double, std::milli>(t_done - t_refine).count());
        for (size_t l = 0; l < secs[q].levels.size(); ++l) std::fprintf(f, "%s%d", l ? ", " : "", secs[q].levels[l]);
        std::fprintf(f, "]}");
      }
      std::fprintf(f, "]}\n");
      std::fclose(f);
    }
  }
  return SU2G_OK;
}
