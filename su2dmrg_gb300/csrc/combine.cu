// Linear combinations of block tensors of one structure, and the device-scalar
// axpy behind the excited-state projector of H_eff.
//
// out = sum_i coef_i op_i is how the reference forms the summed partner of
// each H_eff term (tmp = opr[ir][k]; tmp *= coup; op += tmp,
// dmrg_su2.cpp:588-600) and the site-step sums (hh[i] += hh2[j],
// dmrg_su2_omp.cpp:462-469).  The output holds the union of the operands'
// blocks (tensor_su2::operator+= creates missing blocks, tensor_su2.cpp:152-200);
// every element is summed in operand order, so the result does not depend on
// the launch shape.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <vector>

#include "kernels.hpp"
#include "su2_meta.hpp"
#include "su2g.h"

namespace {

int fail(int code, const std::string& msg) { return su2g::set_last_error(code, msg); }

// A run: consecutive output blocks that the same operands hold, which are
// consecutive in each of those operands too (operands of one flag set make one
// run of the whole tensor).
struct CombRun {
  int64_t dst;    // element offset in out
  int64_t len;
  int64_t tile0;  // first tile of this run in the launch
  int src0, nsrc;  // range in the source list
};
struct CombSrc {
  const double* p;  // the operand's copy of this run
  double c;
};
// The lists travel in the kernel's parameters (3.6 KB, below the 4 KB every
// launch has): nothing is allocated, copied or waited for before the launch.
// More runs take more launches; where a run may have more sources than a list
// holds, all the sources go to device memory in one copy instead.
constexpr int kCombRuns = 32, kCombSrcs = 160;
struct CombList {
  CombRun run[kCombRuns];
  CombSrc src[kCombSrcs];
};

constexpr int kCombThreads = 256, kCombElems = 2;
constexpr int kCombTile = kCombThreads * kCombElems;

// One tile of one run a CTA, two elements a thread (coalesced; two elements
// times four sources in flight, and three CTAs an SM already at 230,000
// elements).  HBM-bound in principle; six operands of 1.9 MB (D = 900) are in
// L2 or launch-bound.  With the lists allocated and copied for each call such
// a sum took its caller 110 us (408 with the default pool cold), now 70, most of
// it the caller's own marshalling.
__global__ void __launch_bounds__(kCombThreads) combine_kernel(const __grid_constant__ CombList list, int nrun,
                                                               const CombSrc* many, double* out) {
  int r = 0;
  while (r + 1 < nrun && list.run[r + 1].tile0 <= blockIdx.x) ++r;
  const CombRun it = list.run[r];
  const int64_t e0 = (blockIdx.x - it.tile0) * kCombTile + threadIdx.x;
  const bool in0 = e0 < it.len, in1 = e0 + kCombThreads < it.len;
  double* o = out + it.dst + e0;
  double a0 = 0.0, a1 = 0.0;
#pragma unroll 4
  for (int s = 0; s < it.nsrc; ++s) {
    const CombSrc q = many ? many[it.src0 + s] : list.src[it.src0 + s];
    const double x0 = in0 ? q.p[e0] : 0.0, x1 = in1 ? q.p[e0 + kCombThreads] : 0.0;
    a0 += q.c * x0;
    a1 += q.c * x1;
  }
  if (in0) o[0] = a0;
  if (in1) o[kCombThreads] = a1;
}

// The launches of one linear combination of n operands: runs and their sources
// are added one by one and sent whenever a list is full; with more operands than
// a list holds, once all are known (200 operands that hold different blocks: 356
// us, 1,294 with a copy and a wait for each run).
class CombLauncher {
 public:
  CombLauncher(int n, double* out, cudaStream_t st) : many_(n > kCombSrcs), out_(out), st_(st) {}
  void add(int64_t dst, int64_t len, const std::vector<CombSrc>& src) {
    if (!many_ && (nrun_ == kCombRuns || nsrc_ + (int)src.size() > kCombSrcs)) send(list_.run, nrun_, nullptr);
    const CombRun r{dst, len, 0, many_ ? (int)srcs_.size() : nsrc_, (int)src.size()};
    if (many_) {
      runs_.push_back(r);
      srcs_.insert(srcs_.end(), src.begin(), src.end());
      return;
    }
    std::copy(src.begin(), src.end(), list_.src + nsrc_);
    nsrc_ += (int)src.size();
    list_.run[nrun_++] = r;
  }
  cudaError_t finish() {
    if (!many_) {
      send(list_.run, nrun_, nullptr);
      return e_;
    }
    void* d = nullptr;
    if (!srcs_.empty()) e_ = su2g::upload_bytes(srcs_.data(), srcs_.size() * sizeof(CombSrc), &d);
    for (size_t r = 0; r < runs_.size() && e_ == cudaSuccess; r += kCombRuns)
      send(runs_.data() + r, (int)std::min<size_t>(kCombRuns, runs_.size() - r), (const CombSrc*)d);
    su2g::dev_free(d, st_);
    return e_;
  }

 private:
  void send(const CombRun* runs, int n, const CombSrc* many) {
    int64_t tiles = 0;
    for (int r = 0; r < n; ++r) {
      list_.run[r] = runs[r];
      list_.run[r].tile0 = tiles;
      tiles += (runs[r].len + kCombTile - 1) / kCombTile;
    }
    if (tiles > 0 && e_ == cudaSuccess) {
      combine_kernel<<<(unsigned)tiles, kCombThreads, 0, st_>>>(list_, n, many, out_);
      e_ = cudaGetLastError();
    }
    nrun_ = nsrc_ = 0;
  }
  const bool many_;
  CombList list_{};
  std::vector<CombRun> runs_;
  std::vector<CombSrc> srcs_;
  int nrun_ = 0, nsrc_ = 0;
  double* out_;
  cudaStream_t st_;
  cudaError_t e_ = cudaSuccess;
};

__global__ void axpy_dev_kernel(double alpha, const double* __restrict__ scale, const double* __restrict__ x,
                                double* __restrict__ y, int64_t n) {
  const double a = alpha * *scale;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    y[i] += a * x[i];
}

bool same_legs(const su2g::Struct& a, const su2g::Struct& b) {
  if (a.nbond != b.nbond || a.locspin != b.locspin) return false;
  for (int l = 0; l < a.nbond; ++l)
    if (a.legs[l].dir != b.legs[l].dir || a.legs[l].angm != b.legs[l].angm || a.legs[l].dim != b.legs[l].dim)
      return false;
  return true;
}

// parses the operands; out gets their common structure with the union of blocks
int combine_struct(int n, const su2g_tensor* ops, std::vector<su2g::Struct>* in, su2g::Struct* out) {
  if (n <= 0 || !ops) return fail(SU2G_EINVAL, "operator_combine: no operands");
  in->assign(n, su2g::Struct());
  std::string e;
  for (int i = 0; i < n; ++i) {
    su2g::Struct& s = (*in)[i];
    if (!ops[i].desc || !s.parse(ops[i].desc, &e)) return fail(SU2G_EINVAL, "operator_combine: operand: " + e);
    s.set_layout(ops[i].flag);
    if (i > 0 && !same_legs(s, (*in)[0]))
      return fail(SU2G_EINVAL, "operator_combine: operands of different structures");
  }
  *out = (*in)[0];
  std::vector<int> u(out->nten, 0);
  for (const su2g::Struct& s : *in)
    for (int b = 0; b < s.nten; ++b) u[b] |= s.flag[b];
  out->set_layout(u.data());
  return SU2G_OK;
}

}  // namespace

namespace su2g {
cudaError_t launch_axpy_dev(double alpha, const double* scale, const double* x, double* y, int64_t n,
                            cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  const int blocks = (int)std::min<int64_t>((n + 255) / 256, 4 * 152);
  axpy_dev_kernel<<<blocks, 256, 0, stream>>>(alpha, scale, x, y, n);
  return cudaGetLastError();
}
}  // namespace su2g

extern "C" int su2g_operator_combine_layout(int n, const su2g_tensor* ops, int* out_flag, int out_flag_cap,
                                            int64_t* out_len) {
  std::vector<su2g::Struct> in;
  su2g::Struct out;
  int rc = combine_struct(n, ops, &in, &out);
  if (rc) return rc;
  if (!out_flag || out_flag_cap < out.nten) return fail(SU2G_EINVAL, "operator_combine_layout: flag array too small");
  std::copy(out.flag.begin(), out.flag.end(), out_flag);
  if (out_len) *out_len = out.total;
  return SU2G_OK;
}

extern "C" int su2g_operator_combine(int n, const su2g_tensor* ops, const double* coef, double* out, void* stream) {
  std::vector<su2g::Struct> in;
  su2g::Struct o;
  int rc = combine_struct(n, ops, &in, &o);
  if (rc) return rc;
  if (!coef || (o.total > 0 && !out)) return fail(SU2G_EINVAL, "operator_combine: null argument");
  // argument errors first, then the launches
  int64_t nblocks = 0;
  for (int b = 0; b < o.nten; ++b) {
    if (!o.flag[b]) continue;
    ++nblocks;
    for (int i = 0; i < n; ++i)
      if (in[i].flag[b] && !ops[i].data) return fail(SU2G_EINVAL, "operator_combine: missing operand data");
  }
  if (nblocks == 0) return SU2G_OK;
  if (nblocks > 65535) return fail(SU2G_EUNSUPPORTED, "operator_combine: more than 65535 blocks");
  cudaStream_t st = (cudaStream_t)stream;
  CombLauncher launcher(n, out, st);
  std::vector<CombSrc> srcs;
  for (int b = 0; b < o.nten;) {
    if (!o.flag[b]) {
      ++b;
      continue;
    }
    srcs.clear();
    for (int i = 0; i < n; ++i)
      if (in[i].flag[b]) srcs.push_back(CombSrc{ops[i].data + in[i].offset[b], coef[i]});
    int next = b;  // after the last block of the run
    int64_t end = o.offset[b];
    for (; next < o.nten; ++next) {
      bool same = true;
      for (int i = 0; i < n && same; ++i) same = !o.flag[next] || in[i].flag[next] == in[i].flag[b];
      if (!same) break;
      if (!o.flag[next]) continue;
      int64_t len = 1;
      for (int l = 0; l < o.nbond; ++l) len *= o.block_dim(next, l);
      end = o.offset[next] + len;
    }
    launcher.add(o.offset[b], end - o.offset[b], srcs);
    b = next;
  }
  cudaError_t e = launcher.finish();
  // the caller may drop the operands on return, whatever stream they belong to
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return fail(SU2G_ECUDA, std::string("operator_combine: ") + cudaGetErrorString(e));
  return SU2G_OK;
}
