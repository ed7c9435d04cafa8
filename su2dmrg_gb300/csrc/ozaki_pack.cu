// Splitting of FP64 operands into BF16 digit slices (layout in ozaki.hpp), in
// two launches: the row exponents (one warp per row), then the digits (one CTA
// per row tile and 32 k).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "kernels.hpp"
#include "overlap.cuh"
#include "ozaki.hpp"

namespace su2g {
namespace oz {
namespace {

constexpr int kPackThreads = 256;

// round(x 2^s) to the nearest integer, halves away from zero, with integer
// operations only.  The caller guarantees |x| 2^s < 2^48, so the mantissa is
// shifted right by at least five bits.
__device__ __forceinline__ long long scale_round(double x, int s) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  int E = (int)((b >> 52) & 0x7FF);
  unsigned long long M = b & 0xFFFFFFFFFFFFFull;
  if (E == 0) {
    if (M == 0) return 0;
    E = 1;  // subnormal
  } else {
    M |= 1ull << 52;
  }
  const int r = 1075 - E - s;  // |x| 2^s = M 2^-r
  unsigned long long q;
  if (r <= 0) {
    q = M << -r;  // excluded by the caller's bound; kept exact
  } else if (r > 63) {
    return 0;  // below 2^53 2^-64 < 1/2
  } else {
    q = ((M >> (r - 1)) + 1) >> 1;
  }
  return (b >> 63) ? -(long long)q : (long long)q;
}

// ilogb of a positive finite double given as its bit pattern
__device__ __forceinline__ int ilogb_bits(unsigned long long b) {
  const int E = (int)(b >> 52);
  if (E > 0) return E - 1023;
  return (63 - __clzll(b & 0xFFFFFFFFFFFFFull)) - 1074;
}

// sum_{q<S} 64 * 128^q: added to N it turns balanced digits into plain ones
template <int S>
constexpr long long kDigitBias = S == 0 ? 0 : 64ll + 128ll * kDigitBias<(S > 0 ? S - 1 : 0)>;
template <>
constexpr long long kDigitBias<0> = 0;

// |x| as a bit pattern.  The sign comes off the high word alone: masking the 64
// bits compiles to an FP64 |x|, sixteen clocks a warp.
__device__ __forceinline__ unsigned long long abs_bits(double x) {
  unsigned hi;
  asm("and.b32 %0, %1, 0x7FFFFFFF;" : "=r"(hi) : "r"(__double2hiint(x)));
  return ((unsigned long long)hi << 32) | (unsigned)__double2loint(x);
}

constexpr int kRowsPerUnit = kTM;  // row slots per unit in the row kernel (RT <= 128)
constexpr int kDigitKt = 2;        // k tiles (16 k each) per CTA of the digit kernel
constexpr int kOwnRowsKt = 4;      // up to this many, it finds the row exponents itself (launch_pack)

// Row exponents: one warp per row of every unit, lanes along k (coalesced):
// |alpha X| 2^-e < 1/2 with e = ilogb(max |alpha X|) + 2, kExpZero for a zero row.
__global__ void __launch_bounds__(kPackThreads) pack_rows_kernel(const PackJob* __restrict__ jobs,
                                                                 const int2* __restrict__ units, int nunits,
                                                                 Bases bases, int* exps, int* clear, int nclear) {
  dependents_may_start();
  const int64_t zero = wait_for_predecessor();
  for (int i = blockIdx.x * kPackThreads + threadIdx.x; i < nclear; i += gridDim.x * kPackThreads) clear[i] = 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t gw = (int64_t)blockIdx.x * (kPackThreads / 32) + warp;
  const int ui = (int)(gw / kRowsPerUnit), row = (int)(gw % kRowsPerUnit);
  if (ui >= nunits) return;
  const int2 u = units[ui];
  const PackJob& job = jobs[u.x];
  if (row >= job.rt || job.rowmax >= 0) return;  // row maxima left by the producing GEMM
  const int r = u.y * job.rt + row;
  unsigned long long m = 0;  // max |x| as a bit pattern (order-preserving for |x|)
  auto bits = [](double x) { return abs_bits(x); };
  if (r < job.R) {
    const double* p = after_wait(resolve(bases, job.src_buf, job.src), zero) + (int64_t)r * job.ld_r;
    int k = lane;
    for (; k + 96 < job.K; k += 128) {  // four loads in flight
      const double a = p[(int64_t)k * job.ld_k], b = p[(int64_t)(k + 32) * job.ld_k];
      const double c = p[(int64_t)(k + 64) * job.ld_k], d = p[(int64_t)(k + 96) * job.ld_k];
      m = max(m, max(max(bits(a), bits(b)), max(bits(c), bits(d))));
    }
    for (; k < job.K; k += 32) m = max(m, bits(p[(int64_t)k * job.ld_k]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) {
    int e = kExpZero;
    if (m != 0) {
      if (job.alpha == 1.0 || job.alpha == -1.0) {
        e = ilogb_bits(m) + 2;
      } else {
        const double mm = __longlong_as_double((long long)m) * fabs(job.alpha);
        if (mm > 0.0) e = ilogb(mm) + 2;
      }
    }
    exps[job.exp + r] = e;
  }
}

// Digits: one CTA per (unit, `span` times kDigitKt k tiles); a warp converts 8
// rows x 32 k at a time, a thread one row x 8 k into S 16-byte core rows, so
// that a warp's stores fill whole 256-byte core-row groups.  The k-chunk-0 CTA
// also records the row tile's largest exponent.
//
// Bound by instruction issue and, at size, nearly by HBM (8 bytes in, 2 S out an
// element).  Rows lie at 8-byte alignment: a warp loads 256 contiguous bytes of
// a row at a time, the next tile while it converts this one, and turns the tile
// through padded shared memory, so that each thread reads its 64 bytes by
// conflict-free 16-byte loads.  One FP64 multiply-add scales, rounds and biases
// an element, and a digit is one mask and one FFMA, where shifts, compares and
// masks of 64-bit integers took some 50 instructions an element.  The
// intermediates at D = 2000 (78 M elements, 7 slices): 321 us of 434, 5.3 TB/s
// or 0.79 of the copy rate; at D = 777 (7.9 M, 6 slices) 41 us of 65; the
// vector's own pack 43 of 60 and 22 of 30 us.  8-byte asynchronous copies
// instead of loads took 381 us, converting half the elements with integer
// instructions the same 321.
constexpr int kPitch = 34;                             // doubles a staged row takes (16-byte aligned, conflict-free)

// The S digits of eight elements given as mantissas 2^51 + N + bias (the low 52
// bits of lo, hi): a thread's 16-byte core row of every slice.  Balanced
// base-128 digits d_q in [-64, 63] (the leading one takes the rest): N + sum_q
// 64 * 128^q has the plain base-128 digits d_q + 64.  A digit's bits under the
// exponent of 2^23 are 2^23 + u 2^b for its place b in the word, and one FFMA
// makes that u - 64, exact, whose BF16 bits are the FP32 value's upper half.
template <int S>
__device__ __forceinline__ void store_digits(const uint32_t (&lo)[8], const uint32_t (&hi)[8], uint8_t* base,
                                             int64_t slice_bytes) {
#pragma unroll
  for (int q = 0; q < S; ++q) {
    constexpr int kTop = kBits * (S - 1);  // place of the leading digit
    const int place = kBits * (S - 1 - q);
    uint32_t fb[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float f;
      if (q == 0) {  // with the 2^51 above it: 2^(51 - kTop) + (N' >> kTop)
        const uint32_t u = (hi[i] >> (kTop - 32)) & ((1u << (52 - kTop)) - 1u);
        f = __uint_as_float(0x4B000000u | u) - (8388608.0f + (float)(1 << (51 - kTop)) + 64.0f);
      } else {
        const int word = place / 21;  // words start at bits 0 and 21
        const int b = place - 21 * word;
        const uint32_t w = word == 0 ? lo[i] : __funnelshift_r(lo[i], hi[i], 21);
        f = __fmaf_rn(__uint_as_float((w & (127u << b)) | 0x4B000000u), 1.0f / (float)(1 << b),
                      -(8388608.0f / (float)(1 << b) + 64.0f));
      }
      fb[i] = __float_as_uint(f);
    }
    uint4 v;
    v.x = __byte_perm(fb[0], fb[1], 0x7632);
    v.y = __byte_perm(fb[2], fb[3], 0x7632);
    v.z = __byte_perm(fb[4], fb[5], 0x7632);
    v.w = __byte_perm(fb[6], fb[7], 0x7632);
    *reinterpret_cast<uint4*>(base + q * slice_bytes) = v;
  }
}

// OwnRows: the row exponents are found here, by every CTA for all k of its rows,
// instead of by pack_rows_kernel before (no row maxima left by a GEMM then).
template <int S, bool OwnRows>
__global__ void __launch_bounds__(kPackThreads, 4) pack_digits_kernel(const PackJob* __restrict__ jobs,
                                                                   const int2* __restrict__ units, Bases bases,
                                                                   uint8_t* packed, int* exps_in, int span, int* clear,
                                                                   int nclear) {
  __shared__ int rexp[kTM];
  __shared__ int tmax;
  __shared__ unsigned long long rmax[OwnRows ? kTM : 1];
  __shared__ __align__(16) double stage[kPackThreads / 32][8 * kPitch];  // a tile a warp
  const int2 u = units[blockIdx.x];
  const PackJob job = jobs[u.x];
  const int kt0 = blockIdx.y * kDigitKt * span;
  dependents_may_start();
  const int64_t zero = wait_for_predecessor();
  if constexpr (OwnRows)
    for (int i = (blockIdx.y * gridDim.x + blockIdx.x) * kPackThreads + threadIdx.x; i < nclear;
         i += gridDim.x * gridDim.y * kPackThreads)
      clear[i] = 0;
  if (kt0 >= job.nkt) return;
  int* const exps = after_wait(exps_in, zero);
  const int rt = u.y, RT = job.rt, r0 = rt * RT;
  const double* src = after_wait(resolve(bases, job.src_buf, job.src), zero);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // a warp's tiles: the 8-row groups warp (and, for 128 rows, warp + 8) of every 32 k
  const int two = RT == kTM ? 1 : 0;
  const int ntiles = min(span, (job.nkt - kt0 + kDigitKt - 1) / kDigitKt) << two;
  double* const mine = stage[warp];
  const bool rows = job.ld_k == 1;  // contiguous rows: a row of 32 k an instruction; else 8 rows x 4 k
  const int tr = rows ? 0 : lane & 7, tk = rows ? lane : lane >> 3;  // this lane's element of a tile's first load,
  const int dr = rows ? 1 : 0, dk = rows ? 0 : 4;                    // and the step to the next
  const int64_t step = rows ? job.ld_r : 4 * job.ld_k;
  double next[8];
  auto group_of = [&](int i) { return warp + ((i & two) << 3); };
  auto fetch = [&](int i) {
    const int r = r0 + group_of(i) * 8, k = (kt0 + (i >> two) * kDigitKt) * kKS;
    const double* p = src + (int64_t)(r + tr) * job.ld_r + (int64_t)(k + tk) * job.ld_k;
    if (r + 8 <= job.R && k + kDigitKt * kKS <= job.K) {
#pragma unroll
      for (int j = 0; j < 8; ++j, p += step) next[j] = *p;
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j, p += step)
        next[j] = (r + tr + j * dr < job.R && k + tk + j * dk < job.K) ? *p : 0.0;
    }
  };
  if (ntiles > 0) fetch(0);
  if (tid == 0) tmax = kExpZero;
  if constexpr (OwnRows) {  // the unit's row maxima, over all k
    if (tid < kTM) rmax[tid] = 0;
    __syncthreads();
    if (rows) {  // a warp a row, four rows at a time
      for (int q = warp; q < RT; q += 4 * (kPackThreads / 32)) {
        unsigned long long m[4] = {0, 0, 0, 0};
        for (int k = lane; k < job.K; k += 32) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int r = r0 + q + j * (kPackThreads / 32);
            if (r < job.R) m[j] = max(m[j], abs_bits(src[(int64_t)r * job.ld_r + k]));
          }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
          for (int j = 0; j < 4; ++j) m[j] = max(m[j], __shfl_xor_sync(0xffffffffu, m[j], o));
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (lane == 0 && q + j * (kPackThreads / 32) < RT) rmax[q + j * (kPackThreads / 32)] = m[j];
      }
    } else {  // a lane a row, the warps share the k
      const int groups = RT / 32, r = (warp % groups) * 32 + lane, step_k = (kPackThreads / 32) / groups;
      unsigned long long m = 0;
      if (r0 + r < job.R) {
#pragma unroll 4
        for (int k = warp / groups; k < job.K; k += step_k)
          m = max(m, abs_bits(src[(int64_t)(r0 + r) * job.ld_r + (int64_t)k * job.ld_k]));
        atomicMax(&rmax[r], m);
      }
    }
  }
  __syncthreads();
  if (tid < RT) {
    int e;
    if constexpr (OwnRows) {
      e = rmax[tid] ? ilogb_bits(rmax[tid]) + 2 : kExpZero;
      if (blockIdx.y == 0) exps[job.exp + r0 + tid] = e;
    } else if (job.rowmax >= 0) {  // |X| 2^-e < 1/2 from the producer's ilogb maxima
      const int v = (r0 + tid < job.R) ? exps[job.rowmax + r0 + tid] : 0;
      e = v > 0 ? v - kRowmaxBias + 2 : kExpZero;
      if (blockIdx.y == 0) exps[job.exp + r0 + tid] = e;
    } else {
      e = exps[job.exp + r0 + tid];
    }
    rexp[tid] = e;
    if (blockIdx.y == 0 && e != kExpZero) atomicMax(&tmax, e);
  }
  __syncthreads();
  if (blockIdx.y == 0 && tid == 0) exps[job.texp + rt] = tmax;

  const bool unit_alpha = job.alpha == 1.0 || job.alpha == -1.0;
  const int64_t unit_bytes = (int64_t)S * RT * kKS * 2;
  const int64_t slice_bytes = (int64_t)RT * kKS * 2;
  uint8_t* dst = packed + job.dst + ((int64_t)rt * job.nkt + kt0) * unit_bytes;
  const int r8 = lane & 7, kc = lane >> 3;  // this thread's row of the group and core column
  const int kin = kc % (kKS / 8);
  constexpr double kMagic = 6755399441055744.0 + (double)kDigitBias<S>;  // 1.5 2^52 + bias
  double* const put = mine + tr * kPitch + tk;
  const int put_step = rows ? kPitch : 4;
  for (int i = 0; i < ntiles; ++i) {
    __syncwarp();  // the tile before has been read
#pragma unroll
    for (int j = 0; j < 8; ++j) put[j * put_step] = next[j];
    __syncwarp();
    if (i + 1 < ntiles) fetch(i + 1);
    const int rg = group_of(i);
    const int kt = (i >> two) * kDigitKt + kc / (kKS / 8);
    if (kt0 + kt >= job.nkt) continue;
    const int r = rg * 8 + r8;
    uint8_t* const out = dst + (int64_t)kt * unit_bytes + (r / 8) * kSBO + kin * 128 + (r % 8) * 16;
    if (r0 + rg * 8 >= job.R) {  // rows past the operand: zeros
#pragma unroll
      for (int q = 0; q < S; ++q) *reinterpret_cast<uint4*>(out + q * slice_bytes) = make_uint4(0, 0, 0, 0);
      continue;
    }
    const int e = rexp[r];
    const int sh = kBits * S - e;
    const double2* x2 = reinterpret_cast<const double2*>(mine + r8 * kPitch + kc * 8);
    double x[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const double2 t = x2[j];
      x[2 * j] = t.x;
      x[2 * j + 1] = t.y;
    }
    if (!unit_alpha) {
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] *= job.alpha;
    }
    uint32_t lo[8], hi[8];
    // 2^sh is a normal number, and e <= 1025 for finite rows; a zero row (e =
    // kExpZero) holds zeros
    if (e == kExpZero || (e <= 1025 && sh <= 1000)) {
      const int field = e == kExpZero ? 0 : sh + 1023;
      const double scale = __hiloint2double((field << 20) | (job.alpha == -1.0 ? (int)0x80000000u : 0), 0);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const double t = __fma_rn(x[j], scale, kMagic);
        lo[j] = (uint32_t)__double2loint(t);
        hi[j] = (uint32_t)__double2hiint(t);
      }
    } else {
#pragma unroll 1
      for (int o = 0; o < 8; ++o) {
        // the loop is not unrolled: this is rare, and its code would be eight times as long
        double xi = 0.0;
#pragma unroll
        for (int j = 0; j < 8; ++j) xi = j == o ? x[j] : xi;
        const long long n = scale_round(job.alpha == -1.0 ? -xi : xi, sh) + kDigitBias<S> + (1ll << 51);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          lo[j] = j == o ? (uint32_t)n : lo[j];
          hi[j] = j == o ? (uint32_t)((unsigned long long)n >> 32) : hi[j];
        }
      }
    }
    store_digits<S>(lo, hi, out, slice_bytes);
  }
}

// Partial tiles of a split output tile, summed in part order (deterministic).
// A thread sums one element, a warp 32 rows of one column, so the loads are
// coalesced and a tile spreads over kTM * kTN / 256 CTAs, four loads in
// flight a thread.  Bound by L2 latency.  One CTA per tile, 32 elements a
// thread one after the other, left most SMs idle: 63.5 us at D = 200 (6 terms,
// 7 slices), 77.8 us at D = 777 (11 terms, 6 slices) and 43.0 us at D = 2000
// (18 terms); spread out 8.2, 14.3 and 22.5 us.
constexpr int kRedThreads = 256;
__global__ void __launch_bounds__(kRedThreads) reduce_partials(const RedTile* __restrict__ reds, Bases bases) {
  const RedTile r = reds[blockIdx.x];
  dependents_may_start();
  const int64_t zero = wait_for_predecessor();
  const int idx = blockIdx.y * kRedThreads + threadIdx.x;
  const int i = idx % kTM, j = idx / kTM;
  if (i >= r.mlen || j >= r.nlen) return;
  const double* P = after_wait(resolve(bases, kBufScratch, r.part), zero) + idx;
  const int nparts = r.nparts;
  double s = 0.0;
  int p = 0;
  for (; p + 4 <= nparts; p += 4) {
    double v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = P[(int64_t)(p + q) * kTM * kTN];
#pragma unroll
    for (int q = 0; q < 4; ++q) s += v[q];
  }
  for (; p < nparts; ++p) s += P[(int64_t)p * kTM * kTN];
  resolve(bases, r.c_buf, r.c)[(int64_t)(r.m0 + i) + (int64_t)(r.n0 + j) * r.ldc] = s;
}

}  // namespace

cudaError_t launch_reduce(const RedTile* reds, int n, const Bases& bases, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  return launch_overlapped(reduce_partials, dim3(n, kTM * kTN / kRedThreads), kRedThreads, 0, 0, stream, reds, bases);
}

int pack_launches(bool rows_pass, bool unit_alpha, int max_nkt) {
  return rows_pass && !(unit_alpha && max_nkt <= kOwnRowsKt) ? 2 : 1;
}

cudaError_t launch_pack(int S, const PackJob* jobs, const int2* units, int nunits, int max_nkt, bool rows_pass,
                        const Bases& bases, uint8_t* packed, int* exps, cudaStream_t stream, bool unit_alpha, int* clear,
                        int nclear) {
  if (nclear > 0 && !(nunits > 0 && rows_pass)) {  // no kernel that does it
    const cudaError_t e = cudaMemsetAsync(clear, 0, nclear * sizeof(int), stream);
    if (e != cudaSuccess) return e;
    nclear = 0;
  }
  if (nunits <= 0) return cudaSuccess;
  // Operands of a scale +-1 without row maxima (psi) and of up to 64 k: the digit
  // kernel finds the exponents itself, one launch less (an application at D =
  // 100: 34.7 -> 31.3 us, at D = 200: 47.4 -> 45.5).  From 65 k on its CTAs, one for each
  // 32 k of a row tile, read the rows too often: D = 400, K <= 108, 100 -> 105 us;
  // D = 777, K <= 210, 239 -> 254.
  const bool own_rows = rows_pass && pack_launches(rows_pass, unit_alpha, max_nkt) == 1;
  if (rows_pass && !own_rows) {
    const int64_t warps = (int64_t)nunits * kRowsPerUnit;
    const int rows_blocks = (int)((warps + kPackThreads / 32 - 1) / (kPackThreads / 32));
    const cudaError_t e = launch_overlapped(pack_rows_kernel, dim3(rows_blocks), kPackThreads, 0, 0, stream, jobs,
                                            units, nunits, bases, exps, clear, nclear);
    if (e != cudaSuccess) return e;
    nclear = 0;
  }
  // CTAs of several chunks (exponents read once, tiles fetched ahead) once
  // there are enough to fill the SMs' slots twice over: 321 us at D = 2000
  // where CTAs of one chunk take 432, 41 at D = 777 where longer ones take 49
  const int chunks = (max_nkt + kDigitKt - 1) / kDigitKt;
  const int span = (int)std::min<int64_t>(std::max<int64_t>((int64_t)nunits * chunks / (8 * kF64Sms), 1), 8);
  const dim3 grid(nunits, (chunks + span - 1) / span);
  auto digits = [&](auto kernel) {
    return launch_overlapped(kernel, grid, kPackThreads, 0, 0, stream, jobs, units, bases, packed, exps, span, clear,
                             nclear);
  };
  if (S == 6) return own_rows ? digits(pack_digits_kernel<6, true>) : digits(pack_digits_kernel<6, false>);
  if (S == 7) return own_rows ? digits(pack_digits_kernel<7, true>) : digits(pack_digits_kernel<7, false>);
  return cudaErrorInvalidValue;
}

}  // namespace oz
}  // namespace su2g
