// Split-precision tile GEMM on the tcgen05 tensor cores (representation in
// ozaki.hpp).  A CTA computes 128 x 64 output tiles with four roles:
//
//   warp 16, lane 0 producer: bulk-copies the packed A (S slices x 128 x 16)
//                   and B (S slices x 64 x 16) units of each K stage into a
//                   kStages-deep shared-memory ring (cp.async.bulk + mbarrier
//                   transaction counts), running ahead of the MMAs;
//   warp 17, lane 0 MMA issuer: for every digit pair (p, q) with
//                   p + q <= S + 1, D[g = p+q] += A_p B_q^T (BF16 MMAs of
//                   K = 16), one FP32 TMEM accumulator of 128 lanes x 64
//                   columns per group g; frees each stage with a commit;
//   warp 18         bookkeeping: gathers each tile's reference exponents into
//                   shared memory while the drain warps work on the one before;
//   warps 0-15      epilogue: warp w reads TMEM lanes 32 (w % 4) .. + 31 (tile
//                   rows) and columns 16 (w / 4) .. + 15; after every K chunk
//                   of 560 (or segment end) it reads the S group sums of its
//                   16 columns (tcgen05.ld), the low groups first, converts
//                   them exactly to integers, weights them by 2^(48 - 7g) and
//                   adds them, aligned to the tile's largest product exponents,
//                   into 16 int64 accumulators per thread; at the end each
//                   thread scales its 16 values to FP64 and stores them.  Four
//                   warps per SM sub-partition hide the latency of these chains.
//
// What bounds it.  The MMAs of a stage take 910 clocks, and what is left
// between chunks is the drain of the low groups, about 1,200.  At D = 2000, 18
// terms, S = 7, the two launches of an application take 1247 + 1297 us (28 BF16
// products per FP64 product: 1540 TFLOP/s, 0.79 of the measured burst rate)
// and the GPU runs into its power limit (1350 W, clocks from 2070 to 2040 MHz).
// They took 1591 + 1691 us while the MMA thread waited and looked at the abort
// flag between stages, one drain of all groups stood between two chunks, and
// every tile's exponents, maxima and conversions were chains of global loads,
// named barriers and FP64 instructions.  At D = 777, 11 terms, the drain warps'
// work on short tiles still shows: 96 + 96 us (S = 7; 129 + 129 before).  Short
// tiles are not bound by the conversions' rate: FADDs instead of F2I wherever
// a short chunk's sums allow them changed nothing, and the added code lost 3%.
//
// Every mbarrier wait is bounded; on time-out the CTA records an error code
// in *err, drains its outstanding tensor-core work and bulk copies (bounded)
// and returns.
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>

#include "kernels.hpp"
#include "overlap.cuh"
#include "ozaki.hpp"

namespace su2g {
namespace oz {
namespace {

constexpr int kEpiWarps = 16;                      // drain warps: 4 lane quarters x 4 column slices
constexpr int kEpiThreads = kEpiWarps * 32;
constexpr int kCols = kTN / (kEpiWarps / 4);         // output columns per drain thread
constexpr int kProducerWarp = kEpiWarps, kMmaWarp = kEpiWarps + 1, kBookWarp = kEpiWarps + 2;
constexpr int kThreads = kEpiThreads + 96;           // + producer, MMA and bookkeeping warps
constexpr long long kWaitIters = 1ll << 24;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t a, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t a, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
               : "=r"(ok)
               : "r"(a), "r"(parity)
               : "memory");
  return ok != 0;
}

// bounded; gives up early once *abort is set (looked at only while it waits)
__device__ __forceinline__ bool mbar_wait(uint32_t a, uint32_t parity, volatile const int* abort = nullptr,
                                          long long limit = kWaitIters) {
  for (long long i = 0; i < limit; ++i) {
    if (mbar_try(a, parity)) return true;
    if (abort && (i & 63) == 63 && *abort) return false;
  }
  return false;
}

__device__ __forceinline__ bool mbar_test(uint32_t a, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
               : "=r"(ok)
               : "r"(a), "r"(parity)
               : "memory");
  return ok != 0;
}

__device__ __forceinline__ void mbar_arrive(uint32_t a) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(a) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t a, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a), "r"(bytes) : "memory");
}

__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t mbar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(mbar)
               : "memory");
}

// K-major, no swizzle: core matrices 8 rows x 16 B; LBO = 128 B between
// K-adjacent cores, SBO = kSBO = 256 B between 8-row groups (16 k per stage).
// The low word of a descriptor holds the address and the LBO (16-byte units;
// shared memory ends below 2^18, so additions stay inside the address field),
// the high word is the same for all.
__device__ __forceinline__ uint32_t smem_desc_lo(uint32_t addr) { return (addr >> 4) | ((uint32_t)(128 >> 4) << 16); }
constexpr uint32_t kDescHi = (uint32_t)(kSBO >> 4) | (1u << 14);

// kind::f16, BF16 x BF16 -> FP32, both K-major, M = 128, N = n
__host__ __device__ constexpr uint32_t idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTM >> 4) << 24);
}

__device__ __forceinline__ void mma(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t id, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 a, b;\n setp.ne.b32 p, %5, 0;\n mov.b64 a, {%1, %3};\n mov.b64 b, {%2, %3};\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, p;\n}\n" ::"r"(d_tmem),
      "r"(a_lo), "r"(b_lo), "r"(kDescHi), "r"(id), "r"(accumulate));
}

__device__ __forceinline__ void mma_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// An FP32 group sum is an integer below 2^24 in magnitude: the conversion is
// exact.  F2I runs at 16 a clock and SM (measured), so the groups that need
// less convert by one FADD instead: adding 1.5 2^(23+e) leaves round(G / 2^e)
// in the low mantissa bits.
__device__ __forceinline__ int f32_to_int_exact(uint32_t bits) { return __float2int_rn(__uint_as_float(bits)); }
template <int E>
__device__ __forceinline__ int f32_to_int_shift(uint32_t bits) {  // round(G 2^-E), |G| < 2^(22+E)
  constexpr float kMagic = 12582912.0f * (float)(1 << E);
  return __float_as_int(__uint_as_float(bits) + kMagic) - (0x4B400000 + (E << 23));
}

// Twice the weighted sum of one column's S group sums, v = sum_g G_g 2^(34 - 7g)
// (group g weighs 2^(kFixedTop - 7(g+2))), from their FP32 bit patterns in two
// parts: the three low groups lo[i] = G_{kHi + i} first (undoubled for 7 slices,
// whose low part then fits 32 bits), then the high ones hi[i] = G_i.
// |G_g| <= (g + 1) 560 65^2 <= 16,562,000 (the exactness bound of a chunk), so
// G_i * 128 + G_{i+1} is exact in int32, as is G_4 2^6 and what lies below, and
// few 64-bit shift-adds remain; |G_0| < 2^22.  The groups from 5 on weigh 1/2
// and 1/256 of the fixed point's unit.  Doubled, group 5 is a whole number:
// 6 slices keep all of it.  7 slices cut it to the unit (error below 1/2) and
// round group 6 to it (1/2), where cutting both left errors below 1/2 and 1.
template <int S>
struct Groups;
template <>
struct Groups<7> {
  static constexpr int kHi = 4;  // groups 0..3 high, 4..6 low
  using Low = int;
  __device__ static Low low(const uint32_t (&r)[3][4], int x) {
    return f32_to_int_exact(r[0][x]) * 64 + (f32_to_int_exact(r[1][x]) >> 1) + f32_to_int_shift<8>(r[2][x]);
  }
  __device__ static long long high(const uint32_t (&r)[kHi][4], int x, Low low) {
    const int Z = f32_to_int_shift<0>(r[0][x]) * 128 + f32_to_int_exact(r[1][x]);
    const int Y = f32_to_int_exact(r[2][x]) * 128 + f32_to_int_exact(r[3][x]);
    return ((long long)Z << 28) + ((long long)Y << 14) + (long long)low * 2;
  }
};
template <>
struct Groups<6> {
  static constexpr int kHi = 3;  // groups 0..2 high, 3..5 low
  using Low = long long;
  __device__ static Low low(const uint32_t (&r)[3][4], int x) {
    const int X = f32_to_int_exact(r[0][x]) * 128 + f32_to_int_exact(r[1][x]);
    return ((long long)X << 7) + f32_to_int_exact(r[2][x]);
  }
  __device__ static long long high(const uint32_t (&r)[kHi][4], int x, Low low) {
    const int Z = f32_to_int_shift<0>(r[0][x]) * 128 + f32_to_int_exact(r[1][x]);
    return ((long long)Z << 28) + ((long long)f32_to_int_exact(r[2][x]) << 21) + low;
  }
};

// ilogb of a subnormal double given as its words, -kRowmaxBias for a zero
__device__ __noinline__ int subnormal_ilogb(int hi, int lo) {
  const unsigned long long b = ((unsigned long long)((unsigned)hi & 0xFFFFFu) << 32) | (unsigned)lo;
  return b ? (63 - __clzll((long long)b)) - 1074 : -kRowmaxBias;
}

// v * 2^e rounded to nearest (ties to even); equal to ldexp((double)v, e)
// whenever the result is a normal number below 2^1023.  *odd: it is not (or
// may not be), and scaled_slow gives it.  Two ways to the same bits: integer
// instructions only, or the FP64 pipe's conversion (2 a clock and SM) and an
// addition to its exponent field.  A thread takes the second for fourteen of its
// sixteen columns: the integer chains of twenty-odd instructions cost more, in
// issue slots and in code, than the conversion's rate (by turns, the two
// launches at D = 2000 take 1272 + 1308 us, so 1247 + 1297; all sixteen 1245 + 1305).
__device__ __forceinline__ double scaled_by_int(long long v, int e, bool* odd) {
  const unsigned sign = (unsigned)(v >> 32) & 0x80000000u;
  const unsigned long long u = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
  unsigned hi = (unsigned)(u >> 32), lo = (unsigned)u;
  const bool wide = hi != 0;
  hi = wide ? hi : lo;
  lo = wide ? lo : 0u;
  const int lz = __clz((int)hi) & 31;
  hi = __funnelshift_l(lo, hi, lz);  // leading one at bit 31
  lo <<= lz;
  unsigned long long m = ((unsigned long long)(hi >> 11) << 32) | __funnelshift_r(lo, hi, 11);  // leading one at bit 52
  m += (lo & 0x7FFu) + ((unsigned)m & 1u) > 0x400u;
  const int biased = (wide ? 1086 : 1054) - lz + e;  // 63 - leading zeros + 1023 + e
  *odd = v != 0 && (unsigned)(biased - 1) >= 2045u;
  // the leading one (or the rounding's carry) adds itself to the exponent field
  m += (unsigned long long)(unsigned)(biased - 1) << 52;
  return v == 0 ? 0.0 : __hiloint2double((int)((unsigned)(m >> 32) | sign), (int)(unsigned)m);
}
__device__ __forceinline__ double scaled_by_fp64(long long v, int e, bool* odd) {
  const double d = __ll2double_rn(v);
  const int hi = __double2hiint(d);
  const int biased = ((hi >> 20) & 0x7FF) + e;
  *odd = v != 0 && (unsigned)(biased - 1) >= 2045u;
  return v == 0 ? 0.0 : __hiloint2double(hi + e * (1 << 20), __double2loint(d));
}
// a call, so that sixteen unrolled columns do not carry its code each
__device__ __noinline__ double scaled_slow(long long v, int e) { return ldexp((double)v, e); }

// What the drain warps need of a tile, gathered by the bookkeeping warp while
// they work on the tile before.
struct Book {
  OzTile t;
  int emax[kTM];           // reference exponents: rows,
  int fmax[kTN];           // columns,
  int cshift[kMaxSegs];    // and the part moved from rows to columns, per segment
};

template <int S>
struct Smem {
  static constexpr int kA = a_unit_bytes(S);
  static constexpr int kB = b_unit_bytes(S);
  static constexpr int kStage = kA + kB;
  static constexpr int kBytes = kStages * kStage + 1024;  // + alignment slack
};

// rowmax_out is the exponent buffer again: the kernel writes only its
// row-maximum region (OzWork::rowmax_base ..), which it never reads through exps.
//
// Persistent: CTA b computes tiles b, b + gridDim.x, ... (heaviest first, as
// the planner sorts them).  The producer runs ahead across tile boundaries,
// the MMAs of tile i+1 start as soon as the drain warps have read tile i's
// last chunk, and the conversion and stores of tile i overlap them.
template <int S>
__global__ void __launch_bounds__(kThreads, 1) ozaki_gemm(const OzTile* __restrict__ tiles, int ntiles,
                                                          const OzSeg* __restrict__ segs,
                                                          const uint8_t* packed_in, const int* exps_in,
                                                          int* rowmax_out, Bases bases, int* err) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  // accumulators full / empty, per half: [0] the low groups, [1] the high ones
  __shared__ __align__(8) uint64_t bar_full[kStages], bar_empty[kStages], bar_accf[2], bar_acce[2], bar_drain;
  __shared__ uint32_t tmem_base_sh;
  __shared__ __align__(8) uint64_t bar_bookf[2], bar_booke[2];
  __shared__ Book book_sh[2];
  __shared__ int shb_sh[kEpiWarps][kCols];  // per drain warp: column shifts of the current segment
  __shared__ int abort_sh, loaded_sh, consumed_sh;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(smem_u32(&bar_full[i]), 1);
      mbar_init(smem_u32(&bar_empty[i]), 1);
    }
    for (int h = 0; h < 2; ++h) {
      mbar_init(smem_u32(&bar_accf[h]), 1);
      mbar_init(smem_u32(&bar_acce[h]), kEpiWarps);
    }
    for (int h = 0; h < 2; ++h) {
      mbar_init(smem_u32(&bar_bookf[h]), 1);
      mbar_init(smem_u32(&bar_booke[h]), kEpiWarps);
    }
    mbar_init(smem_u32(&bar_drain), 1);
    abort_sh = 0;
    loaded_sh = 0;
    consumed_sh = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_sh;
  const int64_t zero = wait_for_predecessor();
  const uint8_t* const packed = after_wait(packed_in, zero);
  const int* const exps = after_wait(exps_in, zero);
  volatile int* abort_v = &abort_sh;
  auto stage_a = [&](int st) { return smem_u32(smem) + (uint32_t)(st * Smem<S>::kStage); };

  if (warp == kProducerWarp) {
    // ============================ producer ============================
    if (lane == 0) {
      int loaded = 0;
      bool ok = true;
      for (int ti = blockIdx.x; ti < ntiles && ok; ti += gridDim.x) {
        const OzTile t = tiles[ti];
        for (int s = 0; s < t.nseg && ok; ++s) {
          const OzSeg g = segs[t.seg0 + s];
          for (int ks = 0; ks < g.nks; ++ks, ++loaded) {
            const int st = loaded % kStages;
            // the stage's previous contents must have been consumed by their MMAs
            if (loaded >= kStages && !mbar_wait(smem_u32(&bar_empty[st]), ((loaded / kStages) - 1) & 1, abort_v)) {
              ok = false;
              break;
            }
            const uint32_t a_dst = stage_a(st), b_dst = a_dst + Smem<S>::kA;
            mbar_expect_tx(smem_u32(&bar_full[st]), Smem<S>::kStage);
            bulk_g2s(a_dst, packed + g.a_unit + (int64_t)ks * a_unit_bytes(S), Smem<S>::kA,
                     smem_u32(&bar_full[st]));
            bulk_g2s(b_dst, packed + g.b_unit + (int64_t)ks * b_unit_bytes(S), Smem<S>::kB,
                     smem_u32(&bar_full[st]));
          }
        }
      }
      if (!ok) {
        atomicExch(err, 1);
        atomicExch(&abort_sh, 1);
      }
      loaded_sh = loaded;
    }
  } else if (warp == kMmaWarp) {
    // =========================== MMA issuer ===========================
    if (lane == 0) {
      // The B digit slices lie back to back (64 rows each, same core-row
      // stride) and so do the group accumulators in TMEM (64 columns each):
      // the pairs (p, q) .. (p, q+n-1) are one MMA of N = 64 n that reads
      // B_q .. B_{q+n-1} as one 64n-row operand and adds into groups p+q-2 ..
      // p+q+n-3.  Up to n = 4 (N = 256): 10 MMAs per stage for S = 7 instead of
      // 28, 8 for S = 6.
      //
      // Issue.  The tensor pipe holds only the next MMA or two, so whatever
      // this thread does between two of them shows unless the ones before are
      // long.  A stage's MMAs go narrow first, wide last, and the barrier of
      // the next stage is looked at before the last two: 910 clocks a stage in
      // a loop of its own (S = 7; 896 at the N = 256 rate, an N = 64 MMA takes
      // 48 instead of 32), where p = 1, 2, .. in turn with a wait and a look at
      // the abort flag between stages takes 1172.
      //
      // Chunk boundaries.  The drain warps read a finished chunk's low groups
      // (index p + q - 2 >= kHi) first, then the high ones.  At a chunk's start
      // the pairs of the low groups run as soon as those are free, for up to
      // kStages stages, and the high pairs of these stages follow once the high
      // groups are: p = 1 touches every group of a half first, so only its MMA
      // starts a chunk's sums from zero.
      constexpr int kHi = Groups<S>::kHi;
      // A_p times slices q0 .. q1 of B, at the stage whose descriptors start at
      // d: two additions and the MMA.  The drain warps share this warp's
      // scheduler, and under their load descriptors built anew for each MMA
      // took 985 clocks a stage instead of 911.
      auto pairs_of = [&](uint32_t d, int p, int q0, int q1, bool zero) {
        mma(tmem + (uint32_t)((p + q0 - 2) * kTN), d + (uint32_t)((p - 1) * (kTM * kKS * 2) / 16),
            d + (uint32_t)((Smem<S>::kA + (q0 - 1) * (kTN * kKS * 2)) / 16), idesc(kTN * (q1 - q0 + 1)), zero ? 0u : 1u);
      };
      const uint32_t desc0 = smem_desc_lo(smem_u32(smem));
      const uint32_t full0 = smem_u32(&bar_full[0]), empty0 = smem_u32(&bar_empty[0]);
      auto desc_of = [&](int st) { return desc0 + (uint32_t)(st * (Smem<S>::kStage / 16)); };
      // the stage at hand (its slot, its barrier's parity), and whether that
      // barrier was seen full ahead of time
      int it = 0, slot = 0;
      uint32_t parity = 0;
      bool full = false;
      auto look_ahead = [&] {
        const bool wrap = slot == kStages - 1;
        full = mbar_test(wrap ? full0 : full0 + 8 * (slot + 1), wrap ? parity ^ 1u : parity);
      };
      auto stage_ready = [&] { return full || mbar_wait(full0 + 8 * slot, parity, abort_v); };
      auto next_stage = [&] {
        ++it;
        if (++slot == kStages) {
          slot = 0;
          parity ^= 1u;
        }
      };
      auto low_pairs = [&](uint32_t d, bool first) {
        if (first) pairs_of(d, 1, kHi + 1, S, true);
#pragma unroll
        for (int p = S; p >= 2; --p) {
          if (p == 2) look_ahead();
          pairs_of(d, p, p <= kHi ? kHi + 2 - p : 1, S + 1 - p, false);
        }
        if (!first) pairs_of(d, 1, kHi + 1, S, false);
      };
      auto high_pairs = [&](uint32_t d, bool first) {
        if (first) pairs_of(d, 1, 1, kHi, true);
#pragma unroll
        for (int p = kHi; p >= 2; --p) pairs_of(d, p, 1, kHi + 1 - p, false);
        if (!first) pairs_of(d, 1, 1, kHi, false);
      };
      auto all_pairs = [&](uint32_t d) {
        if constexpr (S == 7) {
          pairs_of(d, 7, 1, 1, false);
          pairs_of(d, 6, 1, 2, false);
          pairs_of(d, 3, 4, 5, false);
          pairs_of(d, 2, 5, 6, false);
          pairs_of(d, 5, 1, 3, false);
          pairs_of(d, 3, 1, 3, false);
          pairs_of(d, 1, 5, 7, false);
          pairs_of(d, 4, 1, 4, false);
          look_ahead();
          pairs_of(d, 2, 1, 4, false);
          pairs_of(d, 1, 1, 4, false);
        } else {
          pairs_of(d, 6, 1, 1, false);
          pairs_of(d, 5, 1, 2, false);
          pairs_of(d, 1, 5, 6, false);
          pairs_of(d, 2, 4, 5, false);
          pairs_of(d, 4, 1, 3, false);
          pairs_of(d, 2, 1, 3, false);
          look_ahead();
          pairs_of(d, 3, 1, 4, false);
          pairs_of(d, 1, 1, 4, false);
        }
      };
      bool ok = true;
      // the walk over tiles and segments, the next segment's length and the
      // next tile's segments read ahead
      int ti = blockIdx.x, s = 0;
      int seg0 = ti < ntiles ? tiles[ti].seg0 : 0, nseg = ti < ntiles ? tiles[ti].nseg : 0;
      int tn = ti + gridDim.x;
      int seg0_n = tn < ntiles ? tiles[tn].seg0 : 0, nseg_n = tn < ntiles ? tiles[tn].nseg : 0;
      auto settle = [&] {  // to the next segment there is, or ti >= ntiles
        while (s >= nseg && ti < ntiles) {
          ti = tn;
          seg0 = seg0_n;
          nseg = nseg_n;
          s = 0;
          tn += gridDim.x;
          seg0_n = tn < ntiles ? tiles[tn].seg0 : 0;
          nseg_n = tn < ntiles ? tiles[tn].nseg : 0;
        }
        return ti < ntiles ? segs[seg0 + s].nks : 0;
      };
      int nks = settle();
      uint32_t chunk = 0;
      while (nks > 0 && ok) {
        ++s;
        const int nks_n = settle();
        for (int k0 = 0; k0 < nks && ok; k0 += kChunkStages, ++chunk) {
          const int n = min(nks - k0, kChunkStages);
          const int slot0 = slot;
          const uint32_t low_free = smem_u32(&bar_acce[0]), high_free = smem_u32(&bar_acce[1]), before = (chunk - 1) & 1;
          // a new chunk overwrites the group sums: the epilogue must have read them
          if (chunk > 0 && !mbar_wait(low_free, before, abort_v)) {
            ok = false;
            break;
          }
          tc_fence_after();
          int i = 0;  // stages whose low pairs run
          for (bool go = false; !go;) {
            if (!stage_ready()) {
              ok = false;
              break;
            }
            low_pairs(desc_of(slot), i == 0);
            next_stage();
            ++i;
            if (i == n) mma_commit(smem_u32(&bar_accf[0]));
            go = chunk == 0 || mbar_test(high_free, before);
            if (!go && (i == n || i == kStages)) {
              go = mbar_wait(high_free, before, abort_v);
              if (!go) {
                ok = false;
                break;
              }
            }
          }
          if (!ok) break;
          tc_fence_after();
          for (int j = 0, sl = slot0; j < i; ++j) {  // their high pairs
            high_pairs(desc_of(sl), j == 0);
            mma_commit(empty0 + 8 * sl);
            if (++sl == kStages) sl = 0;
          }
          for (; i < n - 1; ++i) {
            if (!stage_ready()) {
              ok = false;
              break;
            }
            all_pairs(desc_of(slot));
            mma_commit(empty0 + 8 * slot);
            next_stage();
          }
          if (i < n && ok) {  // the last stage, its low pairs first
            if (!stage_ready()) {
              ok = false;
              break;
            }
            low_pairs(desc_of(slot), false);
            mma_commit(smem_u32(&bar_accf[0]));
            high_pairs(desc_of(slot), false);
            mma_commit(empty0 + 8 * slot);
            next_stage();
          }
          mma_commit(smem_u32(&bar_accf[1]));
        }
        nks = nks_n;
      }
      if (!ok) {
        atomicExch(err, 1);
        atomicExch(&abort_sh, 1);
      }
      consumed_sh = it;
      // drain: every MMA issued so far has completed once this commit arrives
      mma_commit(smem_u32(&bar_drain));
      if (!mbar_wait(smem_u32(&bar_drain), 0)) atomicExch(err, 2);
    }
  } else if (warp == kBookWarp) {
    // ========================== bookkeeping ===========================
    // Segment s contributes 2^(eA_s(i) + eB_s(j)) times its digit sums; moving
    // c_s = max_i eA_s(i) (over the tile rows) from the A side to the B side
    // leaves every product unchanged but makes the tile's reference exponents
    // emax(i) = max_s (eA_s(i) - c_s) and fmax(j) = max_s (eB_s(j) + c_s) track
    // the largest actual product scale (otherwise an O(1) x O(1e-3) segment and
    // an O(1e-3) x O(1) segment would set a reference 2^10 above both).  c_s =
    // the A row tile's largest exponent, recorded by the pack kernel.
    int n = 0;
    for (int ti = blockIdx.x; ti < ntiles; ti += gridDim.x, ++n) {
      Book& bk = book_sh[n & 1];
      if (n >= 2 && !mbar_wait(smem_u32(&bar_booke[n & 1]), ((n >> 1) - 1) & 1, abort_v)) {
        if (lane == 0) {
          atomicExch(err, 4);
          atomicExch(&abort_sh, 1);
        }
        break;
      }
      const int seg0 = tiles[ti].seg0, nseg = tiles[ti].nseg;
      if (lane == 0) bk.t = tiles[ti];
      for (int s = lane; s < nseg; s += 32) {
        const int m = exps[segs[seg0 + s].a_tmax];
        bk.cshift[s] = (m == kExpZero) ? 0 : m;
      }
      __syncwarp();
      int em[kTM / 32], fm[kTN / 32];
#pragma unroll
      for (int q = 0; q < kTM / 32; ++q) em[q] = kExpZero;
#pragma unroll
      for (int q = 0; q < kTN / 32; ++q) fm[q] = kExpZero;
#pragma unroll 4
      for (int s = 0; s < nseg; ++s) {
        const int* ea = exps + segs[seg0 + s].a_exp + lane;
        const int* eb = exps + segs[seg0 + s].b_exp + lane;
        const int cs = bk.cshift[s];
#pragma unroll
        for (int q = 0; q < kTM / 32; ++q) {
          const int e = ea[32 * q];
          if (e != kExpZero) em[q] = max(em[q], e - cs);
        }
#pragma unroll
        for (int q = 0; q < kTN / 32; ++q) {
          const int e = eb[32 * q];
          if (e != kExpZero) fm[q] = max(fm[q], e + cs);
        }
      }
#pragma unroll
      for (int q = 0; q < kTM / 32; ++q) bk.emax[lane + 32 * q] = em[q];
#pragma unroll
      for (int q = 0; q < kTN / 32; ++q) bk.fmax[lane + 32 * q] = fm[q];
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_bookf[n & 1]));
    }
    dependents_may_start();  // this CTA is at its last tiles
  } else {
    // ============================ epilogue ============================
    // The drain warps share nothing but the accumulators and the tiles' books:
    // each goes through its tiles at its own pace, no block-wide barrier.
    const int lq = warp & 3, col0 = (warp >> 2) * kCols;
    const int row = lq * 32 + lane;  // TMEM lane == tile row
    const uint32_t lane_base = (uint32_t)(lq * 32) << 16;
    int chunk = 0, n = 0;
    bool ok = true;
    for (int ti = blockIdx.x; ti < ntiles && ok; ti += gridDim.x, ++n) {
      const Book& bk = book_sh[n & 1];
      if (!mbar_wait(smem_u32(&bar_bookf[n & 1]), (n >> 1) & 1, abort_v)) {
        ok = false;
        break;
      }
      const int emax = bk.emax[row];
      const int nseg = bk.t.nseg;
      const OzSeg* sg = segs + bk.t.seg0;
      if (lq * 32 >= bk.t.mlen || col0 >= bk.t.nlen) {
        // Every row or column of this warp lies beyond the block's edge: it
        // only keeps the barriers' count (D = 200, where a tile is half full:
        // 18 + 18 -> 16 + 16 us).
        for (int s = 0; s < nseg && ok; ++s) {
          const int nchunks = (sg[s].nks + kChunkStages - 1) / kChunkStages;
          for (int c = 0; c < 2 * nchunks && ok; ++c) {
            ok = mbar_wait(smem_u32(&bar_accf[c & 1]), chunk & 1, abort_v);
            if (lane == 0 && ok) mbar_arrive(smem_u32(&bar_acce[c & 1]));
            chunk += c & 1;
          }
        }
        if (lane == 0 && ok) mbar_arrive(smem_u32(&bar_booke[n & 1]));
        continue;
      }
      long long acc[kCols];
#pragma unroll
      for (int j = 0; j < kCols; ++j) acc[j] = 0;
      // exponents of this lane's row and column, one segment ahead
      int ea = kExpZero, fj = kExpZero, nks = 0;
      if (nseg > 0) {
        ea = exps[sg[0].a_exp + row];
        fj = exps[sg[0].b_exp + col0 + (lane & (kCols - 1))];
        nks = sg[0].nks;
      }
      for (int s = 0; s < nseg && ok; ++s) {
        const int cs = bk.cshift[s];
        const int sha = (ea == kExpZero) ? 1000 : emax - (ea - cs);
        // column shifts of this segment, staged per warp
        __syncwarp();
        if (lane < kCols) shb_sh[warp][lane] = (fj == kExpZero) ? 1000 : bk.fmax[col0 + lane] - (fj + cs);
        __syncwarp();
        const int nchunks = (nks + kChunkStages - 1) / kChunkStages;
        if (s + 1 < nseg) {
          ea = exps[sg[s + 1].a_exp + row];
          fj = exps[sg[s + 1].b_exp + col0 + (lane & (kCols - 1))];
          nks = sg[s + 1].nks;
        }
        for (int c = 0; c < nchunks; ++c, ++chunk) {
          constexpr int kHi = Groups<S>::kHi;
          static_assert(S - kHi == 3, "three low groups");
          typename Groups<S>::Low low[kCols];
          if (!mbar_wait(smem_u32(&bar_accf[0]), chunk & 1, abort_v)) {
            ok = false;
            break;
          }
          tc_fence_after();
#pragma unroll
          for (int cb = 0; cb < kCols / 4; ++cb) {
            // the half's group sums of 4 columns in flight, one wait
            uint32_t r[3][4];
#pragma unroll
            for (int gg = 0; gg < 3; ++gg)
              tmem_ld4(tmem + lane_base + (uint32_t)((kHi + gg) * kTN + col0 + cb * 4), r[gg]);
            tmem_wait_ld();
#pragma unroll
            for (int x = 0; x < 4; ++x) low[cb * 4 + x] = Groups<S>::low(r, x);
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&bar_acce[0]));
          if (!mbar_wait(smem_u32(&bar_accf[1]), chunk & 1, abort_v)) {
            ok = false;
            break;
          }
          tc_fence_after();
#pragma unroll
          for (int cb = 0; cb < kCols / 4; ++cb) {
            uint32_t r[kHi][4];
#pragma unroll
            for (int gg = 0; gg < kHi; ++gg)
              tmem_ld4(tmem + lane_base + (uint32_t)(gg * kTN + col0 + cb * 4), r[gg]);
            tmem_wait_ld();
#pragma unroll
            for (int x = 0; x < 4; ++x) {
              const int j = cb * 4 + x;
              // round(v 2^-sh), halves up: one bit is left for the rounding, and
              // shifts of 63 and more leave nothing
              const long long v2 = Groups<S>::high(r, x, low[j]);
              acc[j] += ((v2 >> min(sha + shb_sh[warp][j], 63)) + 1) >> 1;
            }
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&bar_acce[1]));
        }
      }
      if (!ok) break;
      // ---- store: C = acc * 2^(emax + fmax - kFixedTop) ----
      // A phase-1 block that becomes a phase-2 operand also leaves, per
      // operand row (block columns i*rms ..), the largest ilogb of its values,
      // so that the pack needs no pass of its own over the block: over the
      // warp's rows here, then one global atomic per warp and column.
      const int ebase = emax - kFixedTop;
      double out[kCols];
      unsigned odd = 0;
#pragma unroll
      for (int jj = 0; jj < kCols; ++jj) {
        bool o;
        const int e = ebase + bk.fmax[col0 + jj];
        out[jj] = jj % 8 != 1 ? scaled_by_fp64(acc[jj], e, &o) : scaled_by_int(acc[jj], e, &o);
        odd |= o ? 1u << jj : 0u;
      }
      if (odd) {
#pragma unroll
        for (int jj = 0; jj < kCols; ++jj)
          if (odd >> jj & 1u) out[jj] = scaled_slow(acc[jj], ebase + bk.fmax[col0 + jj]);
      }
      const bool live = row < bk.t.mlen;
      const int nlen = bk.t.nlen - col0;
      if (bk.t.rowmax >= 0) {  // uniform over the CTA
        // kRowmaxBias-coded ilogb |value| of two columns a word, 0 for zeros and
        // absent values; then a butterfly that halves the words while it halves
        // the lanes
        unsigned w[kCols / 2];
#pragma unroll
        for (int i = 0; i < kCols / 2; ++i) {
          unsigned lg[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            // the high word only: masking the sign off the 64 bits compiles to
            // an FP64 |x|, sixteen clocks a warp (5,000 a tile)
            const int field = (__double2hiint(out[2 * i + h]) >> 20) & 0x7FF;
            lg[h] = field > 0 ? field - 1023 + kRowmaxBias : 0;
            if (odd && field == 0)  // zero or subnormal
              lg[h] = subnormal_ilogb(__double2hiint(out[2 * i + h]), __double2loint(out[2 * i + h])) + kRowmaxBias;
            if (!live || 2 * i + h >= nlen) lg[h] = 0;
          }
          w[i] = lg[0] | (lg[1] << 16);
        }
#pragma unroll
        for (int o = 16, k = kCols / 4; k >= 1; o >>= 1, k >>= 1) {
          const bool up = lane & o;
#pragma unroll
          for (int i = 0; i < k; ++i) {
            const unsigned other = __shfl_xor_sync(0xffffffffu, up ? w[i] : w[i + k], o);
            w[i] = __vmaxu2(up ? w[i + k] : w[i], other);
          }
        }
        w[0] = __vmaxu2(w[0], __shfl_xor_sync(0xffffffffu, w[0], 2));
        w[0] = __vmaxu2(w[0], __shfl_xor_sync(0xffffffffu, w[0], 1));
        static_assert(kCols == 16, "three halvings: lanes 4 i .. 4 i + 3 hold columns 2 i, 2 i + 1");
        const int jj = (lane >> 2) * 2 + (lane & 1);
        const int mine = (int)(lane & 1 ? w[0] >> 16 : w[0] & 0xFFFFu);
        if ((lane & 2) == 0 && mine > 0)
          atomicMax(&rowmax_out[bk.t.rowmax + (bk.t.n0 + col0 + jj) / bk.t.rms], mine);
      }
      if (live) {
        const int64_t ldc = bk.t.ldc;
        double* C = resolve(bases, bk.t.c_buf, bk.t.c) + (int64_t)(bk.t.m0 + row) + (int64_t)(bk.t.n0 + col0) * ldc;
#pragma unroll
        for (int jj = 0; jj < kCols; ++jj)
          if (jj < nlen) C[jj * ldc] = out[jj];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_booke[n & 1]));
    }
    if (!ok) {
      atomicExch(err, 3);
      atomicExch(&abort_sh, 1);
    }
  }
  tc_fence_before();
  __syncthreads();
  // bulk copies still in flight (possible only after an abort) must land
  // before the CTA exits: at most one unconsumed load per stage
  if (warp == kProducerWarp && lane == 0 && abort_sh)
    for (int i = consumed_sh; i < loaded_sh; ++i) mbar_wait(smem_u32(&bar_full[i % kStages]), (i / kStages) & 1);
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

}  // namespace

int gemm_smem_bytes(int S) {
  switch (S) {
    case 6: return Smem<6>::kBytes;
    case 7: return Smem<7>::kBytes;
    case 8: return Smem<8>::kBytes;
  }
  return 0;
}

namespace {
// The GEMM's bounded wait on an mbarrier that nothing arrives at: it must give
// up after `limit` polls and report it, leaving the context usable.
__global__ void bounded_wait_selftest_kernel(long long limit, int* timed_out) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&bar), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *timed_out = mbar_wait(smem_u32(&bar), 0, nullptr, limit) ? 0 : 1;
  }
}
}  // namespace

cudaError_t bounded_wait_selftest(long long limit, int* timed_out_host, cudaStream_t stream) {
  int* d = nullptr;
  cudaError_t e = cudaMallocAsync((void**)&d, sizeof(int), stream);
  if (e != cudaSuccess) return e;
  bounded_wait_selftest_kernel<<<1, 32, 0, stream>>>(limit, d);
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(timed_out_host, d, sizeof(int), cudaMemcpyDeviceToHost, stream);
  cudaFreeAsync(d, stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  return e;
}

namespace {
int g_sms = 0;            // one resident CTA per SM (shared memory and TMEM): a persistent grid
bool g_prepared[9] = {};  // per S
std::mutex g_prep_mu;
}  // namespace

int ozaki_persistent_grid() {
  static std::once_flag once;
  static int grid = 152;
  std::call_once(once, [] {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
        n > 0)
      grid = n;
    else
      cudaGetLastError();  // no device here: clear the error it left
  });
  return grid;
}

cudaError_t prepare_ozaki_gemm(int S) {
  if (S != 6 && S != 7) return cudaErrorInvalidValue;
  std::lock_guard<std::mutex> lock(g_prep_mu);
  if (g_prepared[S]) return cudaSuccess;
  int dev = 0, n = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  g_sms = n > 0 ? n : 148;
  const int smem = gemm_smem_bytes(S);
  e = S == 6 ? cudaFuncSetAttribute(ozaki_gemm<6>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)
             : cudaFuncSetAttribute(ozaki_gemm<7>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess) g_prepared[S] = true;
  return e;
}

cudaError_t launch_ozaki_gemm(int S, const OzTile* tiles, int ntiles, const OzSeg* segs, const uint8_t* packed,
                              int* exps, const Bases& bases, int* err, cudaStream_t stream) {
  if (ntiles <= 0) return cudaSuccess;
  cudaError_t e = prepare_ozaki_gemm(S);
  if (e != cudaSuccess) return e;
  const int grid = ntiles < g_sms ? ntiles : g_sms;
  const int smem = gemm_smem_bytes(S);
  return launch_overlapped(S == 6 ? ozaki_gemm<6> : ozaki_gemm<7>, dim3(grid), kThreads, smem, 0, stream, tiles, ntiles,
                           segs, packed, exps, exps, bases, err);
}

}  // namespace oz
}  // namespace su2g
