// Operator-API matmuls of the MX formats with f16 activations at prompt sizes (weights [N, K], K contiguous), on tcgen05.
//
//   y[m,n] = sum_k x[m,k] * s[n, k / group] * element[n,k]
//
// The weights are the 128-row operand of the MMA and go into it through TMEM: a converter thread owns one output column,
// reads its packed codes from shared memory and writes element * scale as f16 pairs into its own TMEM lane.  Nothing of a
// converted weight crosses shared memory, which with both operands in it is what bounds such a kernel (64 k of 128 columns x
// 192 rows move 64 KB there in 384 clocks of MMA; with converted weights stored and read back it would be 96 KB), and an MMA of
// few rows takes 17 clocks at 32 rows where one with both operands in shared memory takes 40.
//
// element * scale goes in exactly.  A significand has at most 6 bits; the power-of-two scales of a column are taken relative
// to the largest of 512 k (a unit), and f16 holds all bits of an element down to 2^-22 (mxfp8) or 2^-36 (mxfp4) of that scale.
// nvfp4's scale * element always fits.  One accumulator runs over a unit; promoters then add it, times the unit's scale, to f32
// registers, so that the tensor core's truncated additions stay short.  A group below that range that is not zero goes in
// as zeros, and its 32 k are added to the column's sums in f32, from global memory, before the result is rounded.
//
// Measured (mxfp8, f16, M = 512; before: a scale group of 32 k per accumulator, both operands in shared memory): four linears
// of 4096 / 14336 wide 857 -> 296 us; 4096 x 28672 462 -> 122 us, 0.60 of the measured bf16 rate; M = 17, 14336 x 4096 36.9 ->
// 17.8 us.  Bound by the converters where rows are few (a stage of 128 k takes 0.47 us, their instructions half of it); at 192 rows
// MMAs are 0.40 of a stage's 0.65 us at 1.9 GHz.  Groups below the range, mxfp8, M = 512, 14336 x 4096 (none: 63 us): one in every
// 128th column 68 us, in every 16th 71, in every column 157; 4096 x 28672 (122 us): 156, 178, 764.
//
// Persistent CTAs, one per SM.  Warps: TMA of activations, TMA of raw weights, the MMA issuer; two warpgroups of
// converters that take the 128-k stages in turn; two warpgroups of promoters, a thread of which holds up to 96 rows of a
// column in registers (setmaxnreg).  Two or more accumulators, so that neither a promotion nor the store of a tile stops the
// tensor core.  Where tiles are few, the CTAs of a cluster share one, each with a slice of K, and add their parts over
// distributed shared memory in a fixed order.
#include "mx_rings.h"
#include "opapi_convert.cuh"
#include "split_k.cuh"

namespace qmm {
namespace opg {
float cuda_core_us(int fmt, bool f32, int M, int N, int K);   // estimate of the CUDA-core kernels
}
namespace mxp {

using namespace opg;

constexpr int BN = 128;               // output columns per tile
constexpr int BK = kStageK;
constexpr int kRawBox = BN * 128;     // 16 KB of raw weights
constexpr int kUnitK = 512;           // k per accumulator, MX formats
constexpr int kInfo = 16;             // tiles whose columns may be marked
constexpr int kMaxRows = 192;
constexpr int kFirstConverter = 4, kFirstPromoter = kFirstConverter + 4 * kGroups, kThreads = (kFirstPromoter + 8) * 32;
constexpr int kLaunchRegs = 65536 / kThreads / 8 * 8;

template <int FMT, int CPT>   // CPT: rows of a tile (accumulator columns) per promoter thread, at most
struct Cfg {
  static constexpr int kBits = FMT == kMxfp8 ? 8 : 4;
  static constexpr bool kE8m0 = FMT == kMxfp4 || FMT == kMxfp8;
  static constexpr Rings kRings = rings(kBits, CPT);
  static_assert(sound(kRings), "waits by parity");
  static constexpr int kStagesPerBox = kRings.stages_per_box, kSlots = kRings.slots, kXStages = kRings.x_stages, kRawBoxes = kRings.raw_boxes;
  static constexpr int kRows = 2 * CPT;
  static constexpr int kXBytes = kRows * BK * 2;
  static constexpr int kAccBase = kSlots * (BK / 2);            // first TMEM column of the accumulators
  static constexpr int kAccBufs = (512 - kAccBase) / kRows;
  static constexpr int kOffRaw = kXStages * kXBytes;
  static constexpr int kOffInfo = kOffRaw + kRawBoxes * kRawBox;
  static constexpr int kOffS = kOffInfo + (kE8m0 ? kInfo * BN * 4 : 0);   // scales: two slots of 16 bytes per converter thread
  static constexpr int kOffBar = kOffS + kGroups * 2 * BN * 16;
  static constexpr int kSmem = kOffBar + 1024 + 1024;
  // scale that brings the largest element of a unit's largest scale just below f16's limit, and the smallest power of
  // two of a group's factor at which the last bit of an element is still there
  static constexpr int kUp = FMT == kMxfp8 ? 7 : 13, kLowest = FMT == kMxfp8 ? -15 : -23;
  static_assert(kAccBufs >= 2 && kSlots + kAccBufs + 3 <= kInfo, "ring sizes");
  // registers of a thread: producers and issuer, converters, promoters
  static constexpr int kMiscRegs = 40, kPromoterRegs = CPT == 96 ? 136 : 120, kConverterRegs = 216 - kPromoterRegs;
  static_assert(kMiscRegs <= kLaunchRegs && kConverterRegs <= kLaunchRegs && kPromoterRegs >= kLaunchRegs, "what shrinks and what grows");
  static_assert(128 * kMiscRegs + kGroups * 128 * kConverterRegs + 256 * kPromoterRegs <= kThreads * kLaunchRegs, "registers of the launch");
  static_assert(kRows * BN * 4 <= kOffInfo, "the result tile reuses the rings");
  static_assert((kUnitK / BK) % kGroups == 0 && kSmem <= 227 * 1024, "groups in a unit; shared memory");
};

struct Args {
  const void* x;
  const uint8_t* w;
  const void* scales;
  void* y;
  int M, N, K;
  int bm, mt, tiles;         // rows per tile, tiles along M, tiles in all
  int blocks, block_k;       // K in blocks of the slice granularity
  uint32_t idesc;
  int* status;
};

// A wait that usually finds its phase complete.
__device__ __forceinline__ bool wait_warp(uint64_t* bar, uint32_t parity, int* status, int tag) {
  if (__all_sync(0xFFFFFFFFu, dev::mbar_try_wait(bar, parity))) return true;
  return dev::mbar_wait_warp(bar, parity, status, tag);
}

// Scales come by asynchronous copies that their own thread waits for: a load into registers holds up, by the scoreboard that
// it shares, whatever the thread waits for next.
template <int BYTES>
__device__ __forceinline__ void copy_scales(void* dst, const uint8_t* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n\tcp.async.commit_group;" ::"r"(dev::smem_u32(dst)), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void wait_scales() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
// Up to 4 * WORDS scale bytes of a row that is not made of such pieces, 0 behind its end.
template <int WORDS>
__device__ __forceinline__ void load_scales(const uint8_t* row, int g0, int G, uint32_t (&r)[WORDS]) {
#pragma unroll
  for (int i = 0; i < WORDS; ++i) {
    r[i] = 0u;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (g0 + 4 * i + j < G) r[i] |= static_cast<uint32_t>(__ldg(row + g0 + 4 * i + j)) << (8 * j);
  }
}
// e8m0 scales of a column's unit
__device__ __forceinline__ uint4 unit_scales(const uint8_t* row, int g0, int G, bool vec) {
  if (vec) return __ldg(reinterpret_cast<const uint4*>(row + g0));
  uint32_t r[4];
  load_scales(row, g0, G, r);
  return make_uint4(r[0], r[1], r[2], r[3]);
}
// the largest of them, NaN codes (255) left out: one more than each, where 255 becomes 0
__device__ __forceinline__ int unit_largest(const uint4& s) {
  const uint32_t w[4] = {s.x, s.y, s.z, s.w};
  uint32_t m[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    m[i] = __vmaxu2(((w[i] & 0x00FF00FFu) + 0x00010001u) & 0x00FF00FFu, (((w[i] >> 8) & 0x00FF00FFu) + 0x00010001u) & 0x00FF00FFu);
  const uint32_t best = __vmaxu2(__vmaxu2(m[0], m[1]), __vmaxu2(m[2], m[3]));
  return max(static_cast<int>(max(best & 0xFFFFu, best >> 16)) - 1, 0);
}

// What the groups below the range of their unit, which go into the MMAs as zeros, contribute to column n, rows m0 .. m0 + 32 * TIMES
// - 1: v[t] of a lane, to row m0 + 32 t + lane.  The whole warp does a column: each lane looks for such groups among 16 scales, then
// takes its rows of each group, 32 k in f32.  Where such a group meets an activation that is not finite, the MMAs' zero times
// that is not what it should be: bit t of the result says that v[t] is the dot product over k_begin .. k_end itself.
template <int FMT, int TIMES>
__device__ __forceinline__ uint32_t small_groups(const __half* x, const uint8_t* w, const uint8_t* scales, int M, int K, int n, int m0,
                                                 int k_begin, int k_end, float (&v)[TIMES]) {
  using C = Cfg<FMT, 96>;
  const int lane = threadIdx.x & 31, G = K / 32, g_end = k_end / 32;
  const bool vec = G % 16 == 0 && (reinterpret_cast<uintptr_t>(scales) & 15) == 0;
  const uint8_t* srow = scales + static_cast<size_t>(n) * G;
  uint32_t lost = 0u;
#pragma unroll
  for (int t = 0; t < TIMES; ++t) v[t] = 0.f;
  for (int first = k_begin / 32; first < g_end; first += 32 * 16) {
    const int g0 = first + lane * 16;
    uint32_t mine = 0u;
    if (g0 < g_end) {
      const uint4 us = unit_scales(srow, g0, G, vec);
      const uint32_t word[4] = {us.x, us.y, us.z, us.w};
      const int ref = unit_largest(us);
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int code = (word[j / 4] >> (8 * (j % 4))) & 0xFF;
        if (g0 + j < g_end && code != 255 && C::kUp - (ref - code) < C::kLowest) mine |= 1u << j;
      }
    }
    for (uint32_t lanes = __ballot_sync(0xFFFFFFFFu, mine != 0u); lanes != 0u; lanes &= lanes - 1u) {
      const int from = __ffs(lanes) - 1;
      for (uint32_t groups = __shfl_sync(0xFFFFFFFFu, mine, from); groups != 0u; groups &= groups - 1u) {
        const int g = first + from * 16 + __ffs(groups) - 1;
        const uint4* codes = reinterpret_cast<const uint4*>(w + (static_cast<size_t>(n) * K + g * 32) / 8 * C::kBits);
        uint4 c[C::kBits / 4];
        uint32_t any = 0u;
#pragma unroll
        for (int i = 0; i < C::kBits / 4; ++i) {
          c[i] = __ldg(codes + i);
          any |= c[i].x | c[i].y | c[i].z | c[i].w;
        }
        if (!(any & (C::kBits == 4 ? 0x77777777u : 0x7F7F7F7Fu))) continue;
        const float scale = opapi::decode_e8m0(__ldg(srow + g));
        float sum[TIMES];
#pragma unroll
        for (int t = 0; t < TIMES; ++t) sum[t] = 0.f;
#pragma unroll
        for (int p = 0; p < 4; ++p) {   // 8 k
          uint4 xv[TIMES];
#pragma unroll
          for (int t = 0; t < TIMES; ++t)
            xv[t] = __ldg(reinterpret_cast<const uint4*>(x + static_cast<size_t>(min(m0 + 32 * t + lane, M - 1)) * K + g * 32) + p);
#pragma unroll
          for (int i = 0; i < 4; ++i) {   // 2 k
            const int bit = (p * 8 + i * 2) * C::kBits;
            const uint4& piece = c[bit / 128];
            const uint32_t words[4] = {piece.x, piece.y, piece.z, piece.w};
            const uint32_t two = words[bit / 32 % 4] >> (bit % 32);
            const float w0 = scale * (C::kBits == 8 ? opapi::decode_e4m3(two & 0xFFu) : opapi::kE2M1[two & 0xFu]);
            const float w1 = scale * (C::kBits == 8 ? opapi::decode_e4m3(two >> 8 & 0xFFu) : opapi::kE2M1[two >> 4 & 0xFu]);
#pragma unroll
            for (int t = 0; t < TIMES; ++t) {
              const uint32_t h[4] = {xv[t].x, xv[t].y, xv[t].z, xv[t].w};
              const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h[i]));
              sum[t] = fmaf(f.y, w1, fmaf(f.x, w0, sum[t]));
            }
          }
        }
#pragma unroll
        for (int t = 0; t < TIMES; ++t) {
          v[t] += sum[t];
          if (!(fabsf(sum[t]) < INFINITY)) lost |= 1u << t;   // finite activations cannot: the scale is far below the largest
        }
      }
    }
  }
#pragma unroll
  for (int t = 0; t < TIMES; ++t)
    if (lost >> t & 1u) v[t] = exact_dot_here<FMT, false>(x, w, scales, nullptr, K, 32, min(m0 + 32 * t + lane, M - 1), n, k_begin, k_end);
  return lost;
}
// For a warp's columns n0 .. n0 + 31, those of `columns`, whose sums are in TMEM (lane = column, `rows` rows from m0 on), and into y.
template <int FMT, int TIMES>
__device__ __noinline__ void add_small_groups(const __half* x, const uint8_t* w, const uint8_t* scales, __half* y, int M, int N, int K,
                                              uint32_t taddr, uint32_t columns, int n0, int m0, int rows) {
  const int lane = threadIdx.x & 31;
  for (uint32_t left = columns; left != 0u; left &= left - 1u) {
    const int owner = __ffs(left) - 1;
    float v[TIMES];
    const uint32_t lost = small_groups<FMT, TIMES>(x, w, scales, M, K, n0 + owner, m0, 0, K, v);
#pragma unroll
    for (int t = 0; t < TIMES; ++t) {
      const uint32_t replaced = __ballot_sync(0xFFFFFFFFu, lost >> t & 1u);
#pragma unroll 1
      for (int b = 0; b < 32 && 32 * t + b < rows; b += 8) {
        uint32_t r[8];
        dev::tmem_ld_32x8(taddr + 32 * t + b, r);
        dev::tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float sum = __shfl_sync(0xFFFFFFFFu, v[t], b + i);
          if (lane == owner) r[i] = __float_as_uint(replaced >> (b + i) & 1u ? sum : __uint_as_float(r[i]) + sum);
        }
        dev::tmem_st_32x8(taddr + 32 * t + b, r);
      }
    }
    dev::tc_wait_st();
  }
#pragma unroll 1
  for (int b = 0; b < rows; b += 8) {
    uint32_t r[8];
    dev::tmem_ld_32x8(taddr + b, r);
    dev::tc_wait_ld();
    if (columns >> lane & 1u) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (m0 + b + i < M) y[static_cast<size_t>(m0 + b + i) * N + n0 + lane] = __float2half_rn(__uint_as_float(r[i]));
    }
    __syncwarp();
  }
}
// The same for a slice of K whose sums are in shared memory, [row][BN columns].
template <int FMT, int TIMES>
__device__ __noinline__ void add_small_groups(const __half* x, const uint8_t* w, const uint8_t* scales, float* part, int M, int K,
                                              uint32_t columns, int n0, int m0, int rows, int k_begin, int k_end) {
  const int lane = threadIdx.x & 31;
  for (; columns != 0u; columns &= columns - 1u) {
    const int owner = __ffs(columns) - 1;
    float v[TIMES];
    const uint32_t lost = small_groups<FMT, TIMES>(x, w, scales, M, K, n0 + owner, m0, k_begin, k_end, v);
#pragma unroll
    for (int t = 0; t < TIMES; ++t) {
      float* at = part + (32 * t + lane) * BN + owner;
      if (32 * t + lane < rows) *at = lost >> t & 1u ? v[t] : *at + v[t];
    }
  }
}

template <int FMT, int CPT>
__global__ void __launch_bounds__(kThreads, 1)
mx_prefill_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap, const __grid_constant__ Args a) {
  using C = Cfg<FMT, CPT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint32_t* marks = reinterpret_cast<uint32_t*>(smem + C::kOffInfo);   // [kInfo][BN]: number of the tile that marked the column
  uint64_t* rfull = reinterpret_cast<uint64_t*>(smem + C::kOffBar);    // raw weights landed
  uint64_t* rempty = rfull + C::kRawBoxes;                                // and converted
  uint64_t* xfull = rempty + C::kRawBoxes;                                // activations landed
  uint64_t* full = xfull + C::kXStages;                                // half a stage ready for its MMAs
  uint64_t* consumed = full + 2 * C::kSlots;                                 // the MMAs of a stage retired
  uint64_t* dfull = consumed + kConsumed;                                  // a unit's accumulator complete
  uint64_t* dempty = dfull + C::kAccBufs;                              // and drained
  uint64_t* info = dempty + C::kAccBufs;                               // marks of a tile written
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(info + kInfo);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int KS = gridDim.x, rank = blockIdx.x;
  const int k_begin = static_cast<int>(static_cast<long long>(a.blocks) * rank / KS) * a.block_k;
  const int k_end = min(a.K, static_cast<int>(static_cast<long long>(a.blocks) * (rank + 1) / KS) * a.block_k);
  const int stages = (k_end - k_begin + BK - 1) / BK;
  const int boxes = (stages + C::kStagesPerBox - 1) / C::kStagesPerBox;
  const int units = (k_end - k_begin + kUnitK - 1) / kUnitK;

  if (warp == 0) {
    if (lane < C::kRawBoxes) { dev::mbar_init(&rfull[lane], 1); dev::mbar_init(&rempty[lane], C::kStagesPerBox * 4); }
    if (lane < C::kXStages) dev::mbar_init(&xfull[lane], 1);
    if (lane < kConsumed) dev::mbar_init(&consumed[lane], 1);
    if (lane < 2 * C::kSlots) dev::mbar_init(&full[lane], 4);
    if (lane < C::kAccBufs) { dev::mbar_init(&dfull[lane], 1); dev::mbar_init(&dempty[lane], 8); }
    if (lane < kInfo) dev::mbar_init(&info[lane], 4 * kGroups);
    dev::fence_mbar_init();
  } else if (warp == 2 && lane == 0) {
    dev::tma_prefetch_desc(&wmap);
    dev::tma_prefetch_desc(&xmap);
  } else if (warp >= kFirstConverter && C::kE8m0) {
    for (int i = threadIdx.x - kFirstConverter * 32; i < kInfo * BN; i += kThreads - kFirstConverter * 32) marks[i] = 0u;
  }
  if (warp == 3) {
    dev::tmem_alloc(tmem_slot, 512);
    dev::tmem_relinquish();
  }
  dev::tc_fence_before();
  __syncthreads();
  dev::tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
  dev::pdl_wait();
  dev::pdl_launch_dependents();

  float* tile_out = reinterpret_cast<float*>(smem);   // [bm][BN] partial results, once the rings are idle (KS > 1)

  if (warp < kFirstConverter) {
    dev::reg_dealloc<C::kMiscRegs>();
    if (warp == 0) {
      // ------------------------ TMA producer: activations --------------------
      if (lane == 0) {
        uint32_t cnt = 0;
        bool ok = true;
        for (int t = blockIdx.y; ok && t < a.tiles; t += gridDim.y) {
          const int m0 = (t % a.mt) * a.bm;
          for (int st = 0; st < stages; ++st, ++cnt) {
            const uint32_t s = cnt % C::kXStages;
            if (cnt >= C::kXStages) {
              const uint32_t p = cnt - C::kXStages;
              if (!dev::mbar_wait_relaxed(&consumed[p % kConsumed], (p / kConsumed) & 1, a.status, 111)) { ok = false; break; }
            }
            dev::mbar_expect_tx(&xfull[s], a.bm * BK * 2);
            dev::tma_load_2d(smem + s * C::kXBytes, &xmap, &xfull[s], k_begin + st * BK, m0);
            dev::tma_load_2d(smem + s * C::kXBytes + C::kXBytes / 2, &xmap, &xfull[s], k_begin + st * BK + 64, m0);
          }
        }
        // every copy has landed before this CTA's shared memory is reused, whatever the other warps did
        for (uint32_t i = cnt > C::kXStages ? cnt - C::kXStages : 0; i < cnt; ++i)
          if (!dev::mbar_wait_relaxed(&xfull[i % C::kXStages], (i / C::kXStages) & 1, a.status, 112)) break;
      }
    } else if (warp == 1) {
      // ------------------------ TMA producer: raw weights --------------------
      if (lane == 0) {
        uint32_t cnt = 0;
        bool ok = true;
        for (int t = blockIdx.y; ok && t < a.tiles; t += gridDim.y) {
          const int n0 = (t / a.mt) * BN;
          for (int b = 0; ok && b < boxes; ++b, ++cnt) {
            const uint32_t s = cnt % C::kRawBoxes;
            if (!dev::mbar_wait_relaxed(&rempty[s], ((cnt / C::kRawBoxes) & 1) ^ 1, a.status, 113)) { ok = false; break; }
            dev::mbar_expect_tx(&rfull[s], kRawBox);
            dev::tma_load_2d(smem + C::kOffRaw + s * kRawBox, &wmap, &rfull[s], k_begin / 8 * C::kBits + b * 128, n0);
          }
        }
        for (uint32_t i = cnt > C::kRawBoxes ? cnt - C::kRawBoxes : 0; i < cnt; ++i)
          if (!dev::mbar_wait_relaxed(&rfull[i % C::kRawBoxes], (i / C::kRawBoxes) & 1, a.status, 114)) break;
      }
    } else if (warp == 2) {
      // ------------------------------ MMA issuer -----------------------------
      if (dev::elect_one()) {
        constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);   // SBO, version, 128-byte swizzle
        const uint32_t x_lo = ((dev::smem_u32(smem) >> 4) & 0x3FFF) | ((16u >> 4) << 16);
        // What the thread executes between two MMAs queues behind the first: whether the next half stage is ready is asked
        // before the MMAs of this one, so that a wait is only made where there is something to wait for.
        uint32_t cnt = 0, xs = 0, buf = 0, bpar = 1;   // bpar: parity of the wait for the accumulator, flips with every round
        bool ok = true, ready = false;
        for (int t = blockIdx.y; ok && t < a.tiles; t += gridDim.y) {
          for (int st = 0; ok && st < stages; ++st, ++cnt) {
            const uint32_t s = cnt % C::kSlots, par = (cnt / C::kSlots) & 1;
            const uint32_t at = tmem_base + s * (BK / 2), b_lo = x_lo + xs * (C::kXBytes >> 4);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              if (!ready && !dev::mbar_wait(&full[2 * s + h], par, a.status, 115)) { ok = false; break; }
              if (h == 0) ready = dev::mbar_test(&full[2 * s + 1], par);
              else ready = dev::mbar_test(&full[2 * ((cnt + 1) % C::kSlots)], ((cnt + 1) / C::kSlots) & 1);
              // a step of 16 k: 8 columns of TMEM, 32 bytes of a row; 64 k of activations are one swizzled tile
              auto step = [&](uint32_t d, int j, uint32_t accumulate) {
                dev::umma_f16_ts(d, at + h * 32 + j * 8, b_lo + h * (C::kXBytes >> 5) + j * 2, kDescHi, a.idesc, accumulate);
              };
              {
                const bool first = st % (kUnitK / BK) == 0 && h == 0;
                if (first && !dev::mbar_wait(&dempty[buf], bpar, a.status, 116)) { ok = false; break; }
                dev::tc_fence_after();
                const uint32_t d = tmem_base + C::kAccBase + buf * C::kRows;
#pragma unroll
                for (int j = 0; j < 4; ++j) step(d, j, !first || j != 0);
                if (h == 1 && (st % (kUnitK / BK) == kUnitK / BK - 1 || st == stages - 1)) {
                  dev::tc_commit(&dfull[buf]);
                  if (++buf == C::kAccBufs) { buf = 0; bpar ^= 1; }
                }
              }
              if (!ok) break;
            }
            if (ok) dev::tc_commit(&consumed[cnt % kConsumed]);
            if (++xs == C::kXStages) xs = 0;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp < kFirstPromoter) {
    // ------------------------------ converters -----------------------------
    dev::reg_dealloc<C::kConverterRegs>();
    const int grp = (warp - kFirstConverter) >> 2, ww = warp & 3;
    const int row = ww * 32 + lane;
    const uint32_t a_lane = tmem_base + (static_cast<uint32_t>(ww * 32) << 16);
    uint32_t cnt0 = 0, box0 = 0, tile_no = 0;
    bool ok = true;
    constexpr int kPieceBytes = C::kE8m0 ? 16 : 8;
    const int G = C::kE8m0 ? a.K / 32 : a.K / 16;
    const bool vec = G % kPieceBytes == 0 && (reinterpret_cast<uintptr_t>(a.scales) & (kPieceBytes - 1)) == 0;
    uint8_t* slots = smem + C::kOffS + (grp * 2 * BN + row) * 16;
    int slot = 0;
    auto ask = [&](const uint8_t* scales_row, int k) {
      if (vec) copy_scales<kPieceBytes>(slots + slot * BN * 16, scales_row + k / (C::kE8m0 ? 32 : 16));
    };
    auto row_of = [&](int tile) {
      return static_cast<const uint8_t*>(a.scales) + static_cast<size_t>(min((tile / a.mt) * BN + row, a.N - 1)) * G;
    };
    // first stage of the group's in the tile whose first stage is number `cnt`
    auto first_stage = [&](uint32_t cnt) { return static_cast<int>((grp + kGroups - cnt % kGroups) % kGroups); };
    // the group's first scales in a tile: none where it has no stage there
    auto ask_tile = [&](int tile, uint32_t cnt) {
      if (tile < a.tiles && first_stage(cnt) < stages) ask(row_of(tile), k_begin + (C::kE8m0 ? 0 : first_stage(cnt) * BK));
    };
    ask_tile(blockIdx.y, 0);
    for (int t = blockIdx.y; ok && t < a.tiles; t += gridDim.y, cnt0 += stages, box0 += boxes, ++tile_no) {
      // MX: the scales of a unit (16 bytes), nvfp4: of a stage (8 bytes); the next ones are on their way to the other slot
      const uint8_t* srow = row_of(t);
      uint4 us = make_uint4(0u, 0u, 0u, 0u);
      int ref = 0, unit = -1;
      // The groups take the stages of all tiles in turn.  What their waits by parity rely on: mx_rings.h.
      const int first = first_stage(cnt0);
      if (first >= stages) ask_tile(t + gridDim.y, cnt0 + stages);
      for (int st = first; st < stages; st += kGroups) {
        const uint32_t c = cnt0 + st, s = c % C::kSlots, xs = c % C::kXStages;
        const uint32_t box = box0 + st / C::kStagesPerBox, rs = box % C::kRawBoxes;
        const int sub = st % C::kStagesPerBox;
        if (!C::kE8m0 || st / (kUnitK / BK) != unit) {
          unit = st / (kUnitK / BK);
          const int k0 = k_begin + (C::kE8m0 ? unit * kUnitK : st * BK);
          if (vec) {
            wait_scales();
            if (C::kE8m0) us = *reinterpret_cast<const uint4*>(slots + slot * BN * 16);
            else *reinterpret_cast<uint2*>(&us) = *reinterpret_cast<const uint2*>(slots + slot * BN * 16);
            slot ^= 1;
            const int next_stage = C::kE8m0 ? (unit + 1) * (kUnitK / BK) : st + kGroups;
            if (next_stage + (C::kE8m0 ? first : 0) < stages) ask(srow, k_begin + next_stage * BK);
            else ask_tile(t + gridDim.y, cnt0 + stages);
          } else if (C::kE8m0) {
            us = unit_scales(srow, k0 / 32, G, false);
          } else {
            uint32_t r[2];
            load_scales(srow, k0 / 16, G, r);
            us.x = r[0];
            us.y = r[1];
          }
          if (C::kE8m0) ref = unit_largest(us);
        }
        if (!wait_warp(&rfull[rs], (box / C::kRawBoxes) & 1, a.status, 117)) { ok = false; break; }
        const uint8_t* raw = smem + C::kOffRaw + rs * kRawBox + row * 128;
        constexpr int kPieces = C::kBits / 4;   // 16-byte pieces of a column's 32 k
        // 64 k of the column -> 32 pairs.  The second half is converted while the first one is multiplied.
        auto convert = [&](int half, uint32_t (&o)[32]) {
#pragma unroll
          for (int g = 0; g < 2; ++g) {   // 32 k
            const int h = half * 2 + g;
            uint4 v[kPieces];
#pragma unroll
            for (int i = 0; i < kPieces; ++i)
              v[i] = *reinterpret_cast<const uint4*>(raw + ((((sub * 4 + h) * kPieces + i) ^ (row & 7)) << 4));
            uint32_t f0 = 0u, f1 = 0u;    // factors of its two halves
            if (C::kE8m0) {
              const int quad = st % (kUnitK / BK);
              const uint32_t word = quad < 2 ? (quad == 0 ? us.x : us.y) : (quad == 2 ? us.z : us.w);
              const int code = (word >> (8 * h)) & 0xFF;
              const int e = C::kUp - (ref - code);
              __half2 f = __float2half2_rn(e < C::kLowest ? 0.f : __uint_as_float(static_cast<uint32_t>(127 + e) << 23));
              f0 = f1 = code == 255 ? 0x7E007E00u : *reinterpret_cast<uint32_t*>(&f);
              if (e < C::kLowest) {
                uint32_t any = 0u;
#pragma unroll
                for (int i = 0; i < kPieces; ++i) any |= v[i].x | v[i].y | v[i].z | v[i].w;
                if (any & (C::kBits == 4 ? 0x77777777u : 0x7F7F7F7Fu)) marks[(tile_no % kInfo) * BN + row] = tile_no + 1;
              }
            } else if (FMT == kNvfp4) {
              const uint32_t word = h < 2 ? us.x : us.y;
              f0 = e4m3_pair<false>((word >> (16 * (h & 1))) & 0xFFu);
              f1 = e4m3_pair<false>((word >> (16 * (h & 1) + 8)) & 0xFFu);
            }
            if (C::kBits == 4) {
              const uint32_t in[4] = {v[0].x, v[0].y, v[0].z, v[0].w};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const uint4 r = convert8<FMT, false>(in[i], 0u, i < 2 ? f0 : f1, false);
                o[16 * g + 4 * i] = r.x; o[16 * g + 4 * i + 1] = r.y; o[16 * g + 4 * i + 2] = r.z; o[16 * g + 4 * i + 3] = r.w;
              }
            } else {
#pragma unroll
              for (int i = 0; i < kPieces; ++i) {
                const uint4 r = convert8<FMT, false>(v[i].x, v[i].y, 0u, false), u = convert8<FMT, false>(v[i].z, v[i].w, 0u, false);
                o[16 * g + 8 * i] = r.x; o[16 * g + 8 * i + 1] = r.y; o[16 * g + 8 * i + 2] = r.z; o[16 * g + 8 * i + 3] = r.w;
                o[16 * g + 8 * i + 4] = u.x; o[16 * g + 8 * i + 5] = u.y; o[16 * g + 8 * i + 6] = u.z; o[16 * g + 8 * i + 7] = u.w;
              }
            }
            if (C::kE8m0) {
#pragma unroll
              for (int i = 0; i < 16; ++i) o[16 * g + i] = mul2<false>(o[16 * g + i], f0);
            }
          }
        };
        uint32_t o[32];
        convert(0, o);
        if (c >= C::kSlots) {   // the MMAs that read this slot's TMEM before have retired
          const uint32_t p = c - C::kSlots;
          if (!wait_warp(&consumed[p % kConsumed], (p / kConsumed) & 1, a.status, 118)) { ok = false; break; }
          dev::tc_fence_after();
        }
        dev::tmem_st_32x32(a_lane + s * (BK / 2), o);
        if (!wait_warp(&xfull[xs], (c / C::kXStages) & 1, a.status, 119)) { ok = false; break; }
        dev::tc_wait_st();
        dev::tc_fence_before();
        __syncwarp();
        if (lane == 0) dev::mbar_arrive(&full[2 * s]);
        convert(1, o);
        dev::tmem_st_32x32(a_lane + s * (BK / 2) + 32, o);
        dev::tc_wait_st();
        dev::tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          dev::mbar_arrive(&full[2 * s + 1]);
          dev::mbar_arrive(&rempty[rs]);
        }
      }
      // a last box that is not full: what its other stages would have handed back
      if (ok) {
        const int missing = boxes * C::kStagesPerBox - stages;
        __syncwarp();
        if (lane == 0) {
          if ((cnt0 + stages - 1) % kGroups == grp)
            for (int i = 0; i < missing; ++i) dev::mbar_arrive(&rempty[(box0 + boxes - 1) % C::kRawBoxes]);
          if (C::kE8m0) dev::mbar_arrive(&info[tile_no % kInfo]);
        }
      }
    }
  } else {
    // ------------------------------ promoters ------------------------------
    dev::reg_alloc<C::kPromoterRegs>();
    const int q = warp & 3, part = (warp - kFirstPromoter) >> 2;
    const int hc = a.bm / 2, c0 = part * hc;   // this thread's rows of the tile: c0 .. c0 + hc - 1
    const uint32_t d_lane = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + C::kAccBase + c0;
    uint32_t buf = 0, bpar = 0, tile_no = 0;
    bool ok = true;
    uint64_t acc[CPT / 2];
    for (int t = blockIdx.y; ok && t < a.tiles; t += gridDim.y, ++tile_no) {
      const int m0 = (t % a.mt) * a.bm, n = (t / a.mt) * BN + q * 32 + lane, nc = min(n, a.N - 1);
#pragma unroll
      for (int i = 0; i < CPT / 2; ++i) acc[i] = 0ull;
      const int G = C::kE8m0 ? a.K / 32 : 0;
      const uint8_t* srow = static_cast<const uint8_t*>(a.scales) + static_cast<size_t>(nc) * G;
      const bool vec = C::kE8m0 && G % 16 == 0 && (reinterpret_cast<uintptr_t>(a.scales) & 15) == 0;
      for (int u = 0; u < units; ++u) {
        float s = 1.f;
        if (C::kE8m0) {
          const int ref = unit_largest(unit_scales(srow, (k_begin + u * kUnitK) / 32, G, vec));
          s = opapi::decode_e8m0(ref) * __uint_as_float(static_cast<uint32_t>(127 - C::kUp) << 23);
        }
        if (!wait_warp(&dfull[buf], bpar, a.status, 121)) { ok = false; break; }
        dev::tc_fence_after();
        const uint64_t s2 = pack2(s, s);
        const uint32_t taddr = d_lane + buf * C::kRows;
        constexpr int kLd = CPT == 96 ? 16 : 32;   // values in flight beside the sums, as registers allow
#pragma unroll
        for (int c = 0; c < CPT; c += kLd) {
          if (c < hc) {
            uint32_t r[kLd];
            if constexpr (kLd == 16) dev::tmem_ld_32x16(taddr + c, r);
            else dev::tmem_ld_32x32(taddr + c, r);
            dev::tc_wait_ld();
            if (c + kLd >= hc) {   // the last values are in registers: the buffer goes back
              dev::tc_fence_before();
              __syncwarp();
              if (lane == 0 && (!C::kE8m0 || u < units - 1)) dev::mbar_arrive(&dempty[buf]);
            }
#pragma unroll
            for (int e = 0; e < kLd / 2; ++e)
              fma2(acc[c / 2 + e], s2, pack2(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1])));
          }
        }
        if (++buf == C::kAccBufs) { buf = 0; bpar ^= 1; }
      }
      if (!ok) break;
      // The last accumulator goes back when it is clear that no column misses groups; else it takes the tile's sums, behind the
      // stores (before them: M = 384, 4096 x 28672 7 % slower without such columns).
      [[maybe_unused]] uint32_t marked = 0u;
      [[maybe_unused]] const uint32_t last = buf == 0 ? C::kAccBufs - 1 : buf - 1;
      if constexpr (C::kE8m0) {
        if (!dev::mbar_wait_warp(&info[tile_no % kInfo], (tile_no / kInfo) & 1, a.status, 122)) { ok = false; break; }
        marked = __ballot_sync(0xFFFFFFFFu, marks[(tile_no % kInfo) * BN + q * 32 + lane] == tile_no + 1);
        if (marked == 0u) {
          if (lane == 0) dev::mbar_arrive(&dempty[last]);
        }
      }
      if (KS > 1) break;   // one tile per cluster: it is put together below
      // ---- results: two rows at a time, neighbouring lanes exchange so that each stores two columns of one row
      __half* y = static_cast<__half*>(a.y);
      const bool pairs = (a.N & 1) == 0;
#pragma unroll
      for (int i = 0; i < CPT / 2; ++i) {
        if (2 * i < hc && m0 + c0 + 2 * i < a.M) {
          float v0, v1;
          unpack2(acc[i], v0, v1);
          const int m = m0 + c0 + 2 * i;
          if (pairs) {
            const float got = __shfl_xor_sync(0xFFFFFFFFu, (lane & 1) ? v0 : v1, 1);
            const __half2 p = (lane & 1) ? __floats2half2_rn(got, v1) : __floats2half2_rn(v0, got);
            const int mm = m + (lane & 1);
            if (mm < a.M && n < a.N) *reinterpret_cast<__half2*>(y + static_cast<size_t>(mm) * a.N + (n & ~1)) = p;
          } else if (n < a.N) {
            y[static_cast<size_t>(m) * a.N + n] = __float2half_rn(v0);
            if (m + 1 < a.M) y[static_cast<size_t>(m + 1) * a.N + n] = __float2half_rn(v1);
          }
        }
      }
      if constexpr (C::kE8m0) {
        if (marked != 0u) {
#pragma unroll
          for (int c = 0; c < CPT; c += 8) {
            if (c < hc) {
              uint32_t r[8];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                float v0, v1;
                unpack2(acc[c / 2 + i], v0, v1);
                r[2 * i] = __float_as_uint(v0);
                r[2 * i + 1] = __float_as_uint(v1);
              }
              dev::tmem_st_32x8(d_lane + last * C::kRows + c, r);
            }
          }
          dev::tc_wait_st();
          __syncwarp();   // a neighbour has stored half of the column
          add_small_groups<FMT, CPT / 32>(static_cast<const __half*>(a.x), a.w, static_cast<const uint8_t*>(a.scales), y, a.M, a.N, a.K,
                                          d_lane + last * C::kRows, marked, (t / a.mt) * BN + q * 32, m0 + c0, hc);
          dev::tc_fence_before();
          __syncwarp();
          if (lane == 0) dev::mbar_arrive(&dempty[last]);
          // not live across the call, around which they would be spilled (40 to 470 bytes, in the loop too: 4096 x 28672, M = 100
          // 46.8 us without any such column, 41.8 so)
#pragma unroll
          for (int i = 0; i < CPT / 2; ++i) acc[i] = 0ull;
        }
      }
    }
    dev::tc_fence_before();
    __syncthreads();   // every warp is done with the rings and with TMEM
    if (KS == 1) return;
    // ---- this slice's results, [row][column], into the idle rings; the cluster's CTAs add up a share of the rows each
#pragma unroll
    for (int i = 0; i < CPT / 2; ++i) {
      if (2 * i < hc) {
        float v0, v1;
        unpack2(acc[i], v0, v1);
        tile_out[(c0 + 2 * i) * BN + q * 32 + lane] = v0;
        tile_out[(c0 + 2 * i + 1) * BN + q * 32 + lane] = v1;
      }
    }
    const int m0 = (blockIdx.y % a.mt) * a.bm, n0 = (blockIdx.y / a.mt) * BN;
    if constexpr (C::kE8m0) {
      const uint32_t marked = __ballot_sync(0xFFFFFFFFu, ok && marks[q * 32 + lane] == 1u);
      __syncwarp();
      if (marked != 0u)
        add_small_groups<FMT, CPT / 32>(static_cast<const __half*>(a.x), a.w, static_cast<const uint8_t*>(a.scales), tile_out + c0 * BN + q * 32,
                                        a.M, a.K, marked, n0 + q * 32, m0 + c0, hc, k_begin, k_end);
    }
    split::cluster_sync();
    const int rows = min(a.bm, a.M - m0);
    const bool pairs = (a.N & 1) == 0;
    constexpr int kAdders = kThreads - kFirstPromoter * 32;
    for (int e = rank * kAdders + threadIdx.x - kFirstPromoter * 32; e < rows * (BN / 2); e += KS * kAdders) {
      const int m = e / (BN / 2), c = (e % (BN / 2)) * 2, n = n0 + c;
      if (n >= a.N) continue;
      float2 v = make_float2(0.f, 0.f);
      for (int r = 0; r < KS; ++r) {
        const float2 p = split::load_peer(reinterpret_cast<const float2*>(tile_out + m * BN + c), r);
        v.x += p.x;
        v.y += p.y;
      }
      __half* y = static_cast<__half*>(a.y) + static_cast<size_t>(m0 + m) * a.N + n;
      if (pairs) *reinterpret_cast<__half2*>(y) = __floats2half2_rn(v.x, v.y);
      else { y[0] = __float2half_rn(v.x); if (n + 1 < a.N) y[1] = __float2half_rn(v.y); }
    }
    split::cluster_sync();   // peers keep their shared memory alive until it has been read
    return;
  }
  dev::tc_fence_before();
  __syncthreads();
  // TMEM goes back before this CTA waits for its cluster: a CTA never holds it while it depends on another one
  if (warp == 3) {
    dev::tc_fence_after();
    dev::tmem_dealloc(tmem_base, 512);
  }
  if (KS > 1) {
    split::cluster_sync();
    split::cluster_sync();
  }
}

template <int FMT, int CPT>
static int resident(int ks) {
  static std::atomic<int> cache[kMaxDevices][split::kMaxCluster + 1];
  return split::resident_clusters(mx_prefill_kernel<FMT, CPT>, kThreads, Cfg<FMT, CPT>::kSmem, 1, ks, cache);
}

// How a call is cut: rows per tile (a multiple of 16) and CTAs that share a tile.  A CTA alone works off tiles one after
// the other and hides its hand-overs behind the next tile; a cluster has one tile.
// The microseconds are a fit to calls of a graph (mxfp8 and nvfp4, K 1024 to 14336, N 1536 to 28672, M 20 to 512, all cuts:
// 9 % off in the mean); what it chooses is 0.8 % slower than the best cut in the mean, 12 % at worst (64 rows instead of 48).
struct Cut {
  int bm, mt, ks;
  int64_t tiles;
  float us;
};
static int rows_per_thread(int bm) { return bm <= 64 ? 32 : (bm <= 128 ? 64 : 96); }
template <typename Fn>
static Cut choose_cut(bool nv, int64_t M, int64_t N, int64_t K, Fn held) {
  Cut best = {16, 1, 1, 0, -1.f};
  const int64_t nt = (N + BN - 1) / BN, stages = (K + BK - 1) / BK, blocks = (K + kUnitK - 1) / kUnitK;
  const int64_t least = (M + kMaxRows - 1) / kMaxRows;
  for (int64_t mt = least; mt <= least + 3; ++mt) {
    const int bm = static_cast<int>(((M + mt - 1) / mt + 15) / 16 * 16);
    if ((M + bm - 1) / bm != mt) continue;
    const float stage = (bm * 0.0034f > 0.468f ? bm * 0.0034f : 0.468f) * (nv ? 0.82f : 1.f);
    for (int ks = 1; ks <= split::kMaxCluster && ks <= blocks; ++ks) {
      if (ks > 1 && nt * mt > 65535) break;
      // the device holds fewer clusters than it answers where their size does not divide a GPC's SMs: 48 clusters of three
      // take two rounds (M = 64, 4096 x 6144: 22.8 us, 74 of two 15.0 us)
      const int c = (ks & (ks - 1)) == 0 ? held(bm, ks) : held(bm, ks) * 15 / 16;
      const float rounds = static_cast<float>((nt * mt + c - 1) / c);
      const int64_t slice = (blocks + ks - 1) / ks * (kUnitK / BK);
      const float run = (slice < stages ? slice : stages) * stage;
      const float us = ks == 1 ? 1.1f + 0.0377f * bm + rounds * (run + 2.1f) : rounds * (4.1f + 0.0363f * bm + run);
      if (best.us < 0.f || us < best.us) best = {bm, static_cast<int>(mt), ks, nt * mt, us};
    }
  }
  return best;
}

template <int FMT, int CPT>
static int launch(Args a, const Cut& cut, cudaStream_t stream) {
  using C = Cfg<FMT, CPT>;
  CUtensorMap wmap, xmap;
  const uint64_t row_bytes = static_cast<uint64_t>(a.K) * C::kBits / 8;
  if (int rc = make_tensor_map_2d(&wmap, a.w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)a.N, row_bytes, row_bytes, BN, 128,
                                  CU_TENSOR_MAP_SWIZZLE_128B))
    return rc;
  if (int rc = make_tensor_map_2d(&xmap, a.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (uint64_t)a.M, (uint64_t)a.K, (uint64_t)a.K * 2,
                                  a.bm, 64, CU_TENSOR_MAP_SWIZZLE_128B))
    return rc;
  static std::atomic<uint64_t> configured{0};
  auto kern = mx_prefill_kernel<FMT, CPT>;
  if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), C::kSmem, configured)) return rc;
  const int held = resident<FMT, CPT>(cut.ks);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cut.ks, cut.ks > 1 || a.tiles < held ? a.tiles : held);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = C::kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  split::set_attrs(cfg, attr, cut.ks);
  QMM_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, wmap, xmap, a));
  return QMM_OK;
}

template <int FMT>
static bool run(Args a, cudaStream_t stream, int* rc) {
  const Cut cut = choose_cut(FMT == kNvfp4, a.M, a.N, a.K, [](int bm, int ks) {
    return bm <= 64 ? resident<FMT, 32>(ks) : (bm <= 128 ? resident<FMT, 64>(ks) : resident<FMT, 96>(ks));
  });
  if (cut.tiles > INT_MAX || (!force_split_k() && cut.us > opg::cuda_core_us(FMT, false, a.M, a.N, a.K))) return false;
  if (int st = read_device_status()) {
    *rc = set_error(QMM_ERR_TIMEOUT, "quantized matmul: an earlier kernel gave up a wait (status 0x%x); "
                    "call qmm_clear_device_status() after handling it", st);
    return true;
  }
  a.status = device_status_word();
  a.bm = cut.bm;
  a.mt = cut.mt;
  a.tiles = static_cast<int>(cut.tiles);
  a.idesc = dev::make_idesc(/*c=f32*/ 1, 0, 0, /*both K-major*/ 0, 0, BN, a.bm);
  switch (rows_per_thread(a.bm)) {
    case 32: *rc = launch<FMT, 32>(a, cut, stream); break;
    case 64: *rc = launch<FMT, 64>(a, cut, stream); break;
    default: *rc = launch<FMT, 96>(a, cut, stream); break;
  }
  return true;
}

}  // namespace mxp

// mode: 0 mxfp4, 1 mxfp8, 2 nvfp4; f16 activations.  K a multiple of 32, weights and activations 16-byte aligned, results
// aligned for pairs, four rows or more, and no slower than the CUDA cores by the estimates of both (few columns and rows over
// a short K).  False: not taken, *rc as it was.
bool mx_prefill(int mode, const void* x, const void* w, const void* scales, void* y, int64_t M, int64_t N, int64_t K,
                void* stream, int* rc) {
  using namespace mxp;
  if (M < 4 || K % 32 != 0 || !aligned(x, 16) || !aligned(w, 16) || !aligned(y, 4)) return false;
  Args a = {};
  a.x = x;
  a.w = static_cast<const uint8_t*>(w);
  a.scales = scales;
  a.y = y;
  a.M = static_cast<int>(M);
  a.N = static_cast<int>(N);
  a.K = static_cast<int>(K);
  a.block_k = kUnitK;   // units, boxes of raw weights and 16-byte pieces of scales begin with a slice
  a.blocks = (a.K + kUnitK - 1) / kUnitK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (mode) {
    case QMM_MXFP4: return run<kMxfp4>(a, st, rc);
    case QMM_MXFP8: return run<kMxfp8>(a, st, rc);
    default: return run<kNvfp4>(a, st, rc);
  }
}

}  // namespace qmm
