// Operator-API matmuls with f16 activations at prompt sizes (weights [N, K], K contiguous), on tcgen05.
//
//   y[m,n] = sum_k x[m,k] * w[n,k],   w = s * element (MX formats)  or  s * q + b (affine)
//
// The weights are the 128-row operand of the MMA and go into it through TMEM: a converter thread owns one output column,
// reads its packed codes from shared memory and writes them as f16 pairs into its own TMEM lane.  Nothing of a converted
// weight crosses shared memory, which with both operands in it is what bounds such a kernel (64 k of 128 columns x
// 192 rows move 64 KB there in 384 clocks of MMA; with converted weights stored and read back it would be 96 KB).
//
//   MX formats: element * scale goes in, exactly.  A significand has at most 6 bits; the power-of-two scales of a column are
//     taken relative to the largest of 512 k (a unit), and f16 holds all bits of an element down to 2^-22 (mxfp8) or 2^-36
//     (mxfp4) of that scale.  nvfp4's scale * element always fits.  One accumulator runs over a unit; promoters then add it,
//     times the unit's scale, to f32 registers, so that the tensor core's truncated additions stay short.  A column with a
//     group below that range that is not zero is computed again from global memory, with the CUDA cores' arithmetic.
//   affine: the codes q go in, exactly, one scale group (at most 64 k) per accumulator; promoters apply s and b in f32:
//     acc += s * D + b * sum(x).  sum(x) comes from mma.sync against ones.  Results that are not finite are computed again.
//
// Persistent CTAs, one per SM.  Warps: TMA of activations, TMA of raw weights, the MMA issuer; three warpgroups of
// converters that take the 128-k stages in turn; two warpgroups of promoters, a thread of which holds up to 96 rows of a
// column in registers (setmaxnreg).  Two or more accumulators, so that
// neither a promotion nor the store of a tile stops the tensor core.  Where tiles are few, the CTAs of a cluster share
// one, each with a slice of K, and add their parts over distributed shared memory in a fixed order.
#include "opapi_convert.cuh"
#include "split_k.cuh"

namespace qmm {
namespace opp {

using namespace opg;

constexpr int BN = 128;               // output columns per tile
constexpr int BK = 128;               // k per stage: waits and arrivals cost a warp some 100 clocks each, a stage of 64 k was bound by them
constexpr int kRawBox = BN * 128;     // 16 KB of raw weights
constexpr int kUnitK = 512;           // k per accumulator, MX formats
constexpr int kInfo = 16;             // units whose activation sums are kept; tiles whose columns may be marked
constexpr int kMaxRows = 192;
constexpr int kMaxCluster = 8;
constexpr int kGroups = 3;            // warpgroups of converters
constexpr int kFirstConverter = 4, kFirstPromoter = kFirstConverter + 4 * kGroups, kThreads = (kFirstPromoter + 8) * 32;
constexpr int kLaunchRegs = 65536 / kThreads / 8 * 8;
constexpr int kSBoxes = 4;            // affine: boxes of scales and biases (four groups each) on their way to the promoters
constexpr int kSBoxBytes = 2 * BN * 16;
constexpr uint32_t kMarked = 0x7FC0F1A6u;   // partial result of a column that has to be computed again

template <int FMT, int CPT>   // CPT: rows of a tile (accumulator columns) per promoter thread, at most
struct Cfg {
  static constexpr int kBits = (FMT == kAffine8 || FMT == kMxfp8) ? 8 : 4;
  static constexpr bool kBias = FMT == kAffine4 || FMT == kAffine8;
  static constexpr bool kE8m0 = FMT == kMxfp4 || FMT == kMxfp8;
  static constexpr int kStagesPerBox = 128 * 8 / kBits / BK;
  static constexpr int kSlots = kBias || CPT == 96 ? 2 : 4;      // stages of converted weights in TMEM
  static constexpr int kRows = 2 * CPT;
  static constexpr int kXBytes = kRows * BK * 2;
  // activations in flight: a copy takes about 1 us from request to arrival, a stage's MMAs 0.02 - 0.2 us
  static constexpr int kXStages = CPT == 96 ? 3 : (CPT == 64 ? 4 : 8);
  static constexpr int kAccBase = kSlots * (BK / 2);            // first TMEM column of the accumulators
  static constexpr int kAccBufs = (512 - kAccBase) / kRows;
  static constexpr int kRawBoxes = kBias || kBits == 8 ? 3 : 4;
  static constexpr int kOffRaw = kXStages * kXBytes;
  static constexpr int kOffInfo = kOffRaw + kRawBoxes * kRawBox;
  static constexpr int kOffS = kOffInfo + (kBias ? kInfo * kRows * 4 : (kE8m0 ? kInfo * BN * 4 : 0));
  static constexpr int kOffBar = kOffS + (kBias ? kSBoxes * kSBoxBytes : 0);
  static constexpr int kSmem = kOffBar + 1024 + 1024;
  // scale that brings the largest element of a unit's largest scale just below f16's limit, and the smallest power of
  // two of a group's factor at which the last bit of an element is still there
  static constexpr int kUp = FMT == kMxfp8 ? 7 : 13, kLowest = FMT == kMxfp8 ? -15 : -23;
  static_assert(kAccBufs >= 2 && kSlots <= kXStages && kSlots + kAccBufs + 3 <= kInfo && (!kBias || 4 * kSlots + kAccBufs <= kInfo), "ring sizes");
  // registers of a thread: producers and issuer, converters, promoters
  static constexpr int kMiscRegs = kBias && CPT == 96 ? 40 : 32, kConverterRegs = kBias && CPT == 96 ? 56 : 64;
  static constexpr int kPromoterRegs = kBias && CPT == 96 ? 136 : 128;
  static_assert(128 * kMiscRegs + kGroups * 128 * kConverterRegs + 256 * kPromoterRegs <= kThreads * kLaunchRegs, "registers of the launch");
  static_assert(kRows * BN * 4 <= kOffInfo, "the result tile reuses the rings");
  static_assert(kSmem <= 227 * 1024, "shared memory");
};

struct Args {
  const void* x;
  const uint8_t* w;
  const void* scales;
  const float* biases;
  void* y;
  int M, N, K, gs, pu;       // pu: k per accumulator
  int bm, mt, tiles;         // rows per tile, tiles along M, tiles in all
  int blocks, block_k;       // K in blocks of the slice granularity
  int sbox_k;                // affine: k per box of scales; 0: promoters read them from global memory
  uint32_t idesc;
  int* status;
};

__device__ __forceinline__ void mma_f16_ones(float (&d)[4], const uint32_t (&a)[4]) {
  constexpr uint32_t kOnes = 0x3C003C00u;
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %8}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(kOnes));
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}

// A wait that usually finds its phase complete.
__device__ __forceinline__ bool wait_warp(uint64_t* bar, uint32_t parity, int* status, int tag) {
  if (__all_sync(0xFFFFFFFFu, dev::mbar_try_wait(bar, parity))) return true;
  return dev::mbar_wait_warp(bar, parity, status, tag);
}

// e8m0 scales of a column's unit: 16 bytes, 0 behind the end of the row
__device__ __forceinline__ uint4 unit_scales(const uint8_t* row, int g0, int G, bool vec) {
  if (vec) return __ldg(reinterpret_cast<const uint4*>(row + g0));
  uint32_t r[4] = {0u, 0u, 0u, 0u};
#pragma unroll
  for (int i = 0; i < 16; ++i)
    if (g0 + i < G) r[i >> 2] |= static_cast<uint32_t>(__ldg(row + g0 + i)) << (8 * (i & 3));
  return make_uint4(r[0], r[1], r[2], r[3]);
}
// the largest of them, NaN codes (255) left out
__device__ __forceinline__ int unit_largest(const uint4& s) {
  int best = 0;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const uint32_t w = i < 4 ? s.x : (i < 8 ? s.y : (i < 12 ? s.z : s.w));
    const int b = (w >> (8 * (i & 3))) & 0xFF;
    if (b != 255) best = max(best, b);
  }
  return best;
}

template <int FMT, int CPT>
__global__ void __launch_bounds__(kThreads, 1)
op_prefill_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap,
                  const __grid_constant__ CUtensorMap smap, const __grid_constant__ CUtensorMap bmap, const __grid_constant__ Args a) {
  using C = Cfg<FMT, CPT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  float* xsum = reinterpret_cast<float*>(smem + C::kOffInfo);          // [kInfo][kRows], affine
  uint32_t* marks = reinterpret_cast<uint32_t*>(smem + C::kOffInfo);   // [kInfo][BN], MX: number of the tile that marked the column
  uint64_t* rfull = reinterpret_cast<uint64_t*>(smem + C::kOffBar);    // raw weights landed
  uint64_t* rempty = rfull + C::kRawBoxes;                                // and converted
  uint64_t* xfull = rempty + C::kRawBoxes;                                // activations landed
  uint64_t* full = xfull + C::kXStages;                                    // stage ready for its MMAs
  uint64_t* consumed = full + C::kSlots;                                 // and multiplied (one per slot of the activations)
  uint64_t* dfull = consumed + C::kXStages;                                // a unit's accumulator complete
  uint64_t* dempty = dfull + C::kAccBufs;                              // and drained
  uint64_t* info = dempty + C::kAccBufs;                               // activation sums of a unit / marks of a tile written
  uint64_t* sfull = info + kInfo;                                      // a box of scales landed
  uint64_t* sempty = sfull + kSBoxes;                                  // and read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sempty + kSBoxes);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int KS = gridDim.x, rank = blockIdx.x;
  const int k_begin = static_cast<int>(static_cast<long long>(a.blocks) * rank / KS) * a.block_k;
  const int k_end = min(a.K, static_cast<int>(static_cast<long long>(a.blocks) * (rank + 1) / KS) * a.block_k);
  const int stages = (k_end - k_begin + BK - 1) / BK;
  const int boxes = (stages + C::kStagesPerBox - 1) / C::kStagesPerBox;
  const int units = (k_end - k_begin + a.pu - 1) / a.pu;
  const int parts = C::kBias ? BK / a.pu : 1;   // units per stage, where a unit is no more than a stage

  if (warp == 0) {
    if (lane < C::kRawBoxes) { dev::mbar_init(&rfull[lane], 1); dev::mbar_init(&rempty[lane], C::kStagesPerBox * 4); }
    if (lane < C::kXStages) { dev::mbar_init(&xfull[lane], 1); dev::mbar_init(&consumed[lane], 1); }
    if (lane < C::kSlots) dev::mbar_init(&full[lane], 4);
    if (lane < C::kAccBufs) { dev::mbar_init(&dfull[lane], 1); dev::mbar_init(&dempty[lane], 8); }
    if (lane < kInfo) dev::mbar_init(&info[lane], C::kBias ? 4 : 4 * kGroups);
    if (lane < kSBoxes) { dev::mbar_init(&sfull[lane], 1); dev::mbar_init(&sempty[lane], 8); }
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
            if (!dev::mbar_wait_relaxed(&consumed[s], ((cnt / C::kXStages) & 1) ^ 1, a.status, 111)) { ok = false; break; }
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
    } else if (warp == 3) {
      // ------------------- TMA producer: affine scales and biases ------------
      if (C::kBias && a.sbox_k && lane == 0) {
        uint32_t cnt = 0;
        bool ok = true;
        for (int t = blockIdx.y; ok && t < a.tiles; t += gridDim.y) {
          for (int k = k_begin; k < k_end; k += a.sbox_k, ++cnt) {
            const uint32_t s = cnt % kSBoxes;
            if (!dev::mbar_wait_relaxed(&sempty[s], ((cnt / kSBoxes) & 1) ^ 1, a.status, 109)) { ok = false; break; }
            uint8_t* dst = smem + C::kOffS + s * kSBoxBytes;
            dev::mbar_expect_tx(&sfull[s], kSBoxBytes);
            dev::tma_load_2d(dst, &smap, &sfull[s], k / a.gs, (t / a.mt) * BN);
            dev::tma_load_2d(dst + BN * 16, &bmap, &sfull[s], k / a.gs, (t / a.mt) * BN);
          }
        }
        for (uint32_t i = cnt > kSBoxes ? cnt - kSBoxes : 0; i < cnt; ++i)
          if (!dev::mbar_wait_relaxed(&sfull[i % kSBoxes], (i / kSBoxes) & 1, a.status, 110)) break;
      }
    } else if (warp == 2) {
      // ------------------------------ MMA issuer -----------------------------
      if (dev::elect_one()) {
        constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);   // SBO, version, 128-byte swizzle
        const uint32_t x_lo = ((dev::smem_u32(smem) >> 4) & 0x3FFF) | ((16u >> 4) << 16);
        uint32_t cnt = 0, xs = 0, buf = 0, bpar = 1;   // bpar: parity of the wait for the accumulator, flips with every round
        bool ok = true;
        for (int t = blockIdx.y; ok && t < a.tiles; t += gridDim.y) {
          for (int st = 0; ok && st < stages; ++st, ++cnt) {
            const uint32_t s = cnt % C::kSlots;
            if (!dev::mbar_wait(&full[s], (cnt / C::kSlots) & 1, a.status, 115)) { ok = false; break; }
            const uint32_t at = tmem_base + s * (BK / 2), b_lo = x_lo + xs * (C::kXBytes >> 4);
            // a step of 16 k: 8 columns of TMEM, 32 bytes of a row; 64 k of activations are one swizzled tile
            auto step = [&](uint32_t d, int j, uint32_t accumulate) {
              dev::umma_f16_ts(d, at + j * 8, b_lo + (j >> 2) * (C::kXBytes >> 5) + (j & 3) * 2, kDescHi, a.idesc, accumulate);
            };
            if (C::kBias) {
              for (int h = 0; h < parts; ++h) {
                if (st * parts + h >= units) break;
                if (!dev::mbar_wait(&dempty[buf], bpar, a.status, 116)) { ok = false; break; }
                dev::tc_fence_after();
                const uint32_t d = tmem_base + C::kAccBase + buf * C::kRows;
                if (parts == 2) {
#pragma unroll
                  for (int j = 0; j < 4; ++j) step(d, h * 4 + j, j != 0);
                } else {
#pragma unroll
                  for (int j = 0; j < 2; ++j) step(d, h * 2 + j, j != 0);
                }
                dev::tc_commit(&dfull[buf]);
                if (++buf == C::kAccBufs) { buf = 0; bpar ^= 1; }
              }
            } else {
              const bool first = st % (kUnitK / BK) == 0;
              if (first && !dev::mbar_wait(&dempty[buf], bpar, a.status, 116)) { ok = false; break; }
              dev::tc_fence_after();
              const uint32_t d = tmem_base + C::kAccBase + buf * C::kRows;
#pragma unroll
              for (int j = 0; j < 8; ++j) step(d, j, !first || j != 0);
              if (st % (kUnitK / BK) == kUnitK / BK - 1 || st == stages - 1) {
                dev::tc_commit(&dfull[buf]);
                if (++buf == C::kAccBufs) { buf = 0; bpar ^= 1; }
              }
            }
            if (ok) dev::tc_commit(&consumed[xs]);
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
    uint32_t cnt0 = 0, box0 = 0, unit0 = 0, tile_no = 0;
    bool ok = true;
    for (int t = blockIdx.y; ok && t < a.tiles; t += gridDim.y, cnt0 += stages, box0 += boxes, unit0 += units, ++tile_no) {
      const int n = min((t / a.mt) * BN + row, a.N - 1);
      // MX: scales of the unit, the largest of them; nvfp4: the eight scales of the next stage
      const int G = C::kE8m0 ? a.K / 32 : a.K / 16;
      const uint8_t* srow = static_cast<const uint8_t*>(a.scales) + static_cast<size_t>(n) * (C::kBias ? 0 : G);
      const bool vec = C::kE8m0 && G % 16 == 0 && (reinterpret_cast<uintptr_t>(a.scales) & 15) == 0;
      const bool pairs8 = FMT == kNvfp4 && G % 8 == 0 && (reinterpret_cast<uintptr_t>(a.scales) & 7) == 0;
      uint4 us = make_uint4(0u, 0u, 0u, 0u), next_us = us;
      int ref = 0, unit = -1;
      uint2 nv = make_uint2(0u, 0u);
      auto load_nv = [&](int st) {
        const int g = (k_begin + st * BK) / 16;
        if (pairs8) return __ldg(reinterpret_cast<const uint2*>(srow + g));
        uint2 r = make_uint2(0u, 0u);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (g + i < G) r.x |= static_cast<uint32_t>(__ldg(srow + g + i)) << (8 * i);
          if (g + 4 + i < G) r.y |= static_cast<uint32_t>(__ldg(srow + g + 4 + i)) << (8 * i);
        }
        return r;
      };
      if (C::kE8m0) next_us = unit_scales(srow, k_begin / 32, G, vec);
      // The groups take the stages of all tiles in turn, so that a group has seen, with its stage before, the phase ahead of
      // the one that it waits for next (a parity says no more than that).
      const int first = static_cast<int>((grp + kGroups - cnt0 % kGroups) % kGroups);
      if (FMT == kNvfp4 && first < stages) nv = load_nv(first);
      for (int st = first; st < stages; st += kGroups) {
        const uint32_t c = cnt0 + st, s = c % C::kSlots, xs = c % C::kXStages;
        const uint32_t box = box0 + st / C::kStagesPerBox, rs = box % C::kRawBoxes;
        const int sub = st % C::kStagesPerBox;
        if (C::kE8m0 && st / (kUnitK / BK) != unit) {
          unit = st / (kUnitK / BK);
          us = next_us;
          ref = unit_largest(us);
          const int next = (k_begin + (unit + 1) * kUnitK) / 32;   // every group has a stage in every unit
          if (next < G) next_us = unit_scales(srow, next, G, vec);
        }
        const uint2 nv_now = nv;
        if (FMT == kNvfp4 && st + kGroups < stages) nv = load_nv(st + kGroups);
        if (!wait_warp(&rfull[rs], (box / C::kRawBoxes) & 1, a.status, 117)) { ok = false; break; }
        const uint8_t* raw = smem + C::kOffRaw + rs * kRawBox + row * 128;
        if (c >= C::kSlots) {   // the MMAs that read this slot's TMEM before have retired
          const uint32_t p = c - C::kSlots;
          if (!wait_warp(&consumed[p % C::kXStages], (p / C::kXStages) & 1, a.status, 118)) { ok = false; break; }
          dev::tc_fence_after();
        }
        constexpr int kPieces = C::kBits / 4;   // 16-byte pieces of a column's 32 k
#pragma unroll
        for (int h = 0; h < 4; ++h) {   // 32 k: 16 TMEM columns
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
            const uint32_t word = h < 2 ? nv_now.x : nv_now.y;
            f0 = e4m3_pair<false>((word >> (16 * (h & 1))) & 0xFFu);
            f1 = e4m3_pair<false>((word >> (16 * (h & 1) + 8)) & 0xFFu);
          }
          uint32_t o[16];
          if (C::kBits == 4) {
            const uint32_t in[4] = {v[0].x, v[0].y, v[0].z, v[0].w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint4 r = convert8<FMT, false>(in[i], 0u, i < 2 ? f0 : f1, false);
              o[4 * i] = r.x; o[4 * i + 1] = r.y; o[4 * i + 2] = r.z; o[4 * i + 3] = r.w;
            }
          } else {
#pragma unroll
            for (int i = 0; i < kPieces; ++i) {
              const uint4 r = convert8<FMT, false>(v[i].x, v[i].y, 0u, false), u = convert8<FMT, false>(v[i].z, v[i].w, 0u, false);
              o[8 * i] = r.x; o[8 * i + 1] = r.y; o[8 * i + 2] = r.z; o[8 * i + 3] = r.w;
              o[8 * i + 4] = u.x; o[8 * i + 5] = u.y; o[8 * i + 6] = u.z; o[8 * i + 7] = u.w;
            }
          }
          if (C::kE8m0) {
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = mul2<false>(o[i], f0);
          }
          dev::tmem_st_32x16(a_lane + s * (BK / 2) + h * 16, o);
        }
        if (!wait_warp(&xfull[xs], (c / C::kXStages) & 1, a.status, 119)) { ok = false; break; }
        if (C::kBias) {
          // activation sums of the stage's units: 16 rows at a time against a column of ones
          const uint32_t unit_no = unit0 + st * parts;
          const uint32_t xt = dev::smem_u32(smem + xs * C::kXBytes);
          for (int rb = ww; rb * 16 < a.bm; rb += 4) {
            const int r = rb * 16 + (lane & 15);
            float d[4][4] = {};   // one per 32 k
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              uint32_t f[4];
              ldmatrix_x4(xt + (j >> 2) * (C::kXBytes / 2) + r * 128 + (((2 * (j & 3) + (lane >> 4)) ^ (r & 7)) << 4), f);
              mma_f16_ones(d[j >> 1], f);
            }
            if ((lane & 3) == 0) {
              const int at = rb * 16 + (lane >> 2);
              if (parts == 2) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                  float* dst = xsum + ((unit_no + h) % kInfo) * C::kRows + at;
                  if (st * 2 + h < units) { dst[0] = d[2 * h][0] + d[2 * h + 1][0]; dst[8] = d[2 * h][2] + d[2 * h + 1][2]; }
                }
              } else {
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                  float* dst = xsum + ((unit_no + h) % kInfo) * C::kRows + at;
                  if (st * 4 + h < units) { dst[0] = d[h][0]; dst[8] = d[h][2]; }
                }
              }
            }
          }
        }
        dev::tc_wait_st();
        dev::tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          dev::mbar_arrive(&full[s]);
          dev::mbar_arrive(&rempty[rs]);
        }
        if (C::kBias && lane < parts && st * parts + lane < units) dev::mbar_arrive(&info[(unit0 + st * parts + lane) % kInfo]);
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
    uint32_t buf = 0, bpar = 0, unit_no = 0, tile_no = 0, sb = 0, sb_par = 0;
    bool ok = true;
    uint64_t acc[CPT / 2];
    for (int t = blockIdx.y; ok && t < a.tiles; t += gridDim.y, ++tile_no) {
      const int m0 = (t % a.mt) * a.bm, n = (t / a.mt) * BN + q * 32 + lane, nc = min(n, a.N - 1);
#pragma unroll
      for (int i = 0; i < CPT / 2; ++i) acc[i] = 0ull;
      const int G = C::kBias ? a.K / a.gs : (C::kE8m0 ? a.K / 32 : 0);
      const uint8_t* srow = static_cast<const uint8_t*>(a.scales) + static_cast<size_t>(nc) * (C::kE8m0 ? G : 0);
      const bool vec = C::kE8m0 && G % 16 == 0 && (reinterpret_cast<uintptr_t>(a.scales) & 15) == 0;
      // affine, scales that do not come in boxes: read one unit ahead
      const float* sp = static_cast<const float*>(a.scales) + static_cast<size_t>(nc) * (C::kBias ? G : 0);
      const float* bp = C::kBias ? a.biases + static_cast<size_t>(nc) * G : nullptr;
      const int units_per_group = C::kBias ? a.gs / a.pu : 1;
      int gi = C::kBias ? k_begin / a.gs : 0, gu = C::kBias ? (k_begin % a.gs) / a.pu : 0;   // group and unit of the next load
      float s0 = 1.f, b0 = 0.f;
      auto next_scale = [&]() {
        const int g = min(gi, G - 1);
        s0 = __ldg(sp + g);
        b0 = __ldg(bp + g);
        if (++gu == units_per_group) { gu = 0; ++gi; }
      };
      const int units_per_box = C::kBias && a.sbox_k ? a.sbox_k / a.pu : 0;
      int in_box = 0;
      if (C::kBias && units_per_box == 0) next_scale();
      for (int u = 0; u < units; ++u, ++unit_no) {
        float s = 1.f;
        if (C::kE8m0) {
          const int ref = unit_largest(unit_scales(srow, (k_begin + u * kUnitK) / 32, G, vec));
          s = opapi::decode_e8m0(ref) * __uint_as_float(static_cast<uint32_t>(127 - C::kUp) << 23);
        }
        if (C::kBias) {
          float b = b0;
          s = s0;
          if (units_per_box) {
            if (in_box == 0 && !wait_warp(&sfull[sb], sb_par, a.status, 108)) { ok = false; break; }
            const uint8_t* at = smem + C::kOffS + sb * kSBoxBytes + (q * 32 + lane) * 16 + in_box / units_per_group * 4;
            s = *reinterpret_cast<const float*>(at);
            b = *reinterpret_cast<const float*>(at + BN * 16);
            if (++in_box == units_per_box || u == units - 1) {
              split::release_slot(&sempty[sb], __float_as_uint(s) ^ __float_as_uint(b), a.M < 0, lane);
              in_box = 0;
              if (++sb == kSBoxes) { sb = 0; sb_par ^= 1; }
            }
          } else {
            next_scale();
          }
          const uint64_t b2 = pack2(b, b);
          // the bias's share first: it needs no accumulator
          if (!wait_warp(&info[unit_no % kInfo], (unit_no / kInfo) & 1, a.status, 120)) { ok = false; break; }
          const float* xs = xsum + (unit_no % kInfo) * C::kRows + c0;
#pragma unroll
          for (int c = 0; c < CPT; c += 8) {
            if (c < hc) {
              const ulonglong2 p = *reinterpret_cast<const ulonglong2*>(xs + c), r = *reinterpret_cast<const ulonglong2*>(xs + c + 4);
              fma2(acc[c / 2], b2, p.x);
              fma2(acc[c / 2 + 1], b2, p.y);
              fma2(acc[c / 2 + 2], b2, r.x);
              fma2(acc[c / 2 + 3], b2, r.y);
            }
          }
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
              if (lane == 0) dev::mbar_arrive(&dempty[buf]);
            }
#pragma unroll
            for (int e = 0; e < kLd / 2; ++e)
              fma2(acc[c / 2 + e], s2, pack2(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1])));
          }
        }
        if (++buf == C::kAccBufs) { buf = 0; bpar ^= 1; }
      }
      if (!ok) break;
      bool marked = false;
      if (C::kE8m0) {
        if (!dev::mbar_wait_warp(&info[tile_no % kInfo], (tile_no / kInfo) & 1, a.status, 122)) { ok = false; break; }
        marked = marks[(tile_no % kInfo) * BN + q * 32 + lane] == tile_no + 1;
      }
      if (KS > 1) break;   // one tile per cluster: it is put together below
      // ---- results: two rows at a time, neighbouring lanes exchange so that each stores two columns of one row
      __half* y = static_cast<__half*>(a.y);
      const bool pairs = (a.N & 1) == 0;
      bool redo = marked;
#pragma unroll
      for (int i = 0; i < CPT / 2; ++i) {
        if (2 * i < hc && m0 + c0 + 2 * i < a.M) {
          float v0, v1;
          unpack2(acc[i], v0, v1);
          if (C::kBias) redo |= !(fabsf(v0) < INFINITY) || !(fabsf(v1) < INFINITY);
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
      if (C::kBias || C::kE8m0) {
        __syncwarp();
        if (redo && n < a.N) {
#pragma unroll 1
          for (int m = m0 + c0; m < min(a.M, m0 + c0 + hc); ++m) {
            __half* dst = y + static_cast<size_t>(m) * a.N + n;
            if (marked || !(fabsf(__half2float(*dst)) < INFINITY))
              *dst = __float2half_rn(exact_dot<FMT, false>(a.x, a.w, a.scales, a.biases, a.K, a.gs, m, n, 0, a.K));
          }
        }
      }
    }
    dev::tc_fence_before();
    __syncthreads();   // every warp is done with the rings and with TMEM
    if (KS == 1) return;
    // ---- this slice's results, [row][column], into the idle rings; the cluster's CTAs add up a share of the rows each
    const bool marked = C::kE8m0 && ok && marks[q * 32 + lane] == 1u;
#pragma unroll
    for (int i = 0; i < CPT / 2; ++i) {
      if (2 * i < hc) {
        float v0, v1;
        unpack2(acc[i], v0, v1);
        if (marked) v0 = v1 = __uint_as_float(kMarked);
        tile_out[(c0 + 2 * i) * BN + q * 32 + lane] = v0;
        tile_out[(c0 + 2 * i + 1) * BN + q * 32 + lane] = v1;
      }
    }
    split::cluster_sync();
    const int m0 = (blockIdx.y % a.mt) * a.bm, n0 = (blockIdx.y / a.mt) * BN;
    const int rows = min(a.bm, a.M - m0);
    const bool pairs = (a.N & 1) == 0;
    constexpr int kAdders = kThreads - kFirstPromoter * 32;
    for (int e = rank * kAdders + threadIdx.x - kFirstPromoter * 32; e < rows * (BN / 2); e += KS * kAdders) {
      const int m = e / (BN / 2), c = (e % (BN / 2)) * 2, n = n0 + c;
      if (n >= a.N) continue;
      float2 v = make_float2(0.f, 0.f);
      bool redo_x = false, redo_y = false;
      for (int r = 0; r < KS; ++r) {
        const float2 p = split::load_peer(reinterpret_cast<const float2*>(tile_out + m * BN + c), r);
        if (C::kE8m0) {
          redo_x |= __float_as_uint(p.x) == kMarked;
          redo_y |= __float_as_uint(p.y) == kMarked;
        }
        v.x += p.x;
        v.y += p.y;
      }
      if (C::kBias) {
        redo_x = !(fabsf(v.x) < INFINITY);
        redo_y = !(fabsf(v.y) < INFINITY);
      }
      if (C::kBias || C::kE8m0) {
        if (redo_x) v.x = exact_dot<FMT, false>(a.x, a.w, a.scales, a.biases, a.K, a.gs, m0 + m, n, 0, a.K);
        if (redo_y && n + 1 < a.N) v.y = exact_dot<FMT, false>(a.x, a.w, a.scales, a.biases, a.K, a.gs, m0 + m, n + 1, 0, a.K);
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
  return split::resident_clusters(op_prefill_kernel<FMT, CPT>, kThreads, Cfg<FMT, CPT>::kSmem, 1, ks, cache);
}

// How a call is cut: rows per tile (a multiple of 16) and CTAs that share a tile.  A CTA alone works off tiles one after
// the other and hides its hand-overs behind the next tile; a cluster has one tile.
struct Cut {
  int bm, mt, ks;
  float us;
};
static int rows_per_thread(int bm) { return bm <= 64 ? 32 : (bm <= 128 ? 64 : 96); }
static float stage_us(int fmt, int bm, int pu) { return bm * 0.00115f + 0.05f; }
template <typename Fn>
static Cut choose_cut(int fmt, int M, int N, int K, int pu, int blocks, Fn held) {
  Cut best = {16, 1, 1, -1.f};
  const int nt = (N + BN - 1) / BN, stages = (K + BK - 1) / BK;
  const int least = (M + kMaxRows - 1) / kMaxRows;
  for (int mt = least; mt <= least + 3 || mt * 32 <= M; ++mt) {
    if (mt > least + 3 && mt > 4 * least) break;
    const int bm = ((M + mt - 1) / mt + 15) / 16 * 16;
    if ((M + bm - 1) / bm != mt) continue;
    for (int ks = 1; ks <= kMaxCluster && ks <= blocks; ++ks) {
      const int c = held(bm, ks);
      const int rounds = (nt * mt + c - 1) / c;
      const int slice = (blocks + ks - 1) / ks * ((stages + blocks - 1) / blocks);
      const float run = (slice < stages ? slice : stages) * stage_us(fmt, bm, pu);
      const float us = ks == 1 ? 4.f + rounds * run : rounds * (6.f + run);
      if (best.us < 0.f || us < best.us) best = {bm, mt, ks, us};
    }
  }
  return best;
}
static int unit_k(int fmt, int gs) { return fmt >= kMxfp4 ? kUnitK : (gs % 64 == 0 ? 64 : 32); }
// k per box of affine scales (16 bytes of a column: four groups), where rows of them are made of such pieces
static int scale_box_k(int fmt, int K, int gs, const void* scales, const void* biases) {
  if (fmt >= kMxfp4 || !aligned(scales, 16) || !aligned(biases, 16)) return 0;
  return gs <= 128 && 128 % gs == 0 && (K / gs) % 4 == 0 ? 4 * gs : 0;
}
static int slice_k(int fmt, int sbox_k) {
  const int box_k = fmt >= kMxfp4 ? kUnitK : (fmt == kAffine4 ? 256 : 128);
  return sbox_k > box_k ? sbox_k : box_k;
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
  CUtensorMap smap = wmap, bmap = wmap;   // placeholders where they are not used
  if (a.sbox_k) {
    const uint64_t G = static_cast<uint64_t>(a.K / a.gs);
    if (int rc = make_tensor_map_2d(&smap, a.scales, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (uint64_t)a.N, G, G * 4, BN, 4,
                                    CU_TENSOR_MAP_SWIZZLE_NONE))
      return rc;
    if (int rc = make_tensor_map_2d(&bmap, a.biases, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (uint64_t)a.N, G, G * 4, BN, 4,
                                    CU_TENSOR_MAP_SWIZZLE_NONE))
      return rc;
  }
  static std::atomic<uint64_t> configured{0};
  auto kern = op_prefill_kernel<FMT, CPT>;
  if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), C::kSmem, configured)) return rc;
  const int held = resident<FMT, CPT>(cut.ks);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cut.ks, cut.ks > 1 || a.tiles < held ? a.tiles : held);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = C::kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  split::set_attrs(cfg, attr, cut.ks);
  QMM_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, wmap, xmap, smap, bmap, a));
  return QMM_OK;
}

template <int FMT>
static int launch_fmt(Args a, cudaStream_t stream) {
  const Cut cut = choose_cut(FMT, a.M, a.N, a.K, a.pu, a.blocks, [](int bm, int ks) {
    return bm <= 64 ? resident<FMT, 32>(ks) : (bm <= 128 ? resident<FMT, 64>(ks) : resident<FMT, 96>(ks));
  });
  a.bm = cut.bm;
  a.mt = cut.mt;
  a.tiles = cut.mt * ((a.N + BN - 1) / BN);
  QMM_REQUIRE(cut.ks == 1 || a.tiles <= 65535, QMM_ERR_UNSUPPORTED, "quantized matmul: too many tiles");
  a.idesc = dev::make_idesc(/*c=f32*/ 1, 0, 0, /*both K-major*/ 0, 0, BN, a.bm);
  switch (rows_per_thread(a.bm)) {
    case 32: return launch<FMT, 32>(a, cut, stream);
    case 64: return launch<FMT, 64>(a, cut, stream);
    default: return launch<FMT, 96>(a, cut, stream);
  }
}

}  // namespace opp

// fmt: 0 affine 4-bit, 1 affine 8-bit, 2 mxfp4, 3 mxfp8, 4 nvfp4.  K and the group a multiple of 32 (nvfp4: K), weights
// and activations 16-byte aligned, results aligned for pairs; f16 activations.
bool op_prefill_covers(int64_t M, int64_t N, int64_t K, int fmt, int64_t gs, const void* x, const void* w, const void* y) {
  using namespace opp;
  if (M < 17 || K % 32 != 0 || (fmt <= kAffine8 && gs % 32 != 0)) return false;
  if (!aligned(x, 16) || !aligned(w, 16) || !aligned(y, 4)) return false;
  return true;
}

int op_prefill_launch(int fmt, const void* x, const void* w, const void* scales, const float* biases, void* y, int64_t M,
                      int64_t N, int64_t K, int64_t gs, void* stream) {
  using namespace opp;
  if (int st = read_device_status())
    return set_error(QMM_ERR_TIMEOUT, "quantized matmul: an earlier kernel gave up a wait (status 0x%x); "
                     "call qmm_clear_device_status() after handling it", st);
  Args a = {};
  a.x = x;
  a.w = static_cast<const uint8_t*>(w);
  a.scales = scales;
  a.biases = biases;
  a.y = y;
  a.M = static_cast<int>(M);
  a.N = static_cast<int>(N);
  a.K = static_cast<int>(K);
  a.gs = static_cast<int>(gs);
  a.pu = unit_k(fmt, a.gs);
  a.sbox_k = scale_box_k(fmt, a.K, a.gs, scales, biases);
  a.block_k = slice_k(fmt, a.sbox_k);
  a.blocks = (a.K + a.block_k - 1) / a.block_k;
  a.status = device_status_word();
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (fmt) {
    case kAffine4: return launch_fmt<kAffine4>(a, st);
    case kAffine8: return launch_fmt<kAffine8>(a, st);
    case kMxfp4: return launch_fmt<kMxfp4>(a, st);
    case kMxfp8: return launch_fmt<kMxfp8>(a, st);
    default: return launch_fmt<kNvfp4>(a, st);
  }
}

}  // namespace qmm
