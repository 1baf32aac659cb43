// Operator-API matmuls (weights [N, K], K contiguous) on the 5th-generation tensor cores: any number of rows, f32
// activations and all five weight formats, f16 activations and the affine formats (the MX formats go to mx_prefill.cu).
//
//   y[m,n] = sum over groups g of  s[n,g] * sum_{k in g} x[m,k] c[n,k]  (+ b[n,g] * sum_{k in g} x[m,k])
//
// The weights go to tcgen05.mma as their bare codes c (an integer, or the e2m1 / e4m3 element), which
// both 16-bit types hold exactly: f16 against f16 activations, bf16 against f32 activations, which are cut into
// three bf16 terms that add up to all 24 bits.  Every product is therefore exact.  The accumulator of one unit of
// k (a scale group or a part of one, up to 64 k) is read back from TMEM and multiplied by the group's f32 scale into f32
// registers, so that scales and biases stay in 32 bits and the tensor core adds up no more than 64 k before a
// correctly rounded f32 addition takes over.  nvfp4, whose groups of 16 would be too short for that, multiplies
// its elements by their e4m3 scale first: 2 + 4 significant bits, exact as well.
//
// A CTA computes 128 columns (the MMA's 128 rows: a lane of the accumulator is a column, so a scale is one
// register) x BM rows over a slice of K; the CTAs of a cluster share an output tile and add their slices over
// distributed shared memory in a fixed order.  Warps: two TMA producers (raw weights in boxes of 128 rows x 128
// bytes with their scales; activations), groups of one MMA issuer and four workers that turn raw codes into the swizzled operand (and f32
// activations into their three terms, and sum the activations of a unit for the biases) and four to
// sixteen promoters that drain the accumulators.
//
// Measured (four linears of a layer, before: one warp per four columns on CUDA cores): affine 4-bit, f32, M = 48, 2048 / 5632
// wide 597 -> 98 us.  Bound by latency, not by a unit: a stage takes 0.9-1.3 us through workers, issuer, tensor core and
// promoter.
//
// What the split cannot represent takes an exact path: a unit whose activations are not finite (inf times
// code plus inf times bias is not what inf times scale * code + bias gives), or, for f32, lie outside 2^-100 .. 2^100, is computed by
// the promoters from global memory with the arithmetic of the CUDA-core kernels; and so are affine results that are not
// finite, because of their scales or biases.
#include <cooperative_groups.h>

#include "opapi_convert.cuh"
#include "split_k.cuh"

namespace cg = cooperative_groups;

namespace qmm {
namespace opg {

constexpr int BN = 128;               // output columns per CTA
constexpr int BK = 64;                // k per operand stage: one 128-byte row of 16-bit values
constexpr int kGroupWarps = 4;        // warps that convert one stage; the groups take the stages in turn
constexpr int kRawBox = BN * 128;     // 16 KB of raw weights
constexpr int kABytes = BN * BK * 2;  // 16 KB
constexpr int kInfo = 32;             // units whose activation sums and flags are kept (power of two)
constexpr int kConsumed = 24;         // stages whose retirement can be asked for (more than twice the deepest ring)
constexpr int kMaxCluster = 8;
constexpr int kSBoxes = 3;            // boxes of scales (and biases) on their way to the promoters
constexpr int kSBoxBytes = 2 * BN * 16;

template <int FMT, bool XF32, int BM>
struct Cfg {
  static constexpr int kBits = (FMT == kAffine8 || FMT == kMxfp8) ? 8 : 4;
  static constexpr bool kBias = FMT == kAffine4 || FMT == kAffine8;
  static_assert(kBias || XF32, "MX formats with f16 activations: mx_prefill.cu");   // sums and / or flags travel with a unit
  static constexpr int kTerms = XF32 ? 3 : 1;
  static constexpr int kBoxK = 128 * 8 / kBits;             // k per raw box
  static constexpr int kStagesPerBox = kBoxK / BK;          // 4 or 2
  static constexpr int kXTile = BM * BK * 2;                // one 16-bit operand tile of activations
  static constexpr int kXRaw = BM * BK * 4;                 // raw f32 activations of a stage
  // Groups of four workers and an issuer take the stages in turn.  With one group of eight warps a stage took 1.2 us
  // (mxfp8) to 3.3 us (f32 activations); with three or four groups the registers per thread fall to 72 and the workers
  // and promoters spill, which cost more than the groups gave (affine4, f32, M = 1, 4096 x 8192: 54 us against 33 us).
  static constexpr int kGroups = 2;
  static constexpr int kWorkerWarps = kGroups * kGroupWarps;
  // A stage takes 2-4 us from raw codes to retired MMAs and an accumulator about 1.5 us from one unit to the next,
  // nearly all of it latency: the rings are as deep as shared memory and TMEM allow.
  static constexpr int kOps = XF32 ? (BM == 32 ? 5 : 3) : (BM == 32 ? 8 : (BM == 64 ? 6 : 4));   // operand stages
  static constexpr int kAccBufs = BM == 128 ? 4 : 8;        // accumulators between the tensor core and the promoters
  static constexpr int kOpBytes = kABytes + (XF32 ? 3 * kXTile : 0);
  static constexpr int kXRing = XF32 ? (BM == 32 ? 4 : 3) : kOps;
  static constexpr int kXBytes = XF32 ? kXRaw : kXTile;
  static constexpr int kRawBoxes = XF32 ? 2 : 3;
  static constexpr int kOffX = kOps * kOpBytes;
  static constexpr int kOffRaw = kOffX + kXRing * kXBytes;
  static constexpr int kOffInfo = kOffRaw + kRawBoxes * kRawBox;
  static constexpr int kOffS = kOffInfo + kInfo * BM * 4;
  static constexpr int kOffFlags = kOffS + (FMT == kNvfp4 ? 0 : kSBoxes * kSBoxBytes);
  static constexpr int kOffBar = kOffFlags + kInfo * kGroupWarps;
  static constexpr int kSmem = kOffBar + 1024 + 1024;
  static constexpr int kPromoters = BM / 8;               // four lane quarters x 32 columns each
  static constexpr int kFirstIssuer = 2;
  static constexpr int kFirstWorker = kFirstIssuer + kGroups;   // one issuing warp per group
  static constexpr int kFirstPromoter = kFirstWorker + kWorkerWarps;
  static constexpr int kThreads = (kFirstPromoter + kPromoters) * 32;
  static constexpr int kCols = 32;                        // accumulator columns per promoter
  // One thread issues all units of one accumulator, in order: its wait for the previous unit to be drained can then not
  // take the drain of the unit before that for it (the parities are the same).
  static_assert(kAccBufs % (2 * kGroups) == 0, "two units per stage, one issuer per group");
  static_assert(BM * BN * 4 <= kOffInfo, "the result tile reuses the rings");
  static_assert((kAccBufs & (kAccBufs - 1)) == 0 && (kInfo & (kInfo - 1)) == 0 && 2 * kOps + kAccBufs + 1 <= kInfo && kInfo <= 32 && 2 * kOps < kConsumed && kConsumed <= 32, "ring sizes");
  static_assert(kSmem <= 227 * 1024, "shared memory");
};

struct Args {
  const void* x;
  const uint8_t* w;
  const void* scales;
  const float* biases;
  void* y;
  int M, N, K, gs, pu;        // pu: k per unit (32 or 64)
  int blocks, block_k;        // K in blocks of the slice granularity
  int sbox_k;                 // k per box of scales; 0: their rows are not made of 16-byte pieces, promoters read them
  uint32_t idesc;
  int* status;
};

// A call either way: which form it has decides how the promoters around it are compiled (arguments one by one against a
// reference: affine, M = 48, 4096 x 14336 77 and 87 us; mxfp4, M = 32 70 and 65 us).
template <int FMT, bool XF32>
__device__ __noinline__ float exact_unit_ref(const Args& a, int m, int n, int k0, int k1) {
  return exact_dot_here<FMT, XF32>(a.x, a.w, a.scales, a.biases, a.K, a.gs, m, n, k0, k1);
}
template <int FMT, bool XF32>
__device__ __forceinline__ float exact_unit(const Args& a, int m, int n, int k0, int k1) {
  if constexpr (FMT <= kAffine8) return exact_dot<FMT, XF32>(a.x, a.w, a.scales, a.biases, a.K, a.gs, m, n, k0, k1);
  else return exact_unit_ref<FMT, XF32>(a, m, n, k0, k1);
}

template <int FMT, bool XF32, int BM>
__global__ void __launch_bounds__(Cfg<FMT, XF32, BM>::kThreads, 1)
opgemm_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap,
              const __grid_constant__ CUtensorMap smap, const __grid_constant__ CUtensorMap bmap, const __grid_constant__ Args a) {
  using C = Cfg<FMT, XF32, BM>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  float* xsum = reinterpret_cast<float*>(smem + C::kOffInfo);        // [kInfo][BM]
  uint8_t* flags = smem + C::kOffFlags;                              // [kInfo][4], one byte per warp of a group
  uint64_t* wfull = reinterpret_cast<uint64_t*>(smem + C::kOffBar);  // raw weights landed
  uint64_t* wempty = wfull + C::kRawBoxes;                           // raw weights read
  uint64_t* xfull = wempty + C::kRawBoxes;                           // activations landed
  uint64_t* xempty = xfull + C::kXRing;                              // raw f32 activations read (f32 only)
  uint64_t* full = xempty + C::kXRing;                               // operand stage written
  uint64_t* consumed = full + C::kOps;                               // the MMAs of a stage retired
  uint64_t* tfull = consumed + kConsumed;                            // a unit's accumulator complete
  uint64_t* tempty = tfull + C::kAccBufs;                               // and drained
  uint64_t* ifull = tempty + C::kAccBufs;                               // sums and flags of a unit written
  uint64_t* sfull = ifull + kInfo;                                   // a box of scales landed
  uint64_t* sempty = sfull + kSBoxes;                                // and read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sempty + kSBoxes);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int KS = gridDim.x, rank = blockIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.z * BN;
  const int k_begin = static_cast<int>(static_cast<long long>(a.blocks) * rank / KS) * a.block_k;
  const int k_end = min(a.K, static_cast<int>(static_cast<long long>(a.blocks) * (rank + 1) / KS) * a.block_k);
  const int stages = (k_end - k_begin + BK - 1) / BK;
  const int units = (k_end - k_begin + a.pu - 1) / a.pu;

  if (warp == 0) {   // one barrier of each kind per lane
    if (lane < C::kRawBoxes) { dev::mbar_init(&wfull[lane], 1); dev::mbar_init(&wempty[lane], C::kStagesPerBox * kGroupWarps); }
    if (lane < C::kXRing) { dev::mbar_init(&xfull[lane], 1); dev::mbar_init(&xempty[lane], kGroupWarps); }
    if (lane < C::kOps) dev::mbar_init(&full[lane], kGroupWarps);
    if (lane < kConsumed) dev::mbar_init(&consumed[lane], 1);
    if (lane < C::kAccBufs) { dev::mbar_init(&tfull[lane], 1); dev::mbar_init(&tempty[lane], C::kPromoters); }
    if (lane < kInfo) dev::mbar_init(&ifull[lane], kGroupWarps);
    if (lane < kSBoxes) { dev::mbar_init(&sfull[lane], 1); dev::mbar_init(&sempty[lane], C::kPromoters); }
    dev::fence_mbar_init();
  } else if (warp == 2 && lane == 0) {
    dev::tma_prefetch_desc(&wmap);
    dev::tma_prefetch_desc(&xmap);
    dev::tma_prefetch_desc(&smap);
    dev::tma_prefetch_desc(&bmap);
  }
  if (warp == 1) {
    dev::tmem_alloc(tmem_slot, C::kAccBufs * BM);
    dev::tmem_relinquish();
  }
  dev::tc_fence_before();
  __syncthreads();
  dev::tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
  dev::pdl_wait();
  dev::pdl_launch_dependents();

  constexpr int kFirstPromoter = C::kFirstPromoter;
  float* tile = reinterpret_cast<float*>(smem);   // [BM][BN] f32 partial results, once the rings are idle

  if (warp == 0) {
    // ------------------------ TMA producer: activations --------------------
    if (lane == 0) {
      int xi = 0;
      for (; xi < stages; ++xi) {
        const int s = xi % C::kXRing;
        if (XF32) {
          if (!dev::mbar_wait_relaxed(&xempty[s], ((xi / C::kXRing) & 1) ^ 1, a.status, 91)) break;
        } else if (xi >= C::kXRing) {
          const int prev = xi - C::kXRing;
          if (!dev::mbar_wait_relaxed(&consumed[prev % kConsumed], (prev / kConsumed) & 1, a.status, 91)) break;
        }
        dev::mbar_expect_tx(&xfull[s], C::kXBytes);
        dev::tma_load_2d(smem + C::kOffX + s * C::kXBytes, &xmap, &xfull[s], k_begin + xi * BK, m0);
      }
      // every copy has landed before this CTA's shared memory is reused, whatever the other warps did
      for (int i = xi > C::kXRing ? xi - C::kXRing : 0; i < xi; ++i)
        if (!dev::mbar_wait_relaxed(&xfull[i % C::kXRing], (i / C::kXRing) & 1, a.status, 93)) break;
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------- TMA producer: raw weights and scales --------------
    // A box of scales goes out just before the weights of its first stage.
    if (lane == 0) {
      const int boxes = (stages + C::kStagesPerBox - 1) / C::kStagesPerBox;
      const bool boxed = FMT != kNvfp4 && a.sbox_k != 0;
      const int sstages = boxed ? a.sbox_k / BK : 1;   // stages per box of scales
      const int sboxes = boxed ? (stages + sstages - 1) / sstages : 0;
      int wi = 0, si = 0;
      while (wi < boxes) {
        while (si < sboxes && si * sstages < (wi + 1) * C::kStagesPerBox) {
          const int s = si % kSBoxes;
          if (!dev::mbar_wait_relaxed(&sempty[s], ((si / kSBoxes) & 1) ^ 1, a.status, 89)) goto drained;
          uint8_t* dst = smem + C::kOffS + s * kSBoxBytes;
          dev::mbar_expect_tx(&sfull[s], C::kBias ? kSBoxBytes : BN * 16);
          const int c = (k_begin + si * a.sbox_k) / a.gs;   // first group of the box
          dev::tma_load_2d(dst, &smap, &sfull[s], c, n0);
          if (C::kBias) dev::tma_load_2d(dst + BN * 16, &bmap, &sfull[s], c, n0);
          ++si;
        }
        const int s = wi % C::kRawBoxes;
        if (!dev::mbar_wait_relaxed(&wempty[s], ((wi / C::kRawBoxes) & 1) ^ 1, a.status, 90)) break;
        dev::mbar_expect_tx(&wfull[s], kRawBox);
        dev::tma_load_2d(smem + C::kOffRaw + s * kRawBox, &wmap, &wfull[s], k_begin * C::kBits / 8 + wi * 128, n0);
        ++wi;
      }
    drained:
      for (int i = wi > C::kRawBoxes ? wi - C::kRawBoxes : 0; i < wi; ++i)
        if (!dev::mbar_wait_relaxed(&wfull[i % C::kRawBoxes], (i / C::kRawBoxes) & 1, a.status, 92)) break;
      for (int i = si > kSBoxes ? si - kSBoxes : 0; i < si; ++i)
        if (!dev::mbar_wait_relaxed(&sfull[i % kSBoxes], (i / kSBoxes) & 1, a.status, 88)) break;
    }
    __syncwarp();
  } else if (warp < C::kFirstWorker) {
    // ------------------------------ MMA issuers ----------------------------
    // One per worker group: an MMA costs its issuing thread some 140 clocks, which with twelve of them per stage (f32)
    // would bound everything; the units of different stages are independent.
    if (lane == 0) {
      constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);   // SBO, version, 128-byte swizzle
      const uint32_t op_lo = ((dev::smem_u32(smem) >> 4) & 0x3FFF) | ((16u >> 4) << 16);
      const uint32_t x_lo = ((dev::smem_u32(smem + C::kOffX) >> 4) & 0x3FFF) | ((16u >> 4) << 16);
      const int units_per_stage = a.pu < BK ? BK / a.pu : 1;
      bool ok = true;
      for (int st = warp - C::kFirstIssuer; ok && st < stages; st += C::kGroups) {
        const int s = st % C::kOps;
        if (!dev::mbar_wait(&full[s], (st / C::kOps) & 1, a.status, 94)) break;
        dev::tc_fence_after();
        const uint32_t a_lo = op_lo + s * (C::kOpBytes >> 4);
        const uint32_t b_lo = XF32 ? a_lo + (kABytes >> 4) : x_lo + (st % C::kXRing) * (C::kXTile >> 4);
        for (int h = 0; h < units_per_stage; ++h) {
          const int u = st * units_per_stage + h;
          const int buf = u % C::kAccBufs;
          if (!dev::mbar_wait(&tempty[buf], ((u / C::kAccBufs) & 1) ^ 1, a.status, 95)) { ok = false; break; }
          if (u >= units) {   // the zero half of a last stage: no MMAs, but its buffer's barrier is the stage's
            dev::tc_commit(&tfull[buf]);
            break;
          }
          dev::tc_fence_after();
          const uint32_t d = tmem_base + buf * BM;
          // the smallest terms first: the accumulator is still small when they are added
          if (units_per_stage == 1) {
#pragma unroll
            for (int t = C::kTerms - 1; t >= 0; --t)
#pragma unroll
              for (int j = 0; j < 4; ++j)
                dev::umma_f16_lh(d, a_lo + j * 2, kDescHi, b_lo + t * (C::kXTile >> 4) + j * 2, kDescHi, a.idesc,
                                 (t != C::kTerms - 1 || j != 0) ? 1u : 0u);
          } else {
#pragma unroll
            for (int t = C::kTerms - 1; t >= 0; --t)
#pragma unroll
              for (int j = 0; j < 2; ++j)
                dev::umma_f16_lh(d, a_lo + h * 4 + j * 2, kDescHi, b_lo + t * (C::kXTile >> 4) + h * 4 + j * 2, kDescHi, a.idesc,
                                 (t != C::kTerms - 1 || j != 0) ? 1u : 0u);
          }
          // A commit costs the thread as much as an MMA: one for the units of a stage, on the barrier of its last buffer.
          // That barrier completes once in every round of the buffers, after the buffer was handed back in the round before
          // (also where there is no unit for it), as the parity that the promoters wait for takes for granted; the one of
          // a stage's first buffer never completes.
          if (h == units_per_stage - 1) dev::tc_commit(&tfull[buf]);
        }
        if (ok) dev::tc_commit(&consumed[st % kConsumed]);
      }
    }
    __syncwarp();
  } else if (warp < kFirstPromoter) {
    // ------------------------------ workers --------------------------------
    const int grp = (warp - C::kFirstWorker) / kGroupWarps, ww = (warp - C::kFirstWorker) % kGroupWarps;
    const int wt = ww * 32 + lane;                    // 0 .. 127
    const int units_per_stage = a.pu < BK ? BK / a.pu : 1;
    // rows behind the last one are left as they are: a row of the results depends on its own activations only (M = 48, f32,
    // 2048 x 11264: 44.0 us with all 64 rows of a tile cut, 42.6 without)
    const int row_blocks = (min(BM, a.M - m0) + 15) / 16;
    constexpr int kW = C::kBits == 4 ? 2 : 4;         // 16-byte pieces of weights per thread: row wrow(i), piece wpiece of the stage
    const int wpiece = C::kBits == 4 ? (wt & 1) : (wt & 3);
    auto wrow = [&](int i) { return C::kBits == 4 ? (wt >> 1) + i * 64 : (wt >> 2) + i * 32; };
    constexpr int kPieceK = C::kBits == 4 ? 32 : 16;  // k of a piece
    // f32 results: scale and bias of this thread's rows in its next stage, for the decision to centre their codes
    constexpr bool kCentre = C::kBias && XF32;
    float csc[kW], cbi[kW];
    auto load_centre = [&](int st) {
      if (kCentre) {
#pragma unroll
        for (int i = 0; i < kW; ++i) {
          const int n = min(n0 + wrow(i), a.N - 1), k = min(k_begin + st * BK + wpiece * kPieceK, a.K - 1);
          const size_t g = static_cast<size_t>(n) * (a.K / a.gs) + k / a.gs;
          csc[i] = __ldg(static_cast<const float*>(a.scales) + g);
          cbi[i] = __ldg(a.biases + g);
        }
      }
    };
    load_centre(grp);
    for (int st = grp; st < stages; st += C::kGroups) {
      const int op = st % C::kOps;
      uint8_t* opA = smem + op * C::kOpBytes;
      const int box = st / C::kStagesPerBox, sub = st % C::kStagesPerBox, rs = box % C::kRawBoxes;
      const uint8_t* raw = smem + C::kOffRaw + rs * kRawBox;
      bool centre[kW];
#pragma unroll
      for (int i = 0; i < kW; ++i) {
        float shifted;
        centre[i] = kCentre && centred<FMT>(csc[i], cbi[i], shifted);
      }
      if (st + C::kGroups < stages) load_centre(st + C::kGroups);
      // nvfp4: the two scales of each piece's 32 k, fetched before the wait for the weights
      uint32_t nsc[kW][2];
      if (FMT == kNvfp4) {
#pragma unroll
        for (int i = 0; i < kW; ++i) {
          const int n = n0 + wrow(i), k = k_begin + st * BK + wpiece * 32;
          nsc[i][0] = nsc[i][1] = 0u;
          if (n < a.N && k < a.K) {
            const uint8_t* sp = static_cast<const uint8_t*>(a.scales) + static_cast<size_t>(n) * (a.K / 16) + k / 16;
            nsc[i][0] = __ldg(sp);
            nsc[i][1] = __ldg(sp + 1);
          }
        }
      }
      if (!dev::mbar_wait_relaxed_warp(&wfull[rs], (box / C::kRawBoxes) & 1, a.status, 96)) break;
      uint4 v[kW];
#pragma unroll
      for (int i = 0; i < kW; ++i) {
        const int row = wrow(i), c = sub * (C::kBits == 4 ? 2 : 4) + wpiece;
        v[i] = *reinterpret_cast<const uint4*>(raw + row * 128 + ((c ^ (row & 7)) << 4));
      }
      if (st >= C::kOps) {   // the MMAs that read this operand stage before have retired
        const int prev = st - C::kOps;
        if (!dev::mbar_wait_relaxed_warp(&consumed[prev % kConsumed], (prev / kConsumed) & 1, a.status, 97)) break;
      }
#pragma unroll
      for (int i = 0; i < kW; ++i) {
        const int row = wrow(i);
        auto put = [&](int chunk, const uint4& o) {
          *reinterpret_cast<uint4*>(opA + row * 128 + ((chunk ^ (row & 7)) << 4)) = o;
        };
        if (C::kBits == 4) {
          uint32_t sc[2] = {0u, 0u};
          if (FMT == kNvfp4) { sc[0] = e4m3_pair<XF32>(nsc[i][0]); sc[1] = e4m3_pair<XF32>(nsc[i][1]); }
          put(wpiece * 4, convert8<FMT, XF32>(v[i].x, 0u, sc[0], centre[i]));
          put(wpiece * 4 + 1, convert8<FMT, XF32>(v[i].y, 0u, sc[0], centre[i]));
          put(wpiece * 4 + 2, convert8<FMT, XF32>(v[i].z, 0u, sc[1], centre[i]));
          put(wpiece * 4 + 3, convert8<FMT, XF32>(v[i].w, 0u, sc[1], centre[i]));
        } else {
          put(wpiece * 2, convert8<FMT, XF32>(v[i].x, v[i].y, 0u, centre[i]));
          put(wpiece * 2 + 1, convert8<FMT, XF32>(v[i].z, v[i].w, 0u, centre[i]));
        }
      }
      // ---- activations: eight lanes per row, eight k each
      const int xs = st % C::kXRing;
      if (!dev::mbar_wait_relaxed_warp(&xfull[xs], (st / C::kXRing) & 1, a.status, 98)) break;
      const int slot = (units_per_stage * st) % kInfo;   // first unit of this stage (a unit with sums is at most a stage)
      {
        const uint8_t* xt = smem + C::kOffX + xs * C::kXBytes;
        uint32_t bad = 0;   // bit 0: first half of the stage, bit 1: second half
        auto rows16 = [&](int i) {
          const int row = (wt >> 3) + i * 16, j = wt & 7;
          float f[8];
          bool odd = false;
          if (XF32) {
            const float4 p = *reinterpret_cast<const float4*>(xt + row * 256 + j * 32);
            const float4 q = *reinterpret_cast<const float4*>(xt + row * 256 + j * 32 + 16);
            f[0] = p.x; f[1] = p.y; f[2] = p.z; f[3] = p.w;
            f[4] = q.x; f[5] = q.y; f[6] = q.z; f[7] = q.w;
            // x = hi + mid + lo
            uint32_t h[4], mi[4], lo[4];
            if constexpr (BM == 32) {   // the top 8 bits, the next 8, the rest (mxfp4, M = 32, 4096 x 14336: 65 us, 70 us as below)
              float r[8], q[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) {
                const uint32_t b = __float_as_uint(f[e]), mag = b & 0x7FFFFFFFu;
                odd |= mag != 0u && mag - (27u << 23) >= (200u << 23);
                r[e] = f[e] - __uint_as_float(b & 0xFFFF0000u);
                q[e] = r[e] - __uint_as_float(__float_as_uint(r[e]) & 0xFFFF0000u);
              }
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                h[e] = __byte_perm(__float_as_uint(f[2 * e]), __float_as_uint(f[2 * e + 1]), 0x7632);
                mi[e] = __byte_perm(__float_as_uint(r[2 * e]), __float_as_uint(r[2 * e + 1]), 0x7632);
                lo[e] = __byte_perm(__float_as_uint(q[2 * e]), __float_as_uint(q[2 * e + 1]), 0x7632);
              }
            } else {   // each the nearest bf16 of what is left: fewer instructions (M = 48: 79 us, 84 us as above)
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                h[e] = dev::pack_bf16x2(f[2 * e], f[2 * e + 1]);
                const float r0 = f[2 * e] - __uint_as_float(h[e] << 16), r1 = f[2 * e + 1] - __uint_as_float(h[e] & 0xFFFF0000u);
                mi[e] = dev::pack_bf16x2(r0, r1);
                lo[e] = dev::pack_bf16x2(r0 - __uint_as_float(mi[e] << 16), r1 - __uint_as_float(mi[e] & 0xFFFF0000u));
              }
              // nonzero magnitudes below 2^-100 (twice the bits, less one: zero is the largest) or from 2^100; a NaN goes through
              // the sums
              uint32_t least = 0xFFFFFFFFu;
              float most = 0.f;
#pragma unroll
              for (int e = 0; e < 8; e += 2) {
                least = __vimin3_u32(least, 2u * __float_as_uint(f[e]) - 1u, 2u * __float_as_uint(f[e + 1]) - 1u);
                most = fmaxf(most, fmaxf(fabsf(f[e]), fabsf(f[e + 1])));
              }
              odd = least < (27u << 24) - 1u || !(most < __uint_as_float(227u << 23));
            }
            uint8_t* xo = opA + kABytes + row * 128 + ((j ^ (row & 7)) << 4);
            *reinterpret_cast<uint4*>(xo) = make_uint4(h[0], h[1], h[2], h[3]);
            *reinterpret_cast<uint4*>(xo + C::kXTile) = make_uint4(mi[0], mi[1], mi[2], mi[3]);
            *reinterpret_cast<uint4*>(xo + 2 * C::kXTile) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
          } else {
            const uint4 p = *reinterpret_cast<const uint4*>(xt + row * 128 + ((j ^ (row & 7)) << 4));
            const uint32_t h[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float2 q = __half22float2(*reinterpret_cast<const __half2*>(&h[e]));
              f[2 * e] = q.x;
              f[2 * e + 1] = q.y;
            }
          }
          if (C::kBias) {
            float sum = ((f[0] + f[1]) + (f[2] + f[3])) + ((f[4] + f[5]) + (f[6] + f[7]));
            sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 1);
            sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 2);
            if (units_per_stage == 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 4);
            if (!XF32) odd = !(fabsf(sum) < INFINITY);   // f16 sums cannot overflow: inf or NaN was among the values
            if (units_per_stage == 2) {
              if ((j & 3) == 0) xsum[((slot + (j >> 2)) % kInfo) * BM + row] = sum;
            } else if (j == 0) {
              xsum[slot * BM + row] = sum;
            }
          }
          const uint32_t b = __ballot_sync(0xFFFFFFFFu, odd);
          bad |= (b & 0x0F0F0F0Fu ? 1u : 0u) | (b & 0xF0F0F0F0u ? 2u : 0u);
        };
        if (row_blocks == BM / 16) {
#pragma unroll (XF32 ? 2 : 4)
          for (int i = 0; i < BM / 16; ++i) rows16(i);
        } else {
#pragma unroll 1
          for (int i = 0; i < row_blocks; ++i) rows16(i);
        }
        if (units_per_stage == 2) {
          if (lane < 2) flags[((slot + lane) % kInfo) * kGroupWarps + ww] = (bad >> lane) & 1;
        } else if (lane == 0) {
          flags[slot * kGroupWarps + ww] = bad != 0;
        }
      }
      dev::fence_proxy_async();
      __syncwarp();
      if (lane == 0) {
        // raw weights and activations go back after the fence that completed the stores made from them: an arrival
        // right behind the loads let a refill overtake them
        dev::mbar_arrive(&wempty[rs]);
        if (XF32) dev::mbar_arrive(&xempty[xs]);
        dev::mbar_arrive(&full[op]);
        dev::mbar_arrive(&ifull[slot]);
        if (units_per_stage == 2) dev::mbar_arrive(&ifull[(slot + 1) % kInfo]);
      }
    }
  } else {
    // ------------------------------ promoters ------------------------------
    const int q = warp & 3, half = (warp - kFirstPromoter) >> 2;
    const int n = n0 + q * 32 + lane;
    const int nc = min(n, a.N - 1);
    const int c0 = half * C::kCols;
    const int units_per_group = (FMT == kNvfp4) ? 1 : a.gs / a.pu;
    const int units_per_stage = a.pu < BK ? BK / a.pu : 1;
    const int u_base = k_begin / a.pu;
    const int G = (FMT == kNvfp4) ? 1 : a.K / a.gs;
    const int total_units = (a.K + a.pu - 1) / a.pu;
    uint64_t acc[C::kCols / 2];
#pragma unroll
    for (int i = 0; i < C::kCols / 2; ++i) acc[i] = 0ull;
    auto load_scale = [&](int u, float& s, float& b) {
      const int uu = min(u_base + u, total_units - 1);
      if (C::kBias) {
        const size_t i = static_cast<size_t>(nc) * G + uu / units_per_group;
        s = __ldg(static_cast<const float*>(a.scales) + i);
        b = __ldg(a.biases + i);
      } else if (FMT != kNvfp4) {
        s = opapi::decode_e8m0(__ldg(static_cast<const uint8_t*>(a.scales) + static_cast<size_t>(nc) * G + uu));
      }
    };
    // Scales come in boxes (one TMA copy for all promoters), else each promoter reads its lanes' values ahead.
    const int units_per_box = FMT != kNvfp4 && a.sbox_k ? a.sbox_k / a.pu : 0;
    float s_next = 1.f, b_next = 0.f;
    if (units_per_box == 0) load_scale(0, s_next, b_next);
    int in_box = 0, in_group = 0, comp = 0;   // unit of the box, unit of the group, group of the box
    uint32_t sb = 0, sb_phase = 0, phase = 0;  // ring slot and parity of the box; parity of the accumulators' round
    for (int u = 0; u < units; ++u) {
      const int buf = u & (C::kAccBufs - 1), slot = u & (kInfo - 1);
      float s = s_next, b = b_next;
      if (units_per_box) {
        if (in_box == 0 && !dev::mbar_wait_relaxed_warp(&sfull[sb], sb_phase, a.status, 101)) break;
        const uint8_t* row = smem + C::kOffS + sb * kSBoxBytes + (q * 32 + lane) * 16;
        if (C::kBias) {
          s = reinterpret_cast<const float*>(row)[comp];
          b = reinterpret_cast<const float*>(row + BN * 16)[comp];
        } else {
          s = opapi::decode_e8m0(row[in_box]);
        }
      } else {
        load_scale(u + 1, s_next, b_next);
      }
      const uint32_t scale_dep = __float_as_uint(s) ^ __float_as_uint(b);
      if (C::kBias && XF32) {
        float shifted;
        if (centred<FMT>(s, b, shifted)) b = shifted;
      }
      if (FMT == kAffine8 && XF32) s *= 64.f;
      if (!dev::mbar_wait_relaxed_warp(&ifull[slot], (u / kInfo) & 1, a.status, 99)) break;
      const bool exact = *reinterpret_cast<const uint32_t*>(flags + slot * kGroupWarps) != 0u;
      // the units of a stage complete together, on the barrier of its last buffer
      const int last = units_per_stage == 2 ? (u | 1) & (C::kAccBufs - 1) : buf;
      if (!dev::mbar_wait_relaxed_warp(&tfull[last], phase, a.status, 100)) break;
      dev::tc_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + buf * BM + c0;
      if (exact) {
        // the unit's exact sums take the accumulator's place (registers cannot be indexed)
        const int k0 = k_begin + u * a.pu, k1 = min(a.K, k0 + a.pu);
#pragma unroll 1
        for (int c = 0; c < C::kCols; ++c)
          dev::tmem_st_32x1(taddr + c, m0 + c0 + c < a.M ? __float_as_uint(exact_unit<FMT, XF32>(a, m0 + c0 + c, nc, k0, k1)) : 0u);
        dev::tc_wait_st();
        s = 1.f;
      }
      const uint64_t s2 = pack2(s, s), b2 = pack2(b, b);
      const bool with_bias = C::kBias && !exact;
#pragma unroll
      for (int c = 0; c < C::kCols; c += 16) {   // 16 at a time: registers
        uint32_t r[16];
        dev::tmem_ld_32x16(taddr + c, r);
        dev::tc_wait_ld();
        if (c + 16 == C::kCols) {                // the last values are in registers: the buffer goes back
          dev::tc_fence_before();
          __syncwarp();
          if (lane == 0) dev::mbar_arrive(&tempty[buf]);
        }
        if (with_bias) {
          // scale and bias terms cancel in part: they meet before they are added to the running sum
          const ulonglong2* xp = reinterpret_cast<const ulonglong2*>(xsum + slot * BM + c0 + c);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const ulonglong2 t = xp[e];
            uint64_t v0 = fmul2(b2, t.x), v1 = fmul2(b2, t.y);
            fma2(v0, s2, pack2(__uint_as_float(r[4 * e]), __uint_as_float(r[4 * e + 1])));
            fma2(v1, s2, pack2(__uint_as_float(r[4 * e + 2]), __uint_as_float(r[4 * e + 3])));
            add2(acc[c / 2 + 2 * e], v0);
            add2(acc[c / 2 + 2 * e + 1], v1);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e)
            fma2(acc[c / 2 + e], s2, pack2(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1])));
        }
      }
      if (buf == C::kAccBufs - 1) phase ^= 1;
      if (++in_group == units_per_group) { in_group = 0; ++comp; }
      if (units_per_box && ++in_box == units_per_box) {
        split::release_slot(&sempty[sb], scale_dep, a.M < 0, lane);
        in_box = comp = 0;
        if (++sb == kSBoxes) { sb = 0; sb_phase ^= 1; }
      }
    }
    // ---- this slice's results, [row][column], into the idle rings (after every warp is done with them)
    dev::tc_fence_before();
    __syncthreads();
#pragma unroll
    for (int c = 0; c < C::kCols; c += 2) {
      float v0, v1;
      unpack2(acc[c / 2], v0, v1);
      tile[(c0 + c) * BN + q * 32 + lane] = v0;
      tile[(c0 + c + 1) * BN + q * 32 + lane] = v1;
    }
  }
  if (warp < kFirstPromoter) {
    dev::tc_fence_before();
    __syncthreads();
  }
  // TMEM goes back before this CTA waits for its cluster: a CTA never holds it while it depends on another one
  if (warp == 1) {
    dev::tc_fence_after();
    dev::tmem_dealloc(tmem_base, C::kAccBufs * BM);
  }
  cg::cluster_group cluster = cg::this_cluster();
  if (KS > 1) cluster.sync();
  else __syncthreads();
  const int rows = min(BM, a.M - m0);
  const bool pairs = (a.N & 1) == 0;
  for (int e = rank * C::kThreads + threadIdx.x; e < rows * (BN / 2); e += KS * C::kThreads) {
    const int m = e / (BN / 2), c = (e % (BN / 2)) * 2, n = n0 + c;
    if (n >= a.N) continue;
    float2 v = make_float2(0.f, 0.f);
    for (int r = 0; r < KS; ++r) {
      const float2 p = *reinterpret_cast<const float2*>((KS > 1 ? cluster.map_shared_rank(tile, r) : tile) + m * BN + c);
      v.x += p.x;
      v.y += p.y;
    }
    if (C::kBias) {
      // A scale or bias that is not finite leaves results that are not; which ones are infinities and which NaN, weight by
      // weight, is not what the scaled sums give (an infinite scale times a code of 0).
      if (!(fabsf(v.x) < INFINITY)) v.x = exact_unit<FMT, XF32>(a, m0 + m, n, 0, a.K);
      if (!(fabsf(v.y) < INFINITY) && n + 1 < a.N) v.y = exact_unit<FMT, XF32>(a, m0 + m, n + 1, 0, a.K);
    }
    const size_t i = static_cast<size_t>(m0 + m) * a.N + n;
    if (XF32) {
      float* y = static_cast<float*>(a.y) + i;
      if (pairs) *reinterpret_cast<float2*>(y) = v;
      else { y[0] = v.x; if (n + 1 < a.N) y[1] = v.y; }
    } else {
      __half* y = static_cast<__half*>(a.y) + i;
      if (pairs) *reinterpret_cast<__half2*>(y) = __floats2half2_rn(v.x, v.y);
      else { y[0] = __float2half_rn(v.x); if (n + 1 < a.N) y[1] = __float2half_rn(v.y); }
    }
  }
  if (KS > 1) cluster.sync();   // peers keep their shared memory alive until it has been read
}

static void set_attrs(cudaLaunchConfig_t& cfg, cudaLaunchAttribute (&attr)[2], int ks) {
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = ks;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
}

// Clusters of `ks` CTAs that the current device holds at once (asked once per device and size).
template <int FMT, bool XF32, int BM>
static int resident_clusters(int ks) {
  static std::atomic<int> cache[kMaxDevices][kMaxCluster + 1];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return num_sms() / ks;
  int n = cache[dev][ks].load(std::memory_order_relaxed);
  if (n > 0) return n;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  cfg.gridDim = dim3(ks, 1, 1024);
  cfg.blockDim = dim3(Cfg<FMT, XF32, BM>::kThreads);
  cfg.dynamicSmemBytes = Cfg<FMT, XF32, BM>::kSmem;
  set_attrs(cfg, attr, ks);
  if (cudaOccupancyMaxActiveClusters(&n, opgemm_kernel<FMT, XF32, BM>, &cfg) != cudaSuccess || n < 1) {
    (void)cudaGetLastError();
    n = num_sms() / ks > 0 ? num_sms() / ks : 1;
  }
  cache[dev][ks].store(n, std::memory_order_relaxed);
  return n;
}

// CTAs that share an output tile: the fewest rounds of resident clusters (six CTAs to a cluster, for one, leave SMs of
// every GPC idle), a round costing its stages and, for the prologue and the hand-over, about as much as kRoundCost more.
constexpr int kRoundCost = 16;
struct Rounds {
  int ks, rounds, stages;   // CTAs to a cluster; rounds of clusters; stages of the longest slice
};
template <typename Fn>
static Rounds choose_rounds(int tiles, int blocks, int stages, Fn resident) {
  Rounds best = {1, 1, stages};
  long long best_cost = -1;
  for (int ks = 1; ks <= kMaxCluster && ks <= blocks; ++ks) {
    const int c = resident(ks);
    const int slice = (blocks + ks - 1) / ks * ((stages + blocks - 1) / blocks);
    const int rounds = (tiles + c - 1) / c;
    const long long cost = static_cast<long long>(rounds) * (slice + kRoundCost);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best = {ks, rounds, slice < stages ? slice : stages};
    }
  }
  return best;
}

// How K is cut.  A unit is a scale group or a part of one, and no more than a stage: its MMAs come from one thread, and the
// tensor core's own, truncated additions have to be cut short against f32 results (128 k: 2.5e-7 of the result, 64 k: 1e-7).
// Slices of K begin on a box of raw weights and on a box of scales.
struct Slicing {
  int pu, sbox_k, block_k, blocks;
};
static Slicing slicing(int fmt, int K, int gs, bool scales_aligned) {
  Slicing c;
  const bool bias = fmt <= kAffine8;
  c.pu = fmt == kNvfp4 || gs % 64 == 0 ? 64 : 32;
  const bool boxed = fmt == kNvfp4 || !scales_aligned ? false
                     : bias                           ? gs <= 128 && (K / gs) % 4 == 0 && 128 % gs == 0
                                                      : K % 512 == 0 && K >= 2048;   // (slices of a short K stay fine)
  c.sbox_k = !boxed ? 0 : (bias ? 4 * gs : 512);
  const int box_k = fmt == kAffine8 || fmt == kMxfp8 ? 128 : 256;
  c.block_k = c.sbox_k > box_k ? c.sbox_k : box_k;
  c.blocks = (K + c.block_k - 1) / c.block_k;
  return c;
}

template <int FMT, bool XF32, int BM>
static int launch(Args a, cudaStream_t stream) {
  using C = Cfg<FMT, XF32, BM>;
  CUtensorMap wmap, xmap;
  const uint64_t row_bytes = static_cast<uint64_t>(a.K) * C::kBits / 8;
  if (int rc = make_tensor_map_2d(&wmap, a.w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)a.N, row_bytes, row_bytes, BN, 128,
                                  CU_TENSOR_MAP_SWIZZLE_128B))
    return rc;
  if (int rc = make_tensor_map_2d(&xmap, a.x, XF32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                                  XF32 ? 4 : 2, (uint64_t)a.M, (uint64_t)a.K, (uint64_t)a.K * (XF32 ? 4 : 2), BM, BK,
                                  XF32 ? CU_TENSOR_MAP_SWIZZLE_NONE : CU_TENSOR_MAP_SWIZZLE_128B))
    return rc;
  static std::atomic<uint64_t> configured{0};
  auto kern = opgemm_kernel<FMT, XF32, BM>;
  if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), C::kSmem, configured)) return rc;
  const Slicing cut = slicing(FMT, a.K, a.gs, aligned(a.scales, 16) && (!C::kBias || aligned(a.biases, 16)));
  a.pu = cut.pu;
  a.sbox_k = cut.sbox_k;
  a.block_k = cut.block_k;
  a.blocks = cut.blocks;
  static_assert(C::kBoxK == (FMT == kAffine8 || FMT == kMxfp8 ? 128 : 256), "box of raw weights");
  CUtensorMap smap = wmap, bmap = wmap;   // placeholders where they are not used
  if (cut.sbox_k) {
    const uint64_t G = static_cast<uint64_t>(a.K / a.gs);
    const auto type = C::kBias ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_UINT8;
    const int esz = C::kBias ? 4 : 1;
    if (int rc = make_tensor_map_2d(&smap, a.scales, type, esz, (uint64_t)a.N, G, G * esz, BN, 16 / esz, CU_TENSOR_MAP_SWIZZLE_NONE))
      return rc;
    if (C::kBias)
      if (int rc = make_tensor_map_2d(&bmap, a.biases, type, esz, (uint64_t)a.N, G, G * esz, BN, 16 / esz, CU_TENSOR_MAP_SWIZZLE_NONE))
        return rc;
  }
  a.idesc = dev::make_idesc(/*c=f32*/ 1, XF32 ? 1 : 0, XF32 ? 1 : 0, /*both K-major*/ 0, 0, BN, a.M < BM ? (a.M + 15) / 16 * 16 : BM);
  a.status = device_status_word();
  const int nt = (a.N + BN - 1) / BN, mt = (a.M + BM - 1) / BM;
  const int ks = choose_rounds(nt * mt, a.blocks, (a.K + BK - 1) / BK, resident_clusters<FMT, XF32, BM>).ks;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ks, mt, nt);
  cfg.blockDim = dim3(C::kThreads);
  cfg.dynamicSmemBytes = C::kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  set_attrs(cfg, attr, ks);
  QMM_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, wmap, xmap, smap, bmap, a));
  return QMM_OK;
}

template <int FMT>
static int launch_f32(const Args& a, cudaStream_t stream) {
  // a stage of 128 rows would need 64 KB for the three terms of the activations alone
  return a.M <= 32 ? launch<FMT, true, 32>(a, stream) : launch<FMT, true, 64>(a, stream);
}
template <int FMT>
static int launch_affine(const Args& a, int f32, cudaStream_t stream) {
  if (f32) return launch_f32<FMT>(a, stream);
  return a.M <= 32 ? launch<FMT, false, 32>(a, stream)
                   : (a.M <= 64 ? launch<FMT, false, 64>(a, stream) : launch<FMT, false, 128>(a, stream));
}

// Microseconds of a call, here and on the CUDA cores (one B200, calls of a graph on operands in L2; K and N from 64 to 4096,
// M from 4 to 500, every format: here within 6 % in the mean, there within 9 %).
//   here: rounds of clusters, each a start and a hand-over, and its stages
//   there: a block of 16 columns and 8 rows runs over K by itself; three blocks fit an SM, and more of them queue
static float gemm_us(int fmt, bool f32, int M, int N, int K, int gs) {
  const int bm = M <= 32 ? 32 : (M <= 64 || f32 ? 64 : 128);
  const int i = bm == 32 ? 0 : (bm == 64 ? 1 : 2);
  static constexpr float kStart[3] = {4.2f, 5.5f, 7.5f};
  // us per stage of 64 k, at 32, 64 and (f16) 128 rows
  static constexpr float kStageF16[2][3] = {{1.33f, 1.71f, 3.5f},    // affine, units of 32 k
                                            {0.91f, 1.12f, 2.0f}};   // affine, 64 k
  static constexpr float kStageF32[4][2] = {{1.48f, 1.84f}, {1.12f, 1.32f},
                                            {1.11f, 1.26f},    // mxfp4, mxfp8
                                            {0.92f, 1.01f}};   // nvfp4
  const Slicing cut = slicing(fmt, K, gs, true);
  const int kind = fmt == kNvfp4 ? 3 : (fmt > kAffine8 ? 2 : (cut.pu == 64 ? 1 : 0));
  const int sms = num_sms();
  const Rounds r = choose_rounds(((N + BN - 1) / BN) * ((M + bm - 1) / bm), cut.blocks, (K + BK - 1) / BK,
                                 [&](int ks) { return sms / ks > 0 ? sms / ks : 1; });
  return r.rounds * (kStart[i] + (f32 ? kStageF32[kind][i] : kStageF16[kind][i]) * r.stages);
}
float cuda_core_us(int fmt, bool f32, int M, int N, int K) {
  const bool wide = fmt == kAffine8 || fmt == kMxfp8;   // 8-bit codes take fewer instructions
  const float least = f32 ? (wide ? 6.5f : 10.4f) : (wide ? 5.6f : 8.6f);
  const float run = 3.f + K * (f32 ? (wide ? 0.0079f : 0.0089f) : (wide ? 0.0057f : 0.0056f));
  float us = least > run ? least : run;
  if (M <= 4) us *= 0.74f;
  const float blocks = static_cast<float>((N + 15) / 16) * ((M + 7) / 8);
  return blocks <= 3 * num_sms() ? us : us * (0.75f + blocks / (3.5f * num_sms()));
}

}  // namespace opg

// Which calls come here: those that take no longer than on the CUDA cores, by the estimates above.  Few blocks of columns
// and rows over a short K stay there (affine8, f32, 512 x 1024 at M = 4: 5.1 us there, 8.3 here; at M = 64 12.9, 10.6), and
// so do up to three rows, which the estimates do not cover (affine4, f32, 4096 x 8192: 30 us at one row, 62 at four, here
// 32 for any of them).
// QMM_FORCE_SPLIT_K=1 brings every call here that the kernel can take (a cross-check; read once per process).
// fmt: 0 affine 4-bit, 1 affine 8-bit, and for f32 activations 2 mxfp4, 3 mxfp8, 4 nvfp4.  K and the group a multiple of 32 (nvfp4: K), weights
// and activations 16-byte aligned, results aligned for pairs.
bool opgemm_covers(int64_t M, int64_t N, int64_t K, int fmt, int64_t gs, int f32, const void* x, const void* w, const void* y) {
  using namespace opg;
  if (M < 4 || K % 32 != 0 || (fmt <= kAffine8 && gs % 32 != 0)) return false;
  if (!aligned(x, 16) || !aligned(w, 16) || !aligned(y, 8)) return false;
  if ((M + 7) / 8 > 65535 || (N + BN - 1) / BN > 65535) return false;
  const int m = static_cast<int>(M), n = static_cast<int>(N), k = static_cast<int>(K);
  return force_split_k() || gemm_us(fmt, f32 != 0, m, n, k, static_cast<int>(gs)) <= cuda_core_us(fmt, f32 != 0, m, n, k);
}

int opgemm_launch(int fmt, const void* x, const void* w, const void* scales, const float* biases, void* y, int64_t M, int64_t N,
                  int64_t K, int64_t gs, int f32, void* stream) {
  using namespace opg;
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
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (fmt) {
    case kAffine4: return launch_affine<kAffine4>(a, f32, st);
    case kAffine8: return launch_affine<kAffine8>(a, f32, st);
    case kMxfp4: return launch_f32<kMxfp4>(a, st);
    case kMxfp8: return launch_f32<kMxfp8>(a, st);
    default: return launch_f32<kNvfp4>(a, st);
  }
}

}  // namespace qmm
