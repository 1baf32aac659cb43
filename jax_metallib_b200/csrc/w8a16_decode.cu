// int8 per-channel weight-only matmul at few rows (sm_100a).
//
//   y[M,N] = bf16( (x[M,K] @ float(w[K,N])) * scale[N] )        x bf16, w int8 row-major, scale f32
//
// and the same with f32 activations and results (any M; three bf16 terms per activation, see split4).
// Measured at M = 1: 4096 x 28672 25 us (4.7 TB/s), 4096 x 6144 8.0 us, 14336 x 4096 14.0 us, the four linears of a layer
// 57 us (one thread per column before: 1905 us); f32, 32 x 1024 x 1024 10.1 -> 6.7 us, 256 x 4096 x 4096 528 -> 140 us.
//
// Bound by HBM: the weights (K*N bytes) are read once.  A cluster of KS CTAs owns blocks of 128
// columns and splits K between its CTAs; every CTA runs a ring of TMA stages (64 k x 128 columns of
// weights, 128-byte swizzle, and the same 64 k of the activations), fed by one warp and drained by
// eight; the ring runs on over the cluster's column blocks, so that the loads of a block overlap the
// hand-over of the one before.  A consumer warp owns 32 columns and half of a stage's k:
// ldmatrix.trans hands it registers with two k of two neighbouring columns, which become two bf16
// pairs by a logic operation and an exact multiply-add each, and mma.sync.m16n8k16 (f32 accumulate) takes
// the weights as its 16-row operand and the activations as its 8-column operand, so that M = 1
// wastes tensor work, which is free here, and not memory traffic.  tcgen05 has nothing to add at
// these sizes: its operand would have to pass through shared memory a second time after the
// conversion.  What is left above the weights' own time is the fill of the ring, the hand-over at the
// end of a tile and, at M = 32, the MMAs.
//
// The partial tiles of a cluster (KS CTAs x two k halves) meet in distributed shared memory; warps
// of their own add each CTA's share of the elements in a fixed order while the consumers go on with
// the next block: deterministic, no workspace, no atomics.
#include <cooperative_groups.h>

#include "split_k.cuh"

namespace cg = cooperative_groups;

namespace qmm {
namespace w8d {

using namespace split;

constexpr int kCols = 128;           // columns per tile
constexpr int kBK = 64;              // k per stage
constexpr int kConsumerWarps = 8;    // 4 column groups of 32 x 2 halves of a stage's k
constexpr int kFirstReducer = kConsumerWarps + 1;
constexpr int kWBytes = kBK * kCols;

template <int MT, bool XF32>
struct Smem {
  static constexpr int kXBox = MT * 8 * 128;               // [MT * 8 rows][128 bytes]: 64 k of bf16 or 32 k of f32
  static constexpr int kX = XF32 ? 2 * kXBox : kXBox;      // activations of a stage
  static constexpr int kStage = kWBytes + kX;
  // resident CTAs: a warp's chain ldmatrix -> convert -> MMA is latency-bound, so as many as registers allow
  static constexpr int kPerSm = 2;
  static constexpr int kReducers = MT <= 2 ? 3 : 4;                     // warps that add the partial tiles
  static constexpr int kThreads = (kFirstReducer + kReducers) * 32;
  static constexpr int kStages = MT == 1 ? 8 : 6;
  static constexpr int kPartBufs = MT <= 2 ? 2 : 1;        // tiles whose partial results may be in flight
  static constexpr int kPart = MT * 8 * kCols * 4;         // partial tile of one k half
  static constexpr int kOffPart = kStages * kStage;
  static constexpr int kOffBar = kOffPart + kPartBufs * 2 * kPart;
  static constexpr int kTotal = kOffBar + (2 * kStages + 2 * kPartBufs) * 8 + 1024;  // + alignment slack
  static_assert(kPerSm * (kTotal + 1024) <= 228 * 1024, "resident CTAs");
};

__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
// The int8 values v in bytes 0 and 2 of a register -> two bf16 v / 64, exactly, in two instructions: v + 128 in the
// low byte of a bf16 reads as (v + 128) * 2^-133 (a subnormal up to 127, the first binade above), and one fused
// multiply-add brings it to (v + 128) / 64 - 2.  The factor 64 goes back in with the channel's scale.
__device__ __forceinline__ uint32_t bytes02_to_bf16x2(uint32_t t) {
  uint32_t u, r;
  asm("lop3.b32 %0, %1, %2, %3, 0x6A;" : "=r"(u) : "r"(t), "r"(0x00FF00FFu), "r"(0x00800080u));  // (t & m) ^ k
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(u), "r"(0x7F007F00u), "r"(0xC000C000u));   // * 2^127 - 2
  return r;
}

// Four f32 -> their bf16 terms, as pairs of k: the top 8 significant bits, the next 8, the rest.  Where the three do not
// hold a value, its third term has bits below them: 16 low bits of `rest` are not all zero.  That is an infinity or NaN
// (whose difference to itself is the NaN 0x7FFFFFFF), or a value whose last bits lie below bf16's smallest (2^-133, so
// |x| < 2^-110).
__device__ __forceinline__ void split4(const uint32_t (&v)[4], uint32_t (&hi)[2], uint32_t (&mid)[2], uint32_t (&lo)[2],
                                       uint32_t& rest) {
  uint32_t m[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m[i] = __float_as_uint(__uint_as_float(v[i]) - __uint_as_float(v[i] & 0xFFFF0000u));
    l[i] = __float_as_uint(__uint_as_float(m[i]) - __uint_as_float(m[i] & 0xFFFF0000u));
    rest |= l[i];
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    hi[i] = __byte_perm(v[2 * i], v[2 * i + 1], 0x7632);
    mid[i] = __byte_perm(m[2 * i], m[2 * i + 1], 0x7632);
    lo[i] = __byte_perm(l[2 * i], l[2 * i + 1], 0x7632);
  }
}
// Two registers of ldmatrix -> the MMA's weight operand for 16 k.
__device__ __forceinline__ void weights4(uint32_t w0, uint32_t w1, uint32_t (&a)[4]) {
  a[0] = bytes02_to_bf16x2(w0);
  a[1] = bytes02_to_bf16x2(w0 >> 8);
  a[2] = bytes02_to_bf16x2(w1);
  a[3] = bytes02_to_bf16x2(w1 >> 8);
}
__device__ __forceinline__ void lds_v4(uint32_t addr, uint32_t (&v)[4]) {
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr));
}
// The sums over a stage's 32 k, 16 columns x 8 rows, where split4 does not hold every value: what it does not hold goes
// into a second sum, times 2^64 (an infinity or NaN as it is).  A call, so that its registers do not count elsewhere.
__device__ __noinline__ float4 awkward_tile(uint32_t w_addr, uint32_t x_addr, int t4, int x_row) {
  uint32_t wr[4];
  ldmatrix_x4_trans(w_addr, wr);
  float d[2][4] = {};
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    uint32_t v[2][4], a[4];
    lds_v4(x_addr + (((q * 4 + t4) ^ x_row) << 4), v[0]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float x = __uint_as_float(v[0][i]), m = x - __uint_as_float(v[0][i] & 0xFFFF0000u);
      const float l = m - __uint_as_float(__float_as_uint(m) & 0xFFFF0000u);
      const bool held = (__float_as_uint(l) & 0xFFFFu) == 0u;
      v[1][i] = held ? 0u : __float_as_uint(x * 18446744073709551616.f);
      if (!held) v[0][i] = 0u;
      if ((v[1][i] & 0x7FFFFFFFu) > 0x7F800000u) v[1][i] |= 0x00400000u;   // stays a NaN when it is cut
    }
    weights4(wr[2 * q], wr[2 * q + 1], a);
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      uint32_t hi[2], mid[2], lo[2], unused = 0;
      split4(v[s], hi, mid, lo, unused);
#pragma unroll
      for (int i = 0; i < 2; ++i) {   // an infinity or NaN is its first term alone
        if ((hi[i] & 0x7F80u) == 0x7F80u) mid[i] &= 0xFFFF0000u, lo[i] &= 0xFFFF0000u;
        if ((hi[i] & 0x7F800000u) == 0x7F800000u) mid[i] &= 0xFFFFu, lo[i] &= 0xFFFFu;
      }
      mma_bf16_16816(d[s], a[0], a[1], a[2], a[3], lo[0], lo[1]);
      mma_bf16_16816(d[s], a[0], a[1], a[2], a[3], mid[0], mid[1]);
      mma_bf16_16816(d[s], a[0], a[1], a[2], a[3], hi[0], hi[1]);
    }
  }
  constexpr float kSmall = 3.469446951953614e-18f;   // 2^-64, and 64 of the weights
  return make_float4(fmaf(d[1][0], kSmall, d[0][0] * 64.f), fmaf(d[1][1], kSmall, d[0][1] * 64.f),
                     fmaf(d[1][2], kSmall, d[0][2] * 64.f), fmaf(d[1][3], kSmall, d[0][3] * 64.f));
}

// LONG: the tensor core cuts its sums off, so that a correctly rounded sum takes over every kLongSlice stages of a long slice
// of K.  That is for a K of 16384 and more with columns for few CTAs to a cluster, and few rows, where registers are left
// (28672 x 8192 at M = 1: 0.12 % of the results off by a rounding, 0.02 % with it; 43.5, 45.4 us).
constexpr int kLongSlice = 16;
template <int MT, bool XF32, bool LONG>
__global__ void __launch_bounds__(Smem<MT, XF32>::kThreads, Smem<MT, XF32>::kPerSm)
w8_decode_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap,
                 const float* __restrict__ scale, void* __restrict__ y, int M, int N, long long ldy, int stages_total,
                 int independent, int* status) {
  using L = Smem<MT, XF32>;
  constexpr int S = L::kStages, PB = L::kPartBufs;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
  uint64_t* empty = full + S;
  uint64_t* ready = empty + S;       // every CTA of the cluster has written its partial tile
  uint64_t* vacant = ready + PB;     // every CTA of the cluster has read this CTA's partial tile
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int KS = gridDim.x, rank = blockIdx.x;      // the cluster is the grid's x extent
  // tile t: rows (t % row_tiles) * MT * 8 .. of column block t / row_tiles
  const int row_tiles = (M + MT * 8 - 1) / (MT * 8);
  const int tiles = ((N + kCols - 1) / kCols) * row_tiles;
  const int it_begin = (stages_total * rank) / KS, it_end = (stages_total * (rank + 1)) / KS;
  cg::cluster_group cluster = cg::this_cluster();

  if (independent) dev::pdl_launch_dependents();
  if (threadIdx.x == 0) {
    dev::tma_prefetch_desc(&wmap);
    dev::tma_prefetch_desc(&xmap);
    for (int s = 0; s < S; ++s) {
      dev::mbar_init(&full[s], 1);
      dev::mbar_init(&empty[s], kConsumerWarps);
    }
    for (int b = 0; b < PB; ++b) {
      dev::mbar_init(&ready[b], KS * kConsumerWarps);
      dev::mbar_init(&vacant[b], KS * L::kReducers);
    }
    dev::fence_mbar_init();
  }
  cluster.sync();   // barriers of every CTA are initialised before a peer arrives on them
  if (!independent) {
    dev::pdl_wait();
    dev::pdl_launch_dependents();
  }

  if (warp == kConsumerWarps) {
    // ------------------------------ producer ------------------------------
    if (lane == 0) {
      const uint64_t policy = dev::policy_evict_first();
      int n = 0;   // stages issued
      bool ok = true;
      for (int t = blockIdx.y; ok && t < tiles; t += gridDim.y) {
        const int col0 = (t / row_tiles) * kCols, row0 = (t % row_tiles) * MT * 8;
        for (int it = it_begin; it < it_end; ++it, ++n) {
          const int s = n % S;
          if (!dev::mbar_wait_relaxed(&empty[s], ((n / S) & 1) ^ 1, status, 80)) { ok = false; break; }
          uint8_t* st = smem + s * L::kStage;
          dev::mbar_expect_tx(&full[s], L::kStage);   // rows and columns past the ends arrive as zeros
          if (row_tiles == 1) dev::tma_load_2d_hint(st, &wmap, &full[s], col0, it * kBK, policy);
          else dev::tma_load_2d(st, &wmap, &full[s], col0, it * kBK);   // the next row tile reads them again
          dev::tma_load_2d(st + kWBytes, &xmap, &full[s], it * kBK, row0);
          if (XF32) dev::tma_load_2d(st + kWBytes + L::kXBox, &xmap, &full[s], it * kBK + 32, row0);
        }
      }
      // no copy may still be on its way into this CTA's shared memory when it leaves, whatever the consumers did
      for (int i = n > S ? n - S : 0; i < n; ++i)
        if (!dev::mbar_wait_relaxed(&full[i % S], (i / S) & 1, status, 81)) break;
    }
    __syncwarp();
  } else if (warp < kConsumerWarps) {
    // ------------------------------ consumers -----------------------------
    const int cgrp = warp & 3, kh = warp >> 2;
    const int g8 = lane >> 2, t4 = lane & 3;
    // weights: lane l addresses one k row, 16-byte chunks 2 cgrp and 2 cgrp + 1 (XOR-swizzled by the row).  bf16
    // activations: row 32 kh + l.  f32 activations: a thread reads four neighbouring k of a row (16 bytes) per 16-k
    // step, so slots 2t, 2t + 1, 2t + 8, 2t + 9 of a step stand for its k 4t .. 4t + 3 and the rows are dealt likewise.
    const int w_k = kh * 32 + (XF32 ? (lane >> 4) * 16 + ((lane & 7) >> 1) * 4 + (lane & 1) + ((lane >> 3) & 1) * 2 : lane);
    const uint32_t w_off0 = w_k * 128 + (((2 * cgrp) ^ (w_k & 7)) << 4);
    const uint32_t w_off1 = w_k * 128 + (((2 * cgrp + 1) ^ (w_k & 7)) << 4);
    // activations: bf16: lane l addresses row l & 7 of the 8-k chunk 4 kh + (l >> 3); f32: row x_row, chunk t4 of the
    // step (rows r and r + 4 share a quarter-warp: no bank conflict)
    const int x_row = XF32 ? ((g8 >> 1) | ((g8 & 1) << 2)) : (lane & 7);
    const uint32_t x_off = kWBytes + (XF32 ? kh * L::kXBox : 0) + x_row * 128 +
                           (XF32 ? 0 : (((4 * kh + (lane >> 3)) ^ x_row) << 4));
    const uint32_t ring = dev::smem_u32(smem);
    int s = 0;
    uint32_t ph = 0;
    int tile = 0;
    bool ok = true;
    const int never = stages_total < 0;   // false, but not to the compiler
    for (int t = blockIdx.y; t < tiles; t += gridDim.y, ++tile) {
      float acc[2][MT][4];
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[j][mt][i] = 0.f;
      [[maybe_unused]] float total[2][MT][4] = {};   // LONG
      for (int it = it_begin, end = LONG ? min(it_begin + kLongSlice, it_end) : it_end; it < end; ++it) {
        if (!dev::mbar_wait_relaxed_warp(&full[s], ph, status, 82)) { ok = false; break; }
        const uint32_t st = ring + s * L::kStage;
        uint32_t dep;
        if constexpr (!XF32) {
          uint32_t wr[2][4], xr[MT][4];
          ldmatrix_x4_trans(st + w_off0, wr[0]);
          ldmatrix_x4_trans(st + w_off1, wr[1]);
          dep = wr[0][3] ^ wr[1][3];
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) ldmatrix_x4(st + x_off + mt * 1024, xr[mt]);
#pragma unroll
          for (int q = 0; q < 2; ++q)   // 16 k each
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              uint32_t a[4];
              weights4(wr[j][2 * q], wr[j][2 * q + 1], a);
#pragma unroll
              for (int mt = 0; mt < MT; ++mt) mma_bf16_16816(acc[j][mt], a[0], a[1], a[2], a[3], xr[mt][2 * q], xr[mt][2 * q + 1]);
            }
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) dep ^= xr[mt][3];
        } else {
          // x = hi + mid + lo, bf16 each and exact together; the smallest terms are added first, into an accumulator
          // that starts at zero every stage: a correctly rounded f32 addition takes over after 32 k
          uint32_t wr[2][4];
          ldmatrix_x4_trans(st + w_off0, wr[0]);
          ldmatrix_x4_trans(st + w_off1, wr[1]);
          dep = wr[0][3] ^ wr[1][3];
          uint32_t term[3][2][MT][2], rest = 0;   // [hi, mid, lo][16-k step][row tile][k pair]
#pragma unroll
          for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
              uint32_t v[4];
              lds_v4(st + x_off + mt * 1024 + (((q * 4 + t4) ^ x_row) << 4), v);
              dep ^= v[3];
              split4(v, term[0][q][mt], term[1][q][mt], term[2][q][mt], rest);
            }
          if (!__any_sync(0xFFFFFFFFu, rest & 0xFFFFu)) {
            float d[2][MT][4];
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
              for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int i = 0; i < 4; ++i) d[j][mt][i] = 0.f;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              uint32_t a[2][4];
#pragma unroll
              for (int q = 0; q < 2; ++q) weights4(wr[j][2 * q], wr[j][2 * q + 1], a[q]);
#pragma unroll
              for (int e = 2; e >= 0; --e)
#pragma unroll
                for (int q = 0; q < 2; ++q)
#pragma unroll
                  for (int mt = 0; mt < MT; ++mt)
                    mma_bf16_16816(d[j][mt], a[q][0], a[q][1], a[q][2], a[q][3], term[e][q][mt][0], term[e][q][mt][1]);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
              for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[j][mt][i] = fmaf(d[j][mt][i], 64.f, acc[j][mt][i]);
          } else {
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
              for (int mt = 0; mt < MT; ++mt) {
                const float4 e = awkward_tile(st + (j ? w_off1 : w_off0), st + x_off + mt * 1024, t4, x_row);
                acc[j][mt][0] += e.x;
                acc[j][mt][1] += e.y;
                acc[j][mt][2] += e.z;
                acc[j][mt][3] += e.w;
                dep ^= __float_as_uint(e.x);
              }
          }
        }
        release_slot(&empty[s], dep, never, lane);
        if (++s == S) { s = 0; ph ^= 1; }
        if constexpr (LONG)
          if (it + 1 == end) {
            end = min(end + kLongSlice, it_end);
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
              for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  total[j][mt][i] += acc[j][mt][i];
                  acc[j][mt][i] = it + 1 < end ? 0.f : total[j][mt][i];
                }
          }
      }
      if (!ok) break;
      // ---- hand the partial tile over to the reducers of the cluster
      const int b = tile % PB;
      if (tile >= PB && !wait_cluster_warp(&vacant[b], ((tile / PB) & 1) ^ 1, status, 83)) break;
      float* part = reinterpret_cast<float*>(smem + L::kOffPart + b * 2 * L::kPart);
      float* mine = part + kh * (L::kPart / 4);
      // rows 2 t4, 2 t4 + 1 (f32: t4, t4 + 4) of columns 2 g8, 2 g8 + 1 of each 16-column block
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int r = 0; r < 2; ++r)
            *reinterpret_cast<float2*>(mine + (mt * 8 + (XF32 ? t4 + 4 * r : 2 * t4 + r)) * kCols + cgrp * 32 + j * 16 + 2 * g8) =
                make_float2(acc[j][mt][r], acc[j][mt][2 + r]);
      __syncwarp();
      if (lane < KS) arrive_remote(&ready[b], lane);
    }
  } else {
    // ------------------------------ reducers ------------------------------
    // CTA `rank` adds every KS-th run of column pairs, in CTA order
    constexpr int kR = L::kReducers * 32;
    const int tid = threadIdx.x - kFirstReducer * 32;
    int tile = 0;
    for (int t = blockIdx.y; t < tiles; t += gridDim.y, ++tile) {
      const int b = tile % PB;
      const float* part = reinterpret_cast<const float*>(smem + L::kOffPart + b * 2 * L::kPart);
      if (!wait_cluster_warp(&ready[b], (tile / PB) & 1, status, 84)) break;
      const int col0 = (t / row_tiles) * kCols, row0 = (t % row_tiles) * MT * 8;
      const int rows = min(MT * 8, M - row0);
      for (int e = rank * kR + tid; e < rows * (kCols / 2); e += KS * kR) {
        const int m = e / (kCols / 2), c = (e % (kCols / 2)) * 2;
        if (col0 + c >= N) continue;
        float2 lo[kMaxCluster], hi[kMaxCluster];
#pragma unroll
        for (int r = 0; r < kMaxCluster; ++r)
          if (r < KS) {
            const float* p = cluster.map_shared_rank(part, r) + m * kCols + c;
            lo[r] = *reinterpret_cast<const float2*>(p);
            hi[r] = *reinterpret_cast<const float2*>(p + L::kPart / 4);
          }
        float2 v = make_float2(0.f, 0.f);
#pragma unroll
        for (int r = 0; r < kMaxCluster; ++r)
          if (r < KS) {
            v.x += lo[r].x + hi[r].x;
            v.y += lo[r].y + hi[r].y;
          }
        const float2 sc = make_float2(__ldg(scale + col0 + c), __ldg(scale + col0 + c + 1));
        const size_t i = static_cast<size_t>(row0 + m) * ldy + col0 + c;
        v.x = XF32 ? v.x * sc.x : v.x * 64.f * sc.x;
        v.y = XF32 ? v.y * sc.y : v.y * 64.f * sc.y;
        if (XF32) *reinterpret_cast<float2*>(static_cast<float*>(y) + i) = v;
        else *reinterpret_cast<uint32_t*>(static_cast<uint16_t*>(y) + i) = dev::pack_bf16x2(v.x, v.y);
      }
      __syncwarp();
      if (lane < KS) arrive_remote(&vacant[b], lane);
    }
  }
  cluster.sync();   // peers keep their shared memory alive until it has been read
}

template <int MT, bool XF32>
static int launch(const CUtensorMap& wmap, const CUtensorMap& xmap, const float* scale, void* y, int M, int N, long long ldy,
                  int stages_total, int independent, cudaStream_t stream) {
  using L = Smem<MT, XF32>;
  static std::atomic<uint64_t> configured{0};  // per device (one mask per template instance)
  static std::atomic<int> resident[kMaxDevices][kMaxCluster + 1];
  auto kern = w8_decode_kernel<MT, XF32, false>;
  if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), L::kTotal, configured)) return rc;
  const Grid g = choose_grid(((N + kCols - 1) / kCols) * ((M + MT * 8 - 1) / (MT * 8)), stages_total, [&](int ks) {
    return resident_clusters(kern, L::kThreads, L::kTotal, L::kPerSm, ks, resident);
  });
  if constexpr (MT == 1 && !XF32)
    if (stages_total > 4 * kLongSlice * g.ks) {
      static std::atomic<uint64_t> configured_long{0};
      kern = w8_decode_kernel<MT, XF32, true>;
      if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), L::kTotal, configured_long)) return rc;
    }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  cfg.gridDim = dim3(g.ks, g.clusters);
  cfg.blockDim = dim3(Smem<MT, XF32>::kThreads);
  cfg.dynamicSmemBytes = L::kTotal;
  cfg.stream = stream;
  set_attrs(cfg, attr, g.ks);
  QMM_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, wmap, xmap, scale, y, M, N, ldy, stages_total, independent, device_status_word()));
  return QMM_OK;
}

}  // namespace w8d

// M <= 32; K % 8 == 0, N % 16 == 0, x and w 16-byte, y 4-byte aligned, ldy even (checked by the caller).
int w8a16_decode(const uint16_t* x, const int8_t* w, const float* scale, uint16_t* y, int64_t M, int64_t N, int64_t K, int64_t ldy,
                 uint32_t flags, cudaStream_t stream) {
  using namespace w8d;
  const int mt = M <= 8 ? 1 : (M <= 16 ? 2 : 4);
  CUtensorMap wmap, xmap;
  if (int rc = make_tensor_map_2d(&wmap, w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)K, (uint64_t)N, (uint64_t)N, kBK, kCols,
                                  CU_TENSOR_MAP_SWIZZLE_128B))
    return rc;
  if (int rc = make_tensor_map_2d(&xmap, x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)M, (uint64_t)K, (uint64_t)K * 2, mt * 8,
                                  kBK, CU_TENSOR_MAP_SWIZZLE_128B))
    return rc;
  const int stages_total = static_cast<int>((K + kBK - 1) / kBK);
  const int ind = (flags & QMM_GEMM_INDEPENDENT) ? 1 : 0;
  const int m = static_cast<int>(M), n = static_cast<int>(N);
  if (mt == 1) return launch<1, false>(wmap, xmap, scale, y, m, n, ldy, stages_total, ind, stream);
  if (mt == 2) return launch<2, false>(wmap, xmap, scale, y, m, n, ldy, stages_total, ind, stream);
  return launch<4, false>(wmap, xmap, scale, y, m, n, ldy, stages_total, ind, stream);
}

// Any M; K % 4 == 0, N % 16 == 0, x and w 16-byte, y 8-byte aligned (checked by the caller).  Row tiles of 8 or 16: the
// three terms of the activations and two sets of accumulators fill the registers.
int w8a32_tc(const float* x, const int8_t* w, const float* scale, float* y, int64_t M, int64_t N, int64_t K, cudaStream_t stream) {
  using namespace w8d;
  const int mt = M <= 8 ? 1 : 2;
  CUtensorMap wmap, xmap;
  if (int rc = make_tensor_map_2d(&wmap, w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)K, (uint64_t)N, (uint64_t)N, kBK, kCols,
                                  CU_TENSOR_MAP_SWIZZLE_128B))
    return rc;
  if (int rc = make_tensor_map_2d(&xmap, x, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (uint64_t)M, (uint64_t)K, (uint64_t)K * 4, mt * 8,
                                  32, CU_TENSOR_MAP_SWIZZLE_128B))
    return rc;
  const int stages_total = static_cast<int>((K + kBK - 1) / kBK);
  const int m = static_cast<int>(M), n = static_cast<int>(N);
  return mt == 1 ? launch<1, true>(wmap, xmap, scale, y, m, n, n, stages_total, 0, stream)
                 : launch<2, true>(wmap, xmap, scale, y, m, n, n, stages_total, 0, stream);
}

}  // namespace qmm
