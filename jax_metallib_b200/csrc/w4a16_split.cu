// int4 group-wise (g128, asymmetric) weight-only matmul at decode sizes (M <= 32), K split over a cluster.
//
//   y[M,N] = bf16( x[M,K] @ ((q[K,N] - z[K/128,N]) * s[K/128,N]) )
//
// The layout of the int8 kernel for few rows: persistent clusters of KS CTAs walk tiles of 128 columns, a ring of TMA
// stages (one 128-k group: 64 rows of 128 packed bytes, the group's activations, scales and zero points) runs on over
// the tiles, and warps of their own add the cluster's partial tiles over distributed shared memory in a fixed order.
//
// A consumer warp owns 32 columns and half of a group's k.  ldmatrix.trans hands it registers whose bytes are two packed
// rows of two neighbouring columns; a mask and one multiply-add per two weights make bf16 (q - z) * 2^-24 of them, exactly (no
// activation overflows in the product; the scale makes up for it).  Low nibbles (even k) fill slots 0-7 of
// mma.sync.m16n8k16, high nibbles slots 8-15, and the activations are paired to match.  Earlier, the codes went in as
// 16 + q and (16 + z) * sum x was taken off afterwards: what cancels there cost precision where activations do not
// average to zero (14336 x 4096, mean 1: 0.05 % of the results off by a rounding, 0.01 % now), and M = 16 took 21.2 us
// for 14336 x 4096, 18.2 us now.
//
// Bound by the latency of a stage's chain and, for small matrices, by prologue and
// hand-over, which this kernel has less of than the one that meets in global memory.  Measured (that kernel, this one) at
// M = 8: 4096 x 6144 11.7, 9.1 us; 4096 x 4096 11.2, 7.5 us; 14336 x 4096 19.6, 14.5 us; 4096 x 28672 23.7, 25.7 us.
// 17 to 32 rows are two tiles of 16, side by side in the walk: one tile of 32 has registers for one CTA per SM only (earlier:
// 4096 x 6144 31.5 us, now 19.9).
#include <cooperative_groups.h>

#include "split_k.cuh"

namespace cg = cooperative_groups;

namespace qmm {
namespace w4s {

using namespace split;

constexpr int kCols = 128;           // columns per tile
constexpr int kGroup = 128;          // k per stage
constexpr int kConsumerWarps = 8;    // 4 column groups of 32 x 2 halves of a stage's k
constexpr int kFirstReducer = kConsumerWarps + 1;
constexpr int kWBytes = kGroup / 2 * kCols;

template <int MT, bool ZP>
struct Smem {
  static constexpr int kXBox = MT * 8 * 128;               // [MT * 8 rows][64 k]
  static constexpr int kOffX = kWBytes;
  static constexpr int kOffS = kOffX + 2 * kXBox;          // 128 bf16 scales
  static constexpr int kOffZ = kOffS + 256;                // 128 zero points, or 64 bytes of two
  static constexpr int kZBytes = ZP ? 64 : 128;
  static constexpr int kStage = (kOffZ + 128 + 1023) / 1024 * 1024;
  static constexpr int kPerSm = 2;
  static constexpr int kReducers = 3;                      // warps that add the partial tiles
  static constexpr int kThreads = (kFirstReducer + kReducers) * 32;
  static constexpr int kStages = MT == 1 ? 8 : 6;
  static constexpr int kPartBufs = 2;             // tiles whose partial results may be in flight
  static constexpr int kPart = MT * 8 * kCols * 4;         // partial tile of one k half
  static constexpr int kOffPart = kStages * kStage;
  static constexpr int kOffBar = kOffPart + kPartBufs * 2 * kPart;
  static constexpr int kTotal = kOffBar + (2 * kStages + 2 * kPartBufs) * 8 + 1024;  // + alignment slack
  static_assert(kPerSm * (kTotal + 1024) <= 228 * 1024, "resident CTAs");
};

__device__ __forceinline__ void bulk_copy_g2s(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   dev::smem_u32(smem_dst)),
               "l"(reinterpret_cast<uint64_t>(gsrc)), "r"(bytes), "r"(dev::smem_u32(bar))
               : "memory");
}
// -z * 2^-24 as bf16, twice: z in the low byte of a bf16 reads as z * 2^-133 (a subnormal up to 127, the first binade above).
__device__ __forceinline__ uint32_t minus_zero_point(uint32_t z) {
  uint32_t r;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(z * 0x00010001u), "r"(0xF600F600u));   // * -2^109
  return r;
}
// The nibbles at bits SHIFT .. of w's halves -> (q - z) * 2^-24, exactly: q reads as q * 2^(SHIFT - 133) where it stands.
template <int SHIFT>
__device__ __forceinline__ uint32_t weights2(uint32_t w, uint32_t minus_z) {
  uint32_t r;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;"
      : "=r"(r)
      : "r"(w & (0x000F000Fu << SHIFT)), "r"(SHIFT ? 0x74007400u : 0x76007600u), "r"(minus_z));
  return r;
}

// TWO: 17 to 32 rows.  A tile's two halves of 16 rows are tiles of their own, next to each other in the walk (the second finds the
// weights in L2).
template <int MT, bool ZP, int TWO>
__global__ void __launch_bounds__(Smem<MT, ZP>::kThreads, Smem<MT, ZP>::kPerSm)
w4a16_split_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap,
                   const uint16_t* __restrict__ scales, const uint8_t* __restrict__ zeros, uint16_t* __restrict__ y, int M, int N,
                   int groups, int static_weights, int* status) {
  using L = Smem<MT, ZP>;
  constexpr int S = L::kStages, PB = L::kPartBufs;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
  uint64_t* empty = full + S;
  uint64_t* ready = empty + S;       // every CTA of the cluster has written its partial tile
  uint64_t* vacant = ready + PB;     // every CTA of the cluster has read this CTA's partial tile
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int KS = gridDim.x, rank = blockIdx.x;      // the cluster is the grid's x extent
  const int tiles = N / kCols << TWO;
  const int it_begin = (groups * rank) / KS, it_end = (groups * (rank + 1)) / KS;
  cg::cluster_group cluster = cg::this_cluster();

  dev::pdl_launch_dependents();
  if (threadIdx.x == 0) {
    dev::tma_prefetch_desc(&wmap);
    dev::tma_prefetch_desc(&xmap);
    for (int s = 0; s < S; ++s) {
      dev::mbar_init(&full[s], 2);   // the weights' copies and the activations' are announced apart
      dev::mbar_init(&empty[s], kConsumerWarps);
    }
    for (int b = 0; b < PB; ++b) {
      dev::mbar_init(&ready[b], KS * kConsumerWarps);
      dev::mbar_init(&vacant[b], KS * L::kReducers);
    }
    dev::fence_mbar_init();
  }
  cluster.sync();   // barriers of every CTA are initialised before a peer arrives on them

  if (warp == kConsumerWarps) {
    // ------------------------------ producer ------------------------------
    if (lane == 0) {
      const uint64_t policy = dev::policy_evict_first();
      auto issue_weights = [&](int s, int t, int it) {
        uint8_t* st = smem + s * L::kStage;
        const size_t col0 = static_cast<size_t>(t >> TWO) * kCols, row = static_cast<size_t>(it) * N;
        dev::mbar_expect_tx(&full[s], kWBytes + 256 + L::kZBytes);
        dev::tma_load_2d_hint(st, &wmap, &full[s], static_cast<int>(col0), it * (kGroup / 2), policy);
        bulk_copy_g2s(st + L::kOffS, scales + row + col0, 256, &full[s]);
        bulk_copy_g2s(st + L::kOffZ, ZP ? zeros + (row + col0) / 2 : zeros + row + col0, L::kZBytes, &full[s]);
      };
      // static weights do not depend on earlier kernels: the ring is filled before those have finished
      int ahead = 0;
      if (static_weights)
        for (int t = blockIdx.y; ahead < S && t < tiles; t += gridDim.y)
          for (int it = it_begin; ahead < S && it < it_end; ++it) issue_weights(ahead++, t, it);
      dev::pdl_wait();
      int n = 0;   // stages issued
      bool ok = true;
      for (int t = blockIdx.y; ok && t < tiles; t += gridDim.y)
        for (int it = it_begin; it < it_end; ++it, ++n) {
          const int s = n % S;
          if (n >= ahead) {
            if (!dev::mbar_wait_relaxed(&empty[s], ((n / S) & 1) ^ 1, status, 120)) { ok = false; break; }
            issue_weights(s, t, it);
          }
          uint8_t* st = smem + s * L::kStage;
          dev::mbar_expect_tx(&full[s], 2 * L::kXBox);   // rows past M arrive as zeros
          dev::tma_load_2d(st + L::kOffX, &xmap, &full[s], it * kGroup, (t & TWO) * 16);
          dev::tma_load_2d(st + L::kOffX + L::kXBox, &xmap, &full[s], it * kGroup + 64, (t & TWO) * 16);
        }
      // no copy may still be on its way into this CTA's shared memory when it leaves, whatever the consumers did
      for (int i = n > S ? n - S : 0; i < n; ++i)
        if (!dev::mbar_wait_relaxed(&full[i % S], (i / S) & 1, status, 121)) break;
    }
    __syncwarp();
  } else if (warp < kConsumerWarps) {
    // ------------------------------ consumers -----------------------------
    // The bounded waits for the ring begin when the activations can arrive: an earlier kernel may run for longer than they last.
    dev::pdl_wait();
    const int cgrp = warp & 3, kh = warp >> 2;
    const int g8 = lane >> 2, t4 = lane & 3;
    // weights: lane l addresses packed row 32 kh + l, 16-byte chunks 2 cgrp and 2 cgrp + 1 (XOR-swizzled by the row)
    const uint32_t w_row = (kh * 32 + lane) * 128;
    const uint32_t w_off0 = w_row + (((2 * cgrp) ^ (lane & 7)) << 4);
    const uint32_t w_off1 = w_row + (((2 * cgrp + 1) ^ (lane & 7)) << 4);
    // activations: box kh, row x_row, the four k 4 t4 .. of each 16-k step (the rows of a half-warp are all even or all odd:
    // no bank conflict)
    const int x_row = ((2 * g8) & 7) | (g8 >> 2);
    const uint32_t x_off = L::kOffX + kh * L::kXBox + x_row * 128 + ((t4 & 1) << 3);
    const int lc = cgrp * 32 + 2 * g8;   // first column of this thread's pair (second pair: + 16)
    const uint32_t ring = dev::smem_u32(smem);
    const int never = groups < 0;   // false, but not to the compiler
    int s = 0;
    uint32_t ph = 0;
    int tile = 0;
    bool ok = true;
    for (int t = blockIdx.y; t < tiles; t += gridDim.y, ++tile) {
      float acc[2][MT][4];
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[j][mt][i] = 0.f;
      for (int it = it_begin; it < it_end; ++it) {
        if (!dev::mbar_wait_relaxed_warp(&full[s], ph, status, 122)) { ok = false; break; }
        const uint32_t st = ring + s * L::kStage;
        uint32_t wr[2][4], xr[4][MT][2];
        ldmatrix_x4_trans(st + w_off0, wr[0]);
        ldmatrix_x4_trans(st + w_off1, wr[1]);
        uint32_t dep = wr[0][3] ^ wr[1][3];
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
            uint32_t lo, hi;   // (x0, x1), (x2, x3)
            asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];"
                         : "=r"(lo), "=r"(hi)
                         : "r"(st + x_off + mt * 1024 + (((2 * q + (t4 >> 1)) ^ x_row) << 4)));
            dep ^= hi;
            xr[q][mt][0] = __byte_perm(lo, hi, 0x5410);   // (x0, x2): the low nibbles of two packed rows
            xr[q][mt][1] = __byte_perm(lo, hi, 0x7632);   // (x1, x3): the high nibbles
          }
        // per-group constants of this thread's four columns: the scale, and -z * 2^-24 in bf16 twice
        float sc[2][2];
        uint32_t nz[2][2];
        const uint8_t* stp = smem + s * L::kStage;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint32_t s2 = *reinterpret_cast<const uint32_t*>(stp + L::kOffS + (lc + 16 * j) * 2);
          sc[j][0] = __uint_as_float(s2 << 16) * 16777216.f;
          sc[j][1] = __uint_as_float(s2 & 0xFFFF0000u) * 16777216.f;
          const uint32_t zb = ZP ? stp[L::kOffZ + (lc + 16 * j) / 2] : *reinterpret_cast<const uint16_t*>(stp + L::kOffZ + lc + 16 * j);
          nz[j][0] = minus_zero_point(ZP ? zb & 0xFu : zb & 0xFFu);
          nz[j][1] = minus_zero_point(ZP ? zb >> 4 : zb >> 8);
          dep ^= s2 ^ zb;
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float d[MT][4];
#pragma unroll
          for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int i = 0; i < 4; ++i) d[mt][i] = 0.f;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint32_t w = wr[j][q], w8 = w >> 8;
            // columns 2 g8 and 2 g8 + 1: even k, odd k
            const uint32_t a0 = weights2<0>(w, nz[j][0]), a2 = weights2<4>(w, nz[j][0]);
            const uint32_t a1 = weights2<0>(w8, nz[j][1]), a3 = weights2<4>(w8, nz[j][1]);
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) mma_bf16_16816(d[mt], a0, a1, a2, a3, xr[q][mt][0], xr[q][mt][1]);
          }
#pragma unroll
          for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[j][mt][i] = fmaf(sc[j][i >> 1], d[mt][i], acc[j][mt][i]);
        }
        release_slot(&empty[s], dep, never, lane);
        if (++s == S) { s = 0; ph ^= 1; }
      }
      if (!ok) break;
      // ---- hand the partial tile over to the reducers of the cluster
      const int b = tile % PB;
      if (tile >= PB && !wait_cluster_warp(&vacant[b], ((tile / PB) & 1) ^ 1, status, 123)) break;
      float* mine = reinterpret_cast<float*>(smem + L::kOffPart + (b * 2 + kh) * L::kPart);
      // accumulator columns 2 t4 and 2 t4 + 1 are rows 4 t4 (mod 8, + t4 / 2) and the one two further
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const int n = 2 * t4 + r, m = mt * 8 + (((2 * n) & 7) | (n >> 2));
            *reinterpret_cast<float2*>(mine + m * kCols + lc + j * 16) = make_float2(acc[j][mt][r], acc[j][mt][2 + r]);
          }
      __syncwarp();
      if (lane < KS) arrive_remote(&ready[b], lane);
    }
  } else {
    // ------------------------------ reducers ------------------------------
    // CTA `rank` adds every KS-th run of column pairs, in CTA order
    dev::pdl_wait();   // before anything is written to the output
    constexpr int kR = L::kReducers * 32;
    const int tid = threadIdx.x - kFirstReducer * 32;
    int tile = 0;
    for (int t = blockIdx.y; t < tiles; t += gridDim.y, ++tile) {
      const int b = tile % PB;
      const float* part = reinterpret_cast<const float*>(smem + L::kOffPart + b * 2 * L::kPart);
      if (!wait_cluster_warp(&ready[b], (tile / PB) & 1, status, 124)) break;
      const int first = (t & TWO) * 16, rows = min(M - first, MT * 8);
      for (int e = rank * kR + tid; e < rows * (kCols / 2); e += KS * kR) {
        const int m = e / (kCols / 2), c = (e % (kCols / 2)) * 2;
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
        *reinterpret_cast<uint32_t*>(y + static_cast<size_t>(first + m) * N + static_cast<size_t>(t >> TWO) * kCols + c) =
            dev::pack_bf16x2(v.x, v.y);
      }
      __syncwarp();
      if (lane < KS) arrive_remote(&vacant[b], lane);
    }
  }
  cluster.sync();   // peers keep their shared memory alive until it has been read
}

template <int MT, bool ZP, int TWO>
static int launch(const CUtensorMap& wmap, const CUtensorMap& xmap, const uint16_t* scales, const uint8_t* zeros, uint16_t* y, int M,
                  int N, int groups, int static_weights, int* status, cudaStream_t stream) {
  using L = Smem<MT, ZP>;
  static std::atomic<uint64_t> configured{0};  // per device (one mask per template instance)
  static std::atomic<int> resident[kMaxDevices][kMaxCluster + 1];
  auto kern = w4a16_split_kernel<MT, ZP, TWO>;
  if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), L::kTotal, configured)) return rc;
  const Grid g = choose_grid(N / kCols << TWO, groups,
                             [&](int ks) { return resident_clusters(kern, L::kThreads, L::kTotal, L::kPerSm, ks, resident); });
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  cfg.gridDim = dim3(g.ks, g.clusters);
  cfg.blockDim = dim3(L::kThreads);
  cfg.dynamicSmemBytes = L::kTotal;
  cfg.stream = stream;
  set_attrs(cfg, attr, g.ks);
  QMM_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, wmap, xmap, scales, zeros, y, M, N, groups, static_weights, status));
  return QMM_OK;
}

}  // namespace w4s

// 1 <= M <= 32, N and K multiples of 128, operands 16-byte aligned (checked by the caller).
int w4a16_split(const uint16_t* x, const uint8_t* wq, const uint16_t* scales, const uint8_t* zeros, int zeros_packed, uint16_t* y,
                int64_t M, int64_t N, int64_t K, int static_weights, int* status, cudaStream_t stream) {
  using namespace w4s;
  const int mt = M <= 8 ? 1 : 2;
  CUtensorMap wmap, xmap;
  if (int rc = make_tensor_map_2d(&wmap, wq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)(K / 2), (uint64_t)N, (uint64_t)N,
                                  kGroup / 2, kCols, CU_TENSOR_MAP_SWIZZLE_128B))
    return rc;
  if (int rc = make_tensor_map_2d(&xmap, x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)M, (uint64_t)K, (uint64_t)K * 2, mt * 8,
                                  64, CU_TENSOR_MAP_SWIZZLE_128B))
    return rc;
  const int m = static_cast<int>(M), n = static_cast<int>(N), g = static_cast<int>(K / kGroup);
#define QMM_W4S_LAUNCH(MT, TWO)                                                                               \
  (zeros_packed ? launch<MT, true, TWO>(wmap, xmap, scales, zeros, y, m, n, g, static_weights, status, stream) \
                : launch<MT, false, TWO>(wmap, xmap, scales, zeros, y, m, n, g, static_weights, status, stream))
  if (mt == 1) return QMM_W4S_LAUNCH(1, 0);
  if (m <= 16) return QMM_W4S_LAUNCH(2, 0);
  return QMM_W4S_LAUNCH(2, 1);
#undef QMM_W4S_LAUNCH
}

}  // namespace qmm
