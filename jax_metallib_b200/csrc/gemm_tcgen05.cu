// tcgen05 / TMEM GEMMs for the prefill-sized quantized matmuls (sm_100a).
//
// Both kernels keep one persistent CTA per SM that walks output tiles, feed
// shared memory with TMA (128-byte swizzle), accumulate in all 512 TMEM columns
// (two 256-column accumulators, one MMA-issuing thread each: a single thread
// cannot issue tcgen05.mma fast enough to keep the tensor pipe busy) and drain
// the accumulators with tcgen05.ld into a fused epilogue.  Every wait is bounded.
//
//  (1) i8gemm: acc[M,N] = a[M,K] . b[K,N], int8/uint8 operands, int32
//      accumulate (kind::i8, exact).  a is K-major, b is consumed N-major
//      straight from its row-major [K,N] layout (MN-major descriptor), so no
//      transposed copy of b is ever made.  Tile 256 (m, two accumulators) x
//      256 (n) x 128 (k).  Warps: one TMA producer, two MMA issuers, eight
//      epilogue warps (optional int32 store and/or float(acc) * row[m] * col[n]).
//      Where the tiles are few, a cluster of up to eight CTAs takes a 128 x 256 block, each a share of its K, and adds the
//      accumulators up over distributed shared memory: M = 64, 4096 x 4096 18.3 us in one CTA to a block, 9.7 now; 8192 x 8192
//      30, 14; M = 512, 8192 x 1024 30, 14.
//
//  (2) w8a16: y[M,N] = bf16((x[M,K] @ float(w[K,N])) * scale[N]), bf16
//      activations, int8 weights.  The weight tile is the 128-row MMA operand and goes
//      into it through TMEM, the activation tile (up to 192 rows) is the other one; a CTA
//      runs two weight blocks against one activation tile (256 channels x 192 rows).
//      With the converted weights in shared memory (written, and read by the MMA) a 64-k
//      stage of 256 x 256 moved 192 KB there in 1024 clocks of MMA, at 128 bytes a clock:
//      0.66 of the MMA rate, as measured; now 104 KB in 768 clocks.  Warps: a TMA
//      producer for activations, one for raw int8 weights, two MMA issuers and
//      16 worker warps in two groups that take every other 64-k stage: a
//      group reads the raw tile (ldmatrix.trans pairs the k of a channel), converts it to
//      bf16 (exactly) and stores it to TMEM; when a tile's stages are done the same warps
//      drain its accumulators.  The accumulator holds the transposed tile
//      (lane = output channel), so the per-channel scale is one register per
//      thread.  Leftover tiles of the last round are cut into halves or
//      quarters.  Where the tiles are few, a cluster of up to eight CTAs takes one, each a share of its K, and adds the
//      accumulators up over distributed shared memory: M = 64, int8 4096 x 4096 29.6 us in one CTA to a tile, 14.3 now;
//      14336 x 4096 89, 25.5; int4 14336 x 2048 112, 26.6; M = 320, 8192 x 8192 59, 44.  The output may be stored with
//      multimem.st to a multicast address (one store reaches the same offset of every rank's buffer: the all-gather of a
//      column-sharded linear happens in the epilogue), and the launch can signal its completion to every rank.
#include <cstdlib>

#include "split_k.cuh"

namespace qmm {
namespace tc {

constexpr uint32_t kSwizzle128 = 2;  // UMMA layout type of the 128-byte swizzle

// ============================================================================
// (1) int8 x int8 -> int32
// ============================================================================
namespace i8 {
constexpr int BMB = 128;            // rows per MMA (its M); a full tile has two such blocks
constexpr int BN = 256, BK = 128;
constexpr int kStages = 3;
constexpr int kABlock = BMB * BK;      // 16 KB: [128 rows][128 k]
constexpr int kABytes = 2 * kABlock;   // 32 KB: both row blocks
constexpr int kBBytes = BK * BN;       // 32 KB: two [128 k][128 n] column blocks
constexpr int kStageBytes = kABytes + kBBytes;  // 64 KB
constexpr int kEpiWarpsI = 8;
// Warp roles: 0 TMA, 1 MMA issue for row block 0, 2-9 epilogue, 10 MMA issue for row block 1.
constexpr int kSecondMmaWarp = 2 + kEpiWarpsI;
constexpr int kThreads = (kSecondMmaWarp + 1) * 32;
// One 32 x 32 chunk of 4-byte results per epilogue warp, 128-byte swizzled, for the TMA stores of a CTA's last
// item.  It lies in the first stage of the operand ring, which is idle by then; shared memory of its own would
// take the CTA past 196 KB, into the SM's largest shared-memory split, for 32 KB that the ring already has.
constexpr int kOutStage = 32 * 128;
constexpr int kOutBase = 0;
static_assert(kEpiWarpsI * kOutStage <= kStageBytes, "the result chunks must fit in one stage of the ring");
constexpr int kSmemBytes = kStages * kStageBytes + 1024 /*barriers*/ + 1024 /*alignment*/;
static_assert(BK == 128, "the issue loop is written out for four 32-byte k-steps");

// Item i of this CTA.  A tile is 256 rows x 256 columns: two row blocks against
// one column tile (a 128 x 256 tile needs 94 bytes per clock and SM from L2 at
// the int8 MMA rate, more than L2 delivers to all SMs at once; sharing the
// column tile between two accumulators needs 63).  When whole tiles would leave
// half of the SMs idle, row blocks are dealt out singly.
struct Work {
  int tm2, tn, h0, nh;
};
template <bool SPLIT>
__device__ __forceinline__ bool get_work(int i, int tiles_m2, int tiles_n, int halves, int M, Work& w) {
  if (SPLIT) {   // one row block to a cluster
    const int blocks_m = (M + BMB - 1) / BMB, bm = blockIdx.y % blocks_m;
    w.tm2 = bm >> 1;
    w.tn = blockIdx.y / blocks_m;
    w.h0 = bm & 1;
    w.nh = 1;
    return i == 0;
  }
  const int v = blockIdx.x + i * gridDim.x;
  const int total = tiles_m2 * tiles_n * (halves ? 2 : 1);
  if (v >= total) return false;
  const int tile = halves ? (v >> 1) : v;
  w.tm2 = tile % tiles_m2;
  w.tn = tile / tiles_m2;
  w.h0 = halves ? (v & 1) : 0;
  w.nh = halves ? 1 : 2;
  const int blocks_left = (M - w.tm2 * 2 * BMB + BMB - 1) / BMB - w.h0;
  w.nh = max(0, min(w.nh, blocks_left));
  return true;
}

// SPLIT (with halves): a row block is one cluster's; its CTAs take a share of K each and add their accumulators up over
// distributed shared memory.  One block a cluster, so that the ring is free for the sums when the last MMA has retired.
template <bool SPLIT>
__global__ void __launch_bounds__(kThreads, 1)
i8gemm_kernel(const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap bmap,
              const __grid_constant__ CUtensorMap accmap, const __grid_constant__ CUtensorMap outmap,
              int32_t* __restrict__ acc_out, float* __restrict__ f_out,
              const float* __restrict__ row_scale, const float* __restrict__ col_scale, int M, int N,
              int K, uint32_t idesc, int halves, int staged_store, int* status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * kStageBytes);
  uint64_t* empty = full + kStages;    // count 2: one commit per issuing thread
  uint64_t* tfull = empty + kStages;   // accumulators ready for the epilogue (count 2)
  uint64_t* tempty = tfull + 1;        // accumulators drained
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_m2 = (M + 2 * BMB - 1) / (2 * BMB), tiles_n = (N + BN - 1) / BN;
  const int all_kblocks = (K + BK - 1) / BK;
  const int kb_begin = SPLIT ? static_cast<int>(static_cast<long long>(all_kblocks) * blockIdx.x / gridDim.x) : 0;
  const int kb_end = SPLIT ? static_cast<int>(static_cast<long long>(all_kblocks) * (blockIdx.x + 1) / gridDim.x) : all_kblocks;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      dev::mbar_init(&full[s], 1);
      dev::mbar_init(&empty[s], 2);
    }
    dev::mbar_init(tfull, 2);
    dev::mbar_init(tempty, kEpiWarpsI);
    dev::fence_mbar_init();
  }
  if (warp == 1) {
    dev::tmem_alloc(tmem_slot, 512);
    dev::tmem_relinquish();
  }
  dev::tc_fence_before();
  __syncthreads();
  dev::tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);

  if (warp == 0) {
    // ------------------------------ TMA producer ---------------------------
    if (lane == 0) {
      dev::tma_prefetch_desc(&amap);
      dev::tma_prefetch_desc(&bmap);
      uint32_t s = 0, ph = 0;
      bool ok = true;
      Work w;
      for (int i = 0; ok && get_work<SPLIT>(i, tiles_m2, tiles_n, halves, M, w); ++i) {
        if (w.nh == 0) continue;
        for (int kb = kb_begin; kb < kb_end; ++kb) {
          if (!dev::mbar_wait(&empty[s], ph ^ 1, status, 11)) { ok = false; break; }
          uint8_t* st = smem + s * kStageBytes;
          dev::mbar_expect_tx(&full[s], w.nh * kABlock + kBBytes);
          for (int h = w.h0; h < w.h0 + w.nh; ++h)
            dev::tma_load_2d(st + h * kABlock, &amap, &full[s], kb * BK, (w.tm2 * 2 + h) * BMB);
          dev::tma_load_2d(st + kABytes, &bmap, &full[s], w.tn * BN, kb * BK);
          dev::tma_load_2d(st + kABytes + BK * 128, &bmap, &full[s], w.tn * BN + 128, kb * BK);
          ph ^= (s == kStages - 1);
          s = (s == kStages - 1) ? 0 : s + 1;
        }
      }
    }
  } else if (warp == 1 || warp == kSecondMmaWarp) {
    // ------------------------------ MMA issuers ----------------------------
    // Issuer j multiplies row block j of every item that has it into accumulator j.  The issuing
    // thread is the serial resource (a tcgen05.mma costs it ~85 cycles, a poll or a commit about
    // as much), so descriptors are advanced by adds on their low halves, the ring index by a
    // select, and an absent block is a predicated-off instruction, not a branch.
    if (lane == 0) {
      const int me = (warp == 1) ? 0 : 1;
      constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (kSwizzle128 << 29);  // SBO, version, swizzle
      // a: K-major, 32 bytes of k per instruction inside the 128-byte swizzle span
      const uint32_t a_lo0 = (((dev::smem_u32(smem) >> 4) & 0x3FFF) | ((16u >> 4) << 16)) + me * (kABlock >> 4);
      // b: MN-major, 32 k-rows (4 KB) per instruction; column blocks 16 KB apart
      const uint32_t b_lo0 = ((dev::smem_u32(smem + kABytes) >> 4) & 0x3FFF) | (((BK * 128u) >> 4) << 16);
      constexpr uint32_t kStageStep = kStageBytes >> 4, kAStepK = 32 >> 4, kBStepK = (32 * 128) >> 4;
      const uint32_t d_tmem = tmem_base + me * BN;
      uint32_t s = 0, ph = 0;
      int items = 0;
      bool ok = true;
      Work w;
      for (int i = 0; ok && get_work<SPLIT>(i, tiles_m2, tiles_n, halves, M, w); ++i) {
        if (w.nh == 0) continue;
        if (!dev::mbar_wait(tempty, (items & 1) ^ 1, status, 12)) break;
        dev::tc_fence_after();
        const uint32_t mine = (me >= w.h0) && (me < w.h0 + w.nh);
        for (int kb = kb_begin; kb < kb_end; ++kb) {
          if (!dev::mbar_wait(&full[s], ph, status, 13)) { ok = false; break; }
          dev::tc_fence_after();
          const uint32_t a_s = a_lo0 + s * kStageStep, b_s = b_lo0 + s * kStageStep;
          dev::umma_i8_lh_if(mine, d_tmem, a_s, kDescHi, b_s, kDescHi, idesc, kb != kb_begin);
          dev::umma_i8_lh_if(mine, d_tmem, a_s + kAStepK, kDescHi, b_s + kBStepK, kDescHi, idesc, 1);
          dev::umma_i8_lh_if(mine, d_tmem, a_s + 2 * kAStepK, kDescHi, b_s + 2 * kBStepK, kDescHi, idesc, 1);
          dev::umma_i8_lh_if(mine, d_tmem, a_s + 3 * kAStepK, kDescHi, b_s + 3 * kBStepK, kDescHi, idesc, 1);
          dev::tc_commit(&empty[s]);  // second arrival: the other issuer
          ph ^= (s == kStages - 1);
          s = (s == kStages - 1) ? 0 : s + 1;
        }
        if (ok) dev::tc_commit(tfull);
        ++items;
      }
    }
  } else {
    // ------------------------------ epilogue -------------------------------
    const int q = warp & 3;         // TMEM lane quarter this warp may access
    const int j = (warp - 2) >> 2;  // accumulator (row block) of this warp
    const uint64_t store_policy = dev::policy_evict_first();
    int items = 0;
    Work w;
    for (int i = 0; get_work<SPLIT>(i, tiles_m2, tiles_n, halves, M, w); ++i) {
      if (w.nh == 0) continue;
      if (!dev::mbar_wait_relaxed_warp(tfull, items & 1, status, 14)) break;
      dev::tc_fence_after();
      // A lane holds one row of a 32 x 32 chunk.  Stored straight from registers, a warp's 16-byte stores
      // would touch 32 different 128-byte lines per instruction; instead the chunk goes to shared memory
      // (row r at r * 128, 16-byte piece p at p ^ (r & 7): conflict-free) and one TMA store writes it out,
      // clipped to the tensor's bounds.
      // results of the CTA's last item leave through shared memory and TMA stores (the ring is idle: every load
      // has been consumed once the accumulators are complete); earlier items overlap their plain stores with the
      // loads of the next item, which the producer has already started into the ring
      Work w_next;
      const bool staged = staged_store && !get_work<SPLIT>(i + 1, tiles_m2, tiles_n, halves, M, w_next);
      const int block = SPLIT ? w.h0 : j;   // (a single block's chunks are shared out among all warps)
      const int row0 = (w.tm2 * 2 + block) * BMB + q * 32;
      const int row = row0 + lane;
      const bool mine = (j >= w.h0) && (j < w.h0 + w.nh) && row < M;
      const float rs = (f_out && mine) ? __ldg(row_scale + row) : 0.f;
      uint8_t* stage = smem + kOutBase + (warp - 2) * kOutStage;
      uint8_t* my_row = stage + lane * 128;
      if (block >= w.h0 && block < w.h0 + w.nh && row0 < M) {
#pragma unroll 1
        for (int ch = SPLIT ? j : 0; ch < BN / 32; ch += SPLIT ? 2 : 1) {
          const int col0 = w.tn * BN + ch * 32;
          if (col0 >= N) break;
          uint32_t r[32];
          dev::tmem_ld_32x32(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + block * BN + ch * 32, r);
          dev::tc_wait_ld();
          if (SPLIT) {   // the sums of this CTA's share of K, [row][256 columns], 16-byte pieces swizzled by the row
#pragma unroll
            for (int i4 = 0; i4 < 8; ++i4)
              *reinterpret_cast<uint4*>(smem + (q * 32 + lane) * (BN * 4) + (((ch * 8 + i4) ^ (lane & 7)) << 4)) =
                  make_uint4(r[4 * i4], r[4 * i4 + 1], r[4 * i4 + 2], r[4 * i4 + 3]);
            continue;
          }
          if (!staged) {
            // straight from registers: 16-byte stores of 32 different rows per instruction
            if (mine) {
              if (acc_out) {
                int32_t* dst = acc_out + static_cast<size_t>(row) * N + col0;
#pragma unroll
                for (int i4 = 0; i4 < 8; ++i4)
                  if (col0 + 4 * i4 < N)
                    *reinterpret_cast<uint4*>(dst + 4 * i4) = make_uint4(r[4 * i4], r[4 * i4 + 1], r[4 * i4 + 2], r[4 * i4 + 3]);
              }
              if (f_out) {
                float* dst = f_out + static_cast<size_t>(row) * N + col0;
#pragma unroll
                for (int i4 = 0; i4 < 8; ++i4)
                  if (col0 + 4 * i4 < N) {
                    const float4 cs = __ldg(reinterpret_cast<const float4*>(col_scale + col0 + 4 * i4));
                    float4 o;
                    o.x = static_cast<float>(static_cast<int32_t>(r[4 * i4])) * rs * cs.x;
                    o.y = static_cast<float>(static_cast<int32_t>(r[4 * i4 + 1])) * rs * cs.y;
                    o.z = static_cast<float>(static_cast<int32_t>(r[4 * i4 + 2])) * rs * cs.z;
                    o.w = static_cast<float>(static_cast<int32_t>(r[4 * i4 + 3])) * rs * cs.w;
                    *reinterpret_cast<float4*>(dst + 4 * i4) = o;
                  }
              }
            }
            continue;
          }
          if (acc_out) {
            if (lane == 0) dev::tma_store_wait_read();   // the previous store has read the buffer
            __syncwarp();
#pragma unroll
            for (int i4 = 0; i4 < 8; ++i4)
              *reinterpret_cast<uint4*>(my_row + ((i4 ^ (lane & 7)) << 4)) =
                  make_uint4(r[4 * i4], r[4 * i4 + 1], r[4 * i4 + 2], r[4 * i4 + 3]);
            dev::fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
              dev::tma_store_2d_hint(&accmap, stage, col0, row0, store_policy);
              dev::tma_store_commit();
            }
          }
          if (f_out) {
            float4 o[8];
#pragma unroll
            for (int i4 = 0; i4 < 8; ++i4) {
              float4 cs = make_float4(0.f, 0.f, 0.f, 0.f);
              if (col0 + 4 * i4 < N) cs = __ldg(reinterpret_cast<const float4*>(col_scale + col0 + 4 * i4));
              o[i4].x = static_cast<float>(static_cast<int32_t>(r[4 * i4])) * rs * cs.x;
              o[i4].y = static_cast<float>(static_cast<int32_t>(r[4 * i4 + 1])) * rs * cs.y;
              o[i4].z = static_cast<float>(static_cast<int32_t>(r[4 * i4 + 2])) * rs * cs.z;
              o[i4].w = static_cast<float>(static_cast<int32_t>(r[4 * i4 + 3])) * rs * cs.w;
            }
            if (lane == 0) dev::tma_store_wait_read();
            __syncwarp();
#pragma unroll
            for (int i4 = 0; i4 < 8; ++i4) *reinterpret_cast<float4*>(my_row + ((i4 ^ (lane & 7)) << 4)) = o[i4];
            dev::fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
              dev::tma_store_2d_hint(&outmap, stage, col0, row0, store_policy);
              dev::tma_store_commit();
            }
          }
        }
      }
      dev::tc_fence_before();
      __syncwarp();
      if (lane == 0) dev::mbar_arrive(tempty);
      ++items;
    }
    if (lane == 0) dev::tma_store_wait_read();   // no store still reads this CTA's shared memory
  }
  if (SPLIT) {
    // Every CTA of the cluster sums every gridDim.x-th run of the results, four columns to a thread.
    __syncwarp();
    split::cluster_sync();
    Work w;
    if (get_work<SPLIT>(0, tiles_m2, tiles_n, halves, M, w) && w.nh > 0) {
      const int row0 = (w.tm2 * 2 + w.h0) * BMB, rows = min(M - row0, BMB);
      const int step = gridDim.x * kThreads, end = rows * (BN / 4);
      for (int e0 = blockIdx.x * kThreads + threadIdx.x; e0 < end; e0 += 2 * step) {
        float4 v[2][split::kMaxCluster];   // two runs at a time: a load from a peer takes about 0.5 us
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int e = min(e0 + k * step, end - 1), r = e / (BN / 4), c = e % (BN / 4);
          const float4* at = reinterpret_cast<const float4*>(smem + r * (BN * 4) + ((c ^ (r & 7)) << 4));
#pragma unroll
          for (int p = 0; p < split::kMaxCluster; ++p)
            if (p < gridDim.x) v[k][p] = split::load_peer(at, p);
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int e = e0 + k * step, r = e / (BN / 4), col = w.tn * BN + e % (BN / 4) * 4;
          if (e >= end || col >= N) continue;
          uint32_t sum[4] = {0u, 0u, 0u, 0u};
#pragma unroll
          for (int p = 0; p < split::kMaxCluster; ++p)
            if (p < gridDim.x) {
              sum[0] += __float_as_uint(v[k][p].x);
              sum[1] += __float_as_uint(v[k][p].y);
              sum[2] += __float_as_uint(v[k][p].z);
              sum[3] += __float_as_uint(v[k][p].w);
            }
          const size_t to = static_cast<size_t>(row0 + r) * N + col;
          if (acc_out) *reinterpret_cast<uint4*>(acc_out + to) = make_uint4(sum[0], sum[1], sum[2], sum[3]);
          if (f_out) {
            const float rs = __ldg(row_scale + row0 + r);
            const float4 cs = __ldg(reinterpret_cast<const float4*>(col_scale + col));
            float4 o;
            o.x = static_cast<float>(static_cast<int32_t>(sum[0])) * rs * cs.x;
            o.y = static_cast<float>(static_cast<int32_t>(sum[1])) * rs * cs.y;
            o.z = static_cast<float>(static_cast<int32_t>(sum[2])) * rs * cs.z;
            o.w = static_cast<float>(static_cast<int32_t>(sum[3])) * rs * cs.w;
            *reinterpret_cast<float4*>(f_out + to) = o;
          }
        }
      }
    }
    __syncwarp();
    split::cluster_sync();   // peers keep their shared memory alive until it has been read
  }
  dev::tc_fence_before();
  __syncthreads();
  if (warp == 1) dev::tmem_dealloc(tmem_base, 512);
}
}  // namespace i8

// ============================================================================
// (2) bf16 activations x int8 weights (per-output-channel scale) -> bf16
// ============================================================================
namespace w8 {
constexpr int BNW = 128;   // output channels per MMA (its M); a full tile has two such blocks
constexpr int kMaxRows = 192;   // activation rows per tile (MMA N), at most: two accumulators of 192 columns leave 128 for the weights
constexpr int BK = 64;     // k per stage
constexpr int kXStages = 4;    // activation ring, held until the MMAs that read a stage retire
constexpr int kWStages = 6;    // raw-weight ring (a multiple of the converter groups), held only until a stage is in registers
constexpr int kCvtWarps = 8;    // converter warps per group
constexpr int kCvtGroups = 2;   // group g converts the stages with cnt % 2 == g
constexpr int kCvtSlots = 2;    // converted stages in TMEM
// Warp roles: 0 TMA (activations), 1 MMA issue for channel block 0, 2-17 workers (convert the
// stages of a tile, then drain its accumulators), 18 TMA (raw weights), 19 MMA issue for channel
// block 1.
constexpr int kFirstCvtWarp = 2;
constexpr int kWorkerWarps = kCvtGroups * kCvtWarps;
constexpr int kWProducerWarp = kFirstCvtWarp + kWorkerWarps;
constexpr int kSecondMmaWarp = kWProducerWarp + 1;
constexpr int kWarps = kSecondMmaWarp + 1;
constexpr int kRawBlock = BK * BNW;               // 8 KB  int8 [k][128 n]
constexpr int kRawBytes = 2 * kRawBlock;          // 16 KB: both channel blocks
constexpr int kXBytes = kMaxRows * BK * 2;        // 24 KB bf16 [m][k]
constexpr int kRawBase = kXStages * kXBytes;                 // 96 KB
constexpr int kBarBase = kRawBase + kWStages * kRawBytes;    // 192 KB
constexpr int kThreads = kWarps * 32;
constexpr int kSmemBytes = kBarBase + 256 + 1024;
constexpr int kSlotCols = 2 * BK / 2;             // TMEM columns of a converted stage: both channel blocks, two k to a column
constexpr int kAccBase = kCvtSlots * kSlotCols;   // first TMEM column of the accumulators
static_assert(kAccBase + 2 * kMaxRows <= 512, "TMEM");
static_assert(kWStages % kCvtGroups == 0, "a group has seen the phase ahead of the one that it waits for");
// Tiles of up to 96 rows leave accumulators unused: with int8 weights, K goes into two to six of them one after the other, and the
// epilogue adds them up in f32, rounded.  The tensor core cuts off what it adds to an accumulator, and a long K in one shows.  Outputs
// that a rounding to bf16 puts elsewhere than it puts the sum in 64 bits, M = 32: 4.0e-4 -> 2.1e-4 for 8192 x 8192, 6.7e-4 -> 3.1e-4 for
// 14336 x 4096, 2.1e-3 -> 2.9e-4 for 28672 x 8192 (the kernel for few rows: 2.4e-4, 1.5e-4, 9.5e-4).  It costs 1 to 3 % (8192 x 8192,
// M = 32 22.1 -> 22.5 us, M = 64 23.5 -> 24.1), 4 % where few rows meet many columns (8192 x 57344 118.1 -> 123.3).  int4 weights, which
// come here from 33 rows on and are rounded themselves, keep one.
constexpr int kLeastPart = 16;   // stages that are worth an accumulator
constexpr int kPanelTiles = 8;  // most activation tiles swept together (fewer when K is long: a panel should stay in L2)
// One "consumed" barrier per stage in a ring: the activation producer waits for stage cnt - 4, the converters for
// stage cnt - 2, and the issuing threads commit once per stage.
constexpr int kConsumed = 6;


// Two int8 -> two bf16, exactly, over 64.  `word` holds u = v + 128 in each byte: u in the low bits of a half reads as the bf16
// u * 2^-133 (a subnormal up to 127, the first binade above), and one fused multiply-add makes u / 64 - 2 = v / 64 of it (|v| <=
// 128 has 8 significant bits).  The epilogue multiplies by 64.
__device__ __forceinline__ uint32_t convert2(uint32_t word, uint32_t selector) {
  uint32_t r;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(__byte_perm(word, 0u, selector)), "r"(0x7F007F00u), "r"(0xC000C000u));
  return r;
}

// The work of one launch.  A full tile is 256 channels x `rows` rows: two channel
// blocks share one activation tile, so a CTA stages up to 40 KB per 64 k for
// 2 x 128 x 192 outputs.  CTA c takes tiles c, c + G, ... for `full_waves`
// rounds; the tiles left over (fewer than G) are cut into `tail_div` parts each
// (1: whole, 2: one channel block, 4: one channel block x half of the rows) and dealt
// round-robin, so that the last round costs 1 / tail_div of a tile.
struct Sched {
  int tiles_n2, tiles_m, full_waves, tail_tiles, tail_div;
  int panel;  // activation tiles per panel
  int rows;   // rows per tile, a multiple of 32
  int ks;     // CTAs that share the K of a piece
  float cost;   // estimate in microseconds
};
struct Work {
  int tn2, tm;   // tile coordinates (units of 256 channels, of `rows` rows)
  int h0, nh;    // channel blocks [h0, h0 + nh); nh == 0: nothing to do
  int m_off, m_cols;  // rows [m_off, m_off + m_cols) of the activation tile
};

// Tile order: activation tiles are swept in panels of `panel` tiles; inside a
// panel the weight tile changes slowest, so the CTAs that run together share
// one panel of activations (it stays in L2) and a handful of weight tiles.
__device__ __forceinline__ void tile_coords(int tile, int tiles_m, int tiles_n, int panel, int& tm, int& tn) {
  const int per_panel = panel * tiles_n;
  const int p = tile / per_panel, r = tile - p * per_panel;
  const int rows = min(panel, tiles_m - p * panel);  // the last panel may be short
  tn = r / rows;
  tm = p * panel + r % rows;
}

// Item `i` of this CTA (of its cluster); false when there is none.  After its full-wave tiles a CTA takes a
// contiguous run of the tail's parts (tile-major: part 2h + mh of a tile cut in four is channel
// block h, row half mh) and works it off in the largest aligned pieces: a whole tile, a channel
// block with all its rows, or a single part, so that neighbouring parts cost one pipeline fill
// and use the full-width MMA.
template <bool SPLIT>
__device__ __forceinline__ bool get_work(const Sched& sc, int i, int M, int N, Work& w) {
  const int cta = SPLIT ? blockIdx.y : blockIdx.x, G = SPLIT ? gridDim.y : gridDim.x;
  int tile, sub = 0, len = 0;  // len: parts covered, in units of 1 / tail_div tile; 0 = whole tile
  const int div = sc.tail_div;
  if (i < sc.full_waves) {
    tile = cta + i * G;
  } else {
    const long long total = static_cast<long long>(sc.tail_tiles) * div;
    int pos = static_cast<int>(cta * total / G);
    const int end = static_cast<int>((cta + 1) * total / G);
    for (int skip = i - sc.full_waves;; --skip) {
      if (pos >= end) return false;
      const int r = pos % div;
      if (r == 0 && pos + div <= end) len = div;                       // whole tile
      else if (div == 4 && (r & 1) == 0 && pos + 2 <= end) len = 2;    // one channel block, all rows
      else len = 1;
      if (skip == 0) break;
      pos += len;
    }
    tile = sc.full_waves * G + pos / div;
    sub = pos % div;
    if (len == div) len = 0;
  }
  tile_coords(tile, sc.tiles_m, sc.tiles_n2, sc.panel, w.tm, w.tn2);
  w.h0 = 0; w.nh = 2; w.m_off = 0; w.m_cols = sc.rows;
  if (len != 0) {
    if (div == 2) { w.h0 = sub; w.nh = 1; }
    if (div == 4) {
      w.h0 = sub >> 1; w.nh = 1;
      if (len == 1) { w.m_off = (sub & 1) * (sc.rows / 2); w.m_cols = sc.rows / 2; }
    }
  }
  const int blocks_left = (N - w.tn2 * 2 * BNW + BNW - 1) / BNW - w.h0;  // channel blocks that exist
  w.nh = max(0, min(w.nh, blocks_left));
  if (w.tm * sc.rows + w.m_off >= M) w.nh = 0;
  return true;
}

// Per-group constants of the int4 variant (null / unused for int8 weights).
struct GroupQuant {
  const uint16_t* scales;  // bf16 [K/128, N]
  const uint8_t* zeros;    // u8 [K/128, N], or two per byte [K/128, N/2]
  int packed;
};

// One packed byte (two k of one channel, low nibble = even k) -> the bf16 pair (q - z) * s.  `w` holds the byte at
// position BYTE, `w4` is w >> 4.  0x4300 | q is the bf16 128 + q exactly, zz holds 128 + z twice, so the subtraction is exact
// and the product is rounded to bf16 once: bit for bit what the StableHLO chain convert -> subtract -> multiply computes in bf16.
template <int BYTE>
__device__ __forceinline__ uint32_t dequant2(uint32_t w, uint32_t w4, uint32_t zz, uint32_t ss) {
  uint32_t t;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(t) : "r"(__byte_perm(w, w4, BYTE | (4 + BYTE) << 8)), "r"(0x000F000Fu), "r"(0x43004300u));
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(t) : "r"(t), "r"(zz));
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(t) : "r"(t), "r"(ss));
  return t;
}

// WBITS = 8: int8 weights [K, N], per-channel f32 scale applied in the epilogue.
// WBITS = 4: packed int4 weights [K/2, N] (byte = two k of one channel), per-(128-k group, channel)
//            bf16 scale and zero point applied by the converter warps; K % 128 == 0.
// SPLIT: a piece of work is one cluster's; its CTAs take a share of K each and add their accumulators up over distributed
// shared memory, in CTA order.  One piece a cluster, so that the rings are free for the sums when the last MMA has retired.
// PARTS: K in several accumulators.
template <int WBITS, bool SPLIT, bool PARTS>
__global__ void __launch_bounds__(kThreads, 1)
w8a16_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap,
             const float* __restrict__ scale, const GroupQuant gq, uint16_t* __restrict__ y, int M, int N, int K,
             long long ldy, uint32_t idesc_full, uint32_t idesc_half, const Sched sc, uint32_t flags,
             uint32_t* signal, uint32_t* arrive, int* status) {
  // a raw stage holds 64 k of both channel blocks: 64 byte-rows of int8, 32 of packed int4
  constexpr int kRawRows = (WBITS == 8) ? BK : BK / 2;
  constexpr int kRawBlockW = kRawRows * BNW;
  extern __shared__ uint8_t smem_raw[];
  // An independent launch lets its successor start at once.  A dependent one does so only after
  // its own wait below: a successor that is itself flagged independent can then overlap this
  // launch, but never anything older than it.
  if (flags & QMM_GEMM_INDEPENDENT) dev::pdl_launch_dependents();
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint64_t* xfull = reinterpret_cast<uint64_t*>(smem + kBarBase);  // activations landed
  uint64_t* wfull = xfull + kXStages;    // raw weights landed
  uint64_t* wempty = wfull + kWStages;   // raw weights are in the converters' registers
  uint64_t* sfull = wempty + kWStages;   // stage ready for the MMAs: converted, and its activations landed
  uint64_t* consumed = sfull + kCvtSlots;   // the MMAs of a stage retired (ring of kConsumed stages)
  uint64_t* tfull = consumed + kConsumed;   // accumulators complete
  uint64_t* tempty = tfull + 1;             // accumulators drained
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int all_kblocks = (K + BK - 1) / BK;
  const int kb_begin = SPLIT ? static_cast<int>(static_cast<long long>(all_kblocks) * blockIdx.x / gridDim.x) : 0;
  const int kb_end = SPLIT ? static_cast<int>(static_cast<long long>(all_kblocks) * (blockIdx.x + 1) / gridDim.x) : all_kblocks;
  // stages that go into one accumulator
  const int spare = PARTS ? kMaxRows / sc.rows : 1, part = PARTS ? max((kb_end - kb_begin + spare - 1) / spare, kLeastPart) : kb_end - kb_begin;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kXStages; ++s) dev::mbar_init(&xfull[s], 1);
    for (int s = 0; s < kWStages; ++s) {
      dev::mbar_init(&wfull[s], 1);
      dev::mbar_init(&wempty[s], kCvtWarps);
    }
    for (int g = 0; g < kCvtSlots; ++g) dev::mbar_init(&sfull[g], kCvtWarps);
    for (int i = 0; i < kConsumed; ++i) dev::mbar_init(&consumed[i], 2);  // one commit per issuing thread
    dev::mbar_init(tfull, 2);
    dev::mbar_init(tempty, kWorkerWarps);
    dev::fence_mbar_init();
  }
  if (warp == 1) {
    dev::tmem_alloc(tmem_slot, 512);
    dev::tmem_relinquish();
  }
  dev::tc_fence_before();
  __syncthreads();
  dev::tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
  // Ordered behind the kernels ahead on the stream before global memory is touched, unless the
  // caller stated that none of them writes this launch's operands or touches its output.
  if (!(flags & QMM_GEMM_INDEPENDENT)) {
    dev::pdl_wait();
    dev::pdl_launch_dependents();
  }
  const bool mc_store = (flags & QMM_GEMM_STORE_MULTIMEM) != 0;

  // Stage `cnt` (counted over the whole launch) uses activation slot cnt % 4,
  // raw-weight slot cnt % 6 and the converted stage cnt % 2 in TMEM.
  if (warp == 0) {
    // ------------------------ TMA producer: activations --------------------
    if (lane == 0) {
      dev::tma_prefetch_desc(&xmap);
      unsigned cnt = 0;
      bool ok = true;
      Work w;
      for (int i = 0; ok && get_work<SPLIT>(sc, i, M, N, w); ++i) {
        if (w.nh == 0) continue;
        for (int kb = kb_begin; kb < kb_end; ++kb, ++cnt) {
          const int xs = cnt % kXStages;
          if (cnt >= kXStages) {  // the slot's previous stage must have been multiplied
            const unsigned prev = cnt - kXStages;
            if (!dev::mbar_wait(&consumed[prev % kConsumed], (prev / kConsumed) & 1, status, 21)) { ok = false; break; }
          }
          dev::mbar_expect_tx(&xfull[xs], sc.rows * BK * 2);
          dev::tma_load_2d(smem + xs * kXBytes, &xmap, &xfull[xs], kb * BK, w.tm * sc.rows);
        }
      }
    }
  } else if (warp == kWProducerWarp) {
    // ------------------------ TMA producer: raw weights --------------------
    if (lane == 0) {
      dev::tma_prefetch_desc(&wmap);
      unsigned cnt = 0;
      bool ok = true;
      Work w;
      for (int i = 0; ok && get_work<SPLIT>(sc, i, M, N, w); ++i) {
        if (w.nh == 0) continue;
        for (int kb = kb_begin; kb < kb_end; ++kb, ++cnt) {
          const int ws = cnt % kWStages;
          if (!dev::mbar_wait(&wempty[ws], ((cnt / kWStages) & 1) ^ 1, status, 20)) { ok = false; break; }
          uint8_t* raw = smem + kRawBase + ws * kRawBytes;
          dev::mbar_expect_tx(&wfull[ws], w.nh * kRawBlockW);
          for (int h = w.h0; h < w.h0 + w.nh; ++h)
            dev::tma_load_2d(raw + h * kRawBlockW, &wmap, &wfull[ws], (w.tn2 * 2 + h) * BNW, kb * kRawRows);
        }
      }
    }
  } else if (warp == 1 || warp == kSecondMmaWarp) {
    // ------------------------------ MMA issuers ----------------------------
    // Issuer j multiplies channel block j of every item that has it into accumulator j; both
    // follow the same barriers and both commit, whether or not they issued anything.  The
    // issuing thread is a slow scalar processor (a branch or a shared-memory poll costs it
    // tens of cycles, a commit ~90), so a stage costs it one wait, one fence, four predicated
    // MMAs with descriptors advanced by adds, and one commit.
    if (lane == 0) {
      const int me = (warp == 1) ? 0 : 1;
      // descriptor halves: the high half is constant, the low half carries the start address
      constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (kSwizzle128 << 29);  // SBO, version, swizzle
      constexpr uint32_t kBStepK = 32 >> 4, kBStepStage = kXBytes >> 4;
      const uint32_t a_t0 = tmem_base + me * (BK / 2);
      const uint32_t b_lo0 = ((dev::smem_u32(smem) >> 4) & 0x3FFF) | ((16u >> 4) << 16);
      const uint32_t d = tmem_base + kAccBase + me * kMaxRows;
      uint32_t g = 0, gpar = 0;   // converted-stage slot and the parity of its use
      uint32_t xs = 0;            // activation slot
      uint32_t c6 = 0;            // consumed-ring index
      int items = 0;
      bool ok = true, ready = false;
      Work w;
      for (int i = 0; ok && get_work<SPLIT>(sc, i, M, N, w); ++i) {
        if (w.nh == 0) continue;
        if (!dev::mbar_wait(tempty, (items & 1) ^ 1, status, 22)) break;
        dev::tc_fence_after();
        const uint32_t idesc = (w.m_cols == sc.rows) ? idesc_full : idesc_half;
        const uint32_t b_item = b_lo0 + ((w.m_off * 128) >> 4);
        const uint32_t mine = (me >= w.h0) && (me < w.h0 + w.nh);
        auto multiply = [&](uint32_t d, int begin, int end) {
          for (int kb = begin; kb < end; ++kb) {
            // whether the next stage is ready is asked while this one's MMAs are still being issued: behind them a question
            // waits for its turn
            if (!ready && !dev::mbar_wait(&sfull[g], gpar, status, 23)) { ok = false; break; }
            dev::tc_fence_after();
            const uint32_t a_c = a_t0 + g * kSlotCols;   // 16 k: eight columns
            const uint32_t b_s = b_item + xs * kBStepStage;
            dev::umma_f16_ts_if(mine, d, a_c, b_s, kDescHi, idesc, kb != begin);
            dev::umma_f16_ts_if(mine, d, a_c + 8, b_s + kBStepK, kDescHi, idesc, 1);
            dev::umma_f16_ts_if(mine, d, a_c + 16, b_s + 2 * kBStepK, kDescHi, idesc, 1);
            ready = dev::mbar_test(&sfull[g ^ 1], gpar ^ g);
            dev::umma_f16_ts_if(mine, d, a_c + 24, b_s + 3 * kBStepK, kDescHi, idesc, 1);
            dev::tc_commit(&consumed[c6]);  // second arrival: the other issuer
            gpar ^= g;  // the parity flips after slot 1's stage
            g ^= 1;
            xs = (xs == kXStages - 1) ? 0 : xs + 1;
            c6 = (c6 == kConsumed - 1) ? 0 : c6 + 1;
          }
        };
        if (PARTS) {
          uint32_t d_part = d;
          for (int kb = kb_begin; ok && kb < kb_end; kb += part, d_part += sc.rows) multiply(d_part, kb, min(kb + part, kb_end));
        } else {
          multiply(d, kb_begin, kb_end);
        }
        if (ok) dev::tc_commit(tfull);
        ++items;
      }
    }
  } else {
    // ------------------------------ workers --------------------------------
    // Conversion: a warp takes one lane quarter (32 channels) of one channel block, all 64 k of a stage.  ldmatrix.trans
    // on 16-bit units leaves, for two neighbouring channels, two k (int8) or two packed pairs of k (int4) in a register;
    // converted, they have the layout of the 16-lane TMEM stores, with channel 2 i in lane i and channel 2 i + 1 in lane
    // i + 8 of the 16.  Two groups of eight warps take every other stage.
    // Epilogue: when the tile's stages are converted the same 16 warps drain its accumulators
    // (warp & 3 selects the 32 TMEM lanes = channels a warp may read; the four warps of a lane
    // quarter share the 32-row chunks).
    const int o = warp - kFirstCvtWarp;
    const int grp = o / kCvtWarps, cw = o % kCvtWarps;
    const int q = warp & 3, esub = o >> 2;
    const int hh = cw >> 2;              // channel block of the item that this warp converts
    const uint32_t a_lane = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    unsigned cnt = 0;  // stages since the start of the launch
    int turn = 0;      // cnt % kCvtGroups
    int items = 0;
    bool ok = true;
    Work w;
    for (int i = 0; ok && get_work<SPLIT>(sc, i, M, N, w); ++i) {
      if (w.nh == 0) continue;
      const int h = w.h0 + hh;
      const bool mine = hh < w.nh;
      uint32_t sv_next[2] = {0u, 0u}, zv_next[2] = {0u, 0u};
      auto load_scales = [&](int kb, int h) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const long long at = static_cast<long long>(kb >> 1) * N + (w.tn2 * 2 + h) * BNW + q * 32 + c * 16 + 2 * (lane >> 2);
          sv_next[c] = __ldg(reinterpret_cast<const uint32_t*>(gq.scales + at));
          zv_next[c] = gq.packed ? __ldg(gq.zeros + at / 2) : __ldg(reinterpret_cast<const uint16_t*>(gq.zeros + at));
        }
      };
      if (WBITS == 4 && mine) {
        const int first = kb_begin + (grp + kCvtGroups - turn) % kCvtGroups;   // the group's first stage of the item
        if (first < kb_end) load_scales(first, h);
      }
      for (int kb = kb_begin; kb < kb_end; ++kb, ++cnt, turn = (turn == kCvtGroups - 1) ? 0 : turn + 1) {
        if (turn != grp) continue;
        const int ws = cnt % kWStages;
        const uint32_t raw = dev::smem_u32(smem + kRawBase + ws * kRawBytes + h * kRawBlockW) + lane * 128;
        const uint32_t a_slot = a_lane + (cnt & 1) * kSlotCols + h * (BK / 2);
        // scales and zero points of the stage's 128-k group and this lane's two channel pairs, read one stage of the group's ahead
        uint32_t sv[2] = {sv_next[0], sv_next[1]}, zv[2] = {zv_next[0], zv_next[1]};
        if (WBITS == 4 && mine && kb + kCvtGroups < kb_end) load_scales(kb + kCvtGroups, h);
        if (!dev::mbar_wait_warp(&wfull[ws], (cnt / kWStages) & 1, status, 26)) { ok = false; break; }
        // 16 channels x 64 k -> 16 registers
        auto convert = [&](int c, uint32_t (&out)[16]) {
          const uint32_t at = raw + (((q * 2 + c) ^ (lane & 7)) << 4);
          if (WBITS == 4) {
            uint32_t in[4];
            split::ldmatrix_x4_trans(at, in);
            const uint32_t s0 = __byte_perm(sv[c], 0u, 0x1010), s1 = __byte_perm(sv[c], 0u, 0x3232);
            // the two zero points: nibbles of a byte, or two bytes
            const uint32_t z0 = 0x43004300u | (gq.packed ? (zv[c] & 0xFu) * 0x10001u : __byte_perm(zv[c], 0u, 0x4040));
            const uint32_t z1 = 0x43004300u | (gq.packed ? (zv[c] >> 4) * 0x10001u : __byte_perm(zv[c], 0u, 0x4141));
#pragma unroll
            for (int m = 0; m < 4; ++m) {
              const uint32_t v = in[m], v4 = in[m] >> 4;
              out[4 * m] = dequant2<0>(v, v4, z0, s0);
              out[4 * m + 1] = dequant2<2>(v, v4, z0, s0);
              out[4 * m + 2] = dequant2<1>(v, v4, z1, s1);
              out[4 * m + 3] = dequant2<3>(v, v4, z1, s1);
            }
          } else {
#pragma unroll
            for (int g = 0; g < 2; ++g) {
              uint32_t in[4];
              split::ldmatrix_x4_trans(at + g * 32 * 128, in);
#pragma unroll
              for (int m = 0; m < 4; ++m) {
                const uint32_t u = in[m] ^ 0x80808080u;
                out[8 * g + 2 * m] = convert2(u, 0x4240);
                out[8 * g + 2 * m + 1] = convert2(u, 0x4341);
              }
            }
          }
        };
        auto store = [&](int c, const uint32_t (&out)[16]) {
          if (WBITS == 4) dev::tmem_st_16x256b_x4(a_slot + (static_cast<uint32_t>(c * 16) << 16), out);
          else dev::tmem_st_16x128b_x8(a_slot + (static_cast<uint32_t>(c * 16) << 16), out);
        };
        // Everything is converted before the wait for the slot: from the end of the MMAs that read it to the start of those
        // that read it next there are only two stores to TMEM.
        uint32_t out[2][16];
        if (mine) {
          convert(0, out[0]);
          convert(1, out[1]);
        }
        // the issuing threads wait only for this group: make sure the activations are there too
        if (!dev::mbar_wait_warp(&xfull[cnt % kXStages], (cnt / kXStages) & 1, status, 28)) { ok = false; break; }
        if (cnt >= 2) {  // the MMAs of the stage that used the slot before must have retired
          const unsigned prev = cnt - 2;
          if (!dev::mbar_wait_warp(&consumed[prev % kConsumed], (prev / kConsumed) & 1, status, 27)) { ok = false; break; }
          dev::tc_fence_after();
        }
        if (mine) {
          store(0, out[0]);
          store(1, out[1]);
          dev::tc_wait_st();
        }
        dev::tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          dev::mbar_arrive(&sfull[cnt & 1]);
          dev::mbar_arrive(&wempty[ws]);   // the raw bytes went through registers into TMEM
        }
      }
      if (!ok) break;
      // ---- epilogue of this item
      if (!dev::mbar_wait_relaxed_warp(tfull, items & 1, status, 25)) break;
      dev::tc_fence_after();
      const int chunks = (w.m_cols + 31) / 32;
      const int m_end = min(M, w.tm * sc.rows + w.m_off + w.m_cols);
#pragma unroll 1
      for (int idx = esub; idx < w.nh * chunks; idx += kWorkerWarps / 4) {
        const int h = w.h0 + idx / chunks, ch = idx % chunks;
        // this thread's output channel: of 16 lanes, the first eight hold the even ones
        const int n = (w.tn2 * 2 + h) * BNW + q * 32 + (lane & 16) + 2 * (lane & 7) + ((lane >> 3) & 1);
        const float scl = (WBITS == 4) ? 1.f : ((n < N) ? __ldg(scale + n) : 0.f);
        uint32_t r[32];
        const uint32_t at = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + kAccBase + h * kMaxRows + ch * 32;
        dev::tmem_ld_32x32(at, r);
        dev::tc_wait_ld();
        if (PARTS) {
#pragma unroll 1
          for (int k = part, p = sc.rows; k < kb_end - kb_begin; k += part, p += sc.rows) {
#pragma unroll
            for (int e = 0; e < 32; e += 8) {   // (16 at a time spill)
              uint32_t more[8];
              dev::tmem_ld_32x8(at + p + e, more);
              dev::tc_wait_ld();
#pragma unroll
              for (int j = 0; j < 8; ++j) r[e + j] = __float_as_uint(__uint_as_float(r[e + j]) + __uint_as_float(more[j]));
            }
          }
        }
        if (SPLIT) {   // the sums of this CTA's share of K, [row][channel], over the rings
          float* mine = reinterpret_cast<float*>(smem) + (h - w.h0) * BNW + (n & (BNW - 1));
#pragma unroll
          for (int j = 0; j < 32; ++j) mine[(ch * 32 + j) * (w.nh * BNW)] = __uint_as_float(r[j]);
          continue;
        }
        if (idx + kWorkerWarps / 4 >= w.nh * chunks) {   // the last values are in registers: the next item may start
          dev::tc_fence_before();
          __syncwarp();
          if (lane == 0) dev::mbar_arrive(tempty);
        }
        const int m0 = w.tm * sc.rows + w.m_off + ch * 32;
        // pair neighbouring channels so that every lane stores 4 bytes: lanes of the
        // even channels write rows m0+2j, those of the odd ones rows m0+2j+1
        const bool odd = (lane & 8) != 0;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float a = (WBITS == 8 ? 64.f * __uint_as_float(r[2 * j]) : __uint_as_float(r[2 * j])) * scl;
          const float b = (WBITS == 8 ? 64.f * __uint_as_float(r[2 * j + 1]) : __uint_as_float(r[2 * j + 1])) * scl;
          const float send = odd ? a : b;
          const float got = __shfl_xor_sync(0xFFFFFFFFu, send, 8);
          const int m = m0 + 2 * j + odd;
          const uint32_t packed = odd ? dev::pack_bf16x2(got, b) : dev::pack_bf16x2(a, got);
          const int n_even = n & ~1;
          if (m < m_end && n_even < N) {
            uint16_t* dst = y + static_cast<size_t>(m) * ldy + n_even;
            if (mc_store) dev::multimem_st_b32(dst, packed);  // the same offset of every rank's buffer
            else *reinterpret_cast<uint32_t*>(dst) = packed;
          }
        }
      }
      if (SPLIT) break;
      if (esub >= w.nh * chunks) {   // a warp without a share
        __syncwarp();
        if (lane == 0) dev::mbar_arrive(tempty);
      }
      ++items;
    }
  }
  if (SPLIT) {
    // Every CTA of the cluster sums every gridDim.x-th run of the results, four channels to a thread.
    __syncwarp();
    split::cluster_sync();
    Work w;
    if (get_work<SPLIT>(sc, 0, M, N, w) && w.nh > 0) {
      const int quads = w.nh * (BNW / 4), m_first = w.tm * sc.rows + w.m_off;
      const int rows = min(M - m_first, w.m_cols), n_first = (w.tn2 * 2 + w.h0) * BNW;
      for (int e = blockIdx.x * kThreads + threadIdx.x; e < rows * quads; e += gridDim.x * kThreads) {
        const int row = e / quads, c = e % quads * 4, n = n_first + c;
        if (n >= N) continue;
        float4 v[split::kMaxCluster];
#pragma unroll
        for (int p = 0; p < split::kMaxCluster; ++p)
          if (p < gridDim.x) v[p] = split::load_peer(reinterpret_cast<const float4*>(smem + (row * quads * 4 + c) * 4), p);
        float4 sum = v[0];
#pragma unroll
        for (int p = 1; p < split::kMaxCluster; ++p)
          if (p < gridDim.x) {
            sum.x += v[p].x;
            sum.y += v[p].y;
            sum.z += v[p].z;
            sum.w += v[p].w;
          }
        if (WBITS == 8) {
          sum.x = 64.f * sum.x * __ldg(scale + n);
          sum.y = 64.f * sum.y * __ldg(scale + n + 1);
          sum.z = 64.f * sum.z * __ldg(scale + n + 2);
          sum.w = 64.f * sum.w * __ldg(scale + n + 3);
        }
        uint32_t* dst = reinterpret_cast<uint32_t*>(y + static_cast<size_t>(m_first + row) * ldy + n);
        dst[0] = dev::pack_bf16x2(sum.x, sum.y);
        dst[1] = dev::pack_bf16x2(sum.z, sum.w);
      }
    }
    __syncwarp();
    split::cluster_sync();   // peers keep their shared memory alive until it has been read
  }
  // Completion signal: every thread that stored makes its stores visible system-wide, the CTAs
  // count themselves on a local counter (which wraps back to zero), and the last one adds 1 to
  // the signal word with release semantics: on every rank at once when the word is a multicast
  // address.  A reader that sees the new count with an acquire load sees the whole output block.
  if (signal != nullptr) dev::fence_sys();
  dev::tc_fence_before();
  __syncthreads();
  if (warp == 1) dev::tmem_dealloc(tmem_base, 512);
  if (signal != nullptr && threadIdx.x == 0) {
    const unsigned prev = atomicInc(arrive, gridDim.x - 1);
    if (prev == gridDim.x - 1) {
      dev::fence_sys();
      if (mc_store) dev::multimem_red_release_add_u32(signal, 1u);
      else dev::red_release_sys_add_u32(signal, 1u);
    }
  }
}
}  // namespace w8

}  // namespace tc
}  // namespace qmm

// ----------------------------------------------------------------------------
// Host entry points (the tensor-core route; callers fall back for other shapes)
// ----------------------------------------------------------------------------
namespace qmm {

// CTAs that share the K of a 128 x 256 block.  The costs are a fit to 1200 calls (M 2 to 1024, K 64 to 16384, N 256 to 16384,
// every cluster size: 3 % off in the median): microseconds per 128 k, and per call for its start, its rows and the sums.
template <typename Fn>
static int split_of(int64_t M, int blocks, int stages, Fn resident) {
  const float rows = M < 128 ? static_cast<float>(M) : 128.f;
  int best = 1;
  float best_cost = 0.34f * stages + 6.9f + 0.009f * rows;
  for (int ks = 2; ks <= split::kMaxCluster && ks <= stages && blocks * ks <= num_sms(); ++ks) {
    if (blocks > resident(ks)) continue;
    const float cost = 0.34f * ((stages + ks - 1) / ks) + 4.6f + 0.2f * ks + (0.023f + 0.03f / ks) * rows;
    if (cost < best_cost) {
      best_cost = cost;
      best = ks;
    }
  }
  return best;
}

int i8gemm_tcgen05(const void* a, const void* b, int32_t* acc, const float* row_scale,
                   const float* col_scale, float* out, int64_t M, int64_t N, int64_t K,
                   int a_unsigned, int b_unsigned, cudaStream_t stream) {
  using namespace tc::i8;
  CUtensorMap amap, bmap;
  if (int rc = make_tensor_map_2d(&amap, a, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)M,
                                  (uint64_t)K, (uint64_t)K, BMB, 128, CU_TENSOR_MAP_SWIZZLE_128B))
    return rc;
  if (int rc = make_tensor_map_2d(&bmap, b, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)K,
                                  (uint64_t)N, (uint64_t)N, BK, 128, CU_TENSOR_MAP_SWIZZLE_128B))
    return rc;
  // results leave through TMA stores of 32 x 32 chunks (128 bytes of a row per chunk)
  CUtensorMap accmap = amap, outmap = amap;   // placeholders where an output is absent (never used by the kernel)
  if (acc)
    if (int rc = make_tensor_map_2d(&accmap, acc, CU_TENSOR_MAP_DATA_TYPE_INT32, 4, (uint64_t)M, (uint64_t)N,
                                    (uint64_t)N * 4, 32, 32, CU_TENSOR_MAP_SWIZZLE_128B))
      return rc;
  if (out)
    if (int rc = make_tensor_map_2d(&outmap, out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (uint64_t)M, (uint64_t)N,
                                    (uint64_t)N * 4, 32, 32, CU_TENSOR_MAP_SWIZZLE_128B))
      return rc;
  static std::atomic<uint64_t> configured[2] = {};  // per device
  static std::atomic<int> resident[kMaxDevices][split::kMaxCluster + 1];
  auto kern = i8gemm_kernel<false>;
  auto split_kern = i8gemm_kernel<true>;
  if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), kSmemBytes, configured[0])) return rc;
  if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(split_kern), kSmemBytes, configured[1])) return rc;
  const uint32_t idesc = dev::make_idesc(/*c=s32*/ 2, a_unsigned ? 0 : 1, b_unsigned ? 0 : 1,
                                         /*a K-major*/ 0, /*b MN-major*/ 1, BMB, BN);
  const int tiles = static_cast<int>(((M + 2 * BMB - 1) / (2 * BMB)) * ((N + BN - 1) / BN));
  const int ctas = gemm_ctas();
  const int halves = (tiles * 2 <= ctas) ? 1 : 0;  // few tiles: one row block per CTA
  const int items = tiles * (halves ? 2 : 1);
  const int grid = items < ctas ? items : ctas;
  const int blocks = static_cast<int>((M + BMB - 1) / BMB * ((N + BN - 1) / BN));
  int ks = 1;   // callers with a limit on the CTAs keep one to a block
  if (ctas == num_sms())
    ks = split_of(M, blocks, static_cast<int>((K + BK - 1) / BK),
                  [&](int n) { return split::resident_clusters(split_kern, kThreads, kSmemBytes, 1, n, resident); });
  if (ks > 1) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ks;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(ks, blocks);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    QMM_CUDA_TRY(cudaLaunchKernelEx(&cfg, split_kern, amap, bmap, accmap, outmap, acc, out, row_scale, col_scale, (int)M, (int)N,
                                    (int)K, idesc, 1, 0, device_status_word()));
    return QMM_OK;
  }
  static std::atomic<int> staged_cache{INT32_MIN};
  const int staged = env_int_once("QMM_I8_STAGED_STORE", 1, staged_cache);   // 0: results stored straight from registers
  kern<<<grid, kThreads, kSmemBytes, stream>>>(amap, bmap, accmap, outmap, acc, out, row_scale, col_scale,
                                                        (int)M, (int)N, (int)K, idesc, halves, staged,
                                                        device_status_word());
  QMM_CHECK_LAUNCH("i8gemm_kernel");
  return QMM_OK;
}

// How M x N is cut into tiles for `sms` CTAs: rows per tile (as few tiles as there may be, or up to three more, of equal
// height) and the parts of the tiles that are left after the last full round.  Parts pay where each CTA has one at most.
// The costs are a fit to 600 calls of a graph (M 64 to 3000, K 1024 to 14336, N 1536 to 28672, every cut: 4 to 6 % off in the
// mean): microseconds per 64 k of a whole tile and of one channel block, with a floor (the chain converter - MMA - converter of
// two stages in TMEM) and a slope per row, and per piece for its first stages and its results.  What they choose is 0.2 %
// slower than the best cut in the mean (4096 x 4096, M = 777, int4: 47 us; cut in quarters, which cost no fewer clocks, 72).
// Tiles, or channel blocks, that a share of the SMs holds go to clusters where that is estimated to be quicker; those costs are
// a fit to 3600 calls (M 33 to 512, K 512 to 14336, N 1024 to 14336, every cut and cluster size: 5 to 7 % off).
// `resident(ks)`: clusters of ks CTAs that the device holds at once, 0 where K must not be split.
template <typename Fn>
static tc::w8::Sched schedule(int64_t M, int64_t N, int64_t K, int wbits, int sms, Fn resident) {
  using namespace tc::w8;
  struct Cost { float floor, row, piece; };
  static constexpr Cost kWhole[2] = {{0.43f, 0.0030f, 6.6f}, {0.59f, 0.0033f, 5.9f}};   // int8, int4
  static constexpr Cost kBlock[2] = {{0.39f, 0.0022f, 5.0f}, {0.48f, 0.00265f, 4.8f}};
  static constexpr Cost kSplitWhole[2] = {{0.43f, 0.0027f, 5.6f}, {0.59f, 0.0032f, 5.2f}};
  static constexpr Cost kSplitBlock[2] = {{0.36f, 0.0021f, 5.9f}, {0.47f, 0.0025f, 5.6f}};
  constexpr float kSumCta = 0.18f, kSumRow = 0.036f;   // the sums: per CTA of a cluster, per row of 256 channels
  const float stages = static_cast<float>((K + BK - 1) / BK);
  auto us = [&](const Cost& c, int rows, int ks = 1) {
    const int share = (static_cast<int>(stages) + ks - 1) / ks;
    return (rows * c.row > c.floor ? rows * c.row : c.floor) * share + c.piece;
  };
  Sched best = {};
  float best_cost = -1.f;
  const int least = static_cast<int>((M + kMaxRows - 1) / kMaxRows);
  for (int tiles_m = least; tiles_m <= least + 3; ++tiles_m) {
    Sched sc = {};
    sc.tiles_n2 = static_cast<int>((N + 2 * BNW - 1) / (2 * BNW));
    sc.ks = 1;
    sc.rows = static_cast<int>(((M + tiles_m - 1) / tiles_m + 31) / 32 * 32);
    sc.tiles_m = static_cast<int>((M + sc.rows - 1) / sc.rows);
    const int tiles = sc.tiles_n2 * sc.tiles_m;
    sc.full_waves = tiles / sms;
    sc.tail_tiles = tiles - sc.full_waves * sms;
    // a panel of activation tiles (K bf16 a row) should fit in half of L2 (measured at K = 28672, N = 8192, tiles of 256 rows:
    // panels of 8 / 4 / 3 / 2 tiles give 1180 / 1218 / 1149 / 1134 TFLOP/s)
    const long long tile_bytes = 2ll * sc.rows * K;
    const long long pt = (64ll << 20) / (tile_bytes > 0 ? tile_bytes : 1);
    sc.panel = static_cast<int>(pt < 2 ? 2 : (pt > kPanelTiles ? kPanelTiles : pt));
    const float whole = us(kWhole[wbits == 4], sc.rows);
    for (sc.tail_div = 1; sc.tail_div <= 4; sc.tail_div *= 2) {
      if (sc.tail_div > 1 && (sc.tail_tiles == 0 || sc.tail_tiles * sc.tail_div > sms)) break;
      const float tail = sc.tail_tiles == 0 ? 0.f
                         : sc.tail_div == 1 ? whole
                                            : us(kBlock[wbits == 4], sc.tail_div == 2 ? sc.rows : sc.rows / 2);
      const float cost = sc.full_waves * whole + tail;
      if (best_cost < 0.f || cost < best_cost) {
        best_cost = cost;
        best = sc;
        best.cost = cost;
      }
    }
    // pieces that a share of the SMs holds at once: clusters of CTAs, each with a part of K
    sc.full_waves = 0;
    sc.tail_tiles = tiles;
    for (sc.tail_div = 1; sc.tail_div <= 2 && tiles * sc.tail_div <= sms / 2; sc.tail_div *= 2)
      for (sc.ks = 2; sc.ks <= split::kMaxCluster && sc.ks <= stages; ++sc.ks) {
        if (tiles * sc.tail_div * sc.ks > sms || tiles * sc.tail_div > resident(sc.ks)) break;
        const float cost = us((sc.tail_div == 1 ? kSplitWhole : kSplitBlock)[wbits == 4], sc.rows, sc.ks) + kSumCta * sc.ks +
                           kSumRow * sc.rows / sc.tail_div;
        if (cost < best_cost) {
          best_cost = cost;
          best = sc;
          best.cost = cost;
        }
      }
  }
  return best;
}

// Shared launch path of the weight-only GEMMs (int8 per-channel, int4 group-wise).
template <int WBITS>
static int launch_weight_only(const uint16_t* x, const void* w, const float* scale, const tc::w8::GroupQuant& gq,
                              uint16_t* y, int64_t M, int64_t N, int64_t K, int64_t ldy, uint32_t flags,
                              uint32_t* signal, uint32_t* arrive, cudaStream_t stream) {
  using namespace tc::w8;
  const int sms = gemm_ctas();  // persistent CTAs of a launch
  static std::atomic<int> resident[kMaxDevices][split::kMaxCluster + 1];
  static std::atomic<uint64_t> configured[4] = {};  // per device (one mask per instance of the kernel)
  decltype(&w8a16_kernel<WBITS, false, false>) kerns[2] = {w8a16_kernel<WBITS, false, false>, w8a16_kernel<WBITS, false, WBITS == 8>};
  decltype(&w8a16_kernel<WBITS, false, false>) split_kerns[2] = {w8a16_kernel<WBITS, true, false>, w8a16_kernel<WBITS, true, WBITS == 8>};
  for (int i = 0; i < 2; ++i) {
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kerns[i]), kSmemBytes, configured[i])) return rc;
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(split_kerns[i]), kSmemBytes, configured[2 + i])) return rc;
  }
  // results that go to several GPUs or are announced, and callers with a limit on the CTAs, keep one CTA to a piece
  const bool may_split = sms == num_sms() && !(flags & QMM_GEMM_STORE_MULTIMEM) && signal == nullptr;
  auto plan = [&](int64_t rows) {
    return schedule(rows, N, K, WBITS, sms, [&](int ks) {
      return may_split ? split::resident_clusters(split_kerns[0], kThreads, kSmemBytes, 1, ks, resident) : 0;
    });
  };
  Sched sc = plan(M), rest = {};
  // Few rounds of tiles that fill the SMs badly: the first rows go in one launch and the others in a second, which splits K where
  // its tiles are few, if that is estimated to be quicker by more than the estimate's error.  One launch, two: 14336 x 4096, M = 777
  // int8 108 -> 95 us, int4 138 -> 105; 8192 x 8192, M = 777 123 -> 99, 148 -> 112; 16128 x 5120, M = 1587 243 -> 204, 288 -> 232;
  // 4096 x 4096, M = 2048 68 -> 62, 81 -> 70.  The worst of 200 calls (M 400 to 3333) is 2 % slower (4096 x 6144, M = 2048 80.4,
  // 82.2).  Below 50 us the second launch costs too much (2048 x 11264, M = 640, int4 47.7, 51.3), and with more than three rounds
  // the gaps are small and the estimate is off by as much (5120 x 32256, M = 2048, int4 626, 682).  Independent launches fill one
  // another's gaps and stay whole.
  int64_t first = M;
  if (may_split && !(flags & QMM_GEMM_INDEPENDENT) && sc.full_waves <= 3 && sc.cost > 50.f) {
    const int64_t tiles_m = (M + kMaxRows - 1) / kMaxRows;
    float best = 0.96f * sc.cost;
    for (int64_t t = tiles_m > 6 ? tiles_m - 5 : 1; t < tiles_m; ++t) {
      const Sched head = plan(t * kMaxRows), tail = plan(M - t * kMaxRows);
      if (head.cost + tail.cost + 2.f < best) {
        best = head.cost + tail.cost + 2.f;
        first = t * kMaxRows;
        sc = head;
        rest = tail;
      }
    }
  }
  auto launch = [&](const Sched& sc, int64_t row, int64_t rows) -> int {
    uint16_t* out = y + row * ldy;
    CUtensorMap wmap, xmap;
    constexpr int kRawRows = (WBITS == 8) ? BK : BK / 2;
    if (int rc = make_tensor_map_2d(&wmap, w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)(WBITS == 8 ? K : K / 2),
                                    (uint64_t)N, (uint64_t)N, kRawRows, BNW, CU_TENSOR_MAP_SWIZZLE_128B))
      return rc;
    if (int rc = make_tensor_map_2d(&xmap, x + row * K, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)rows,
                                    (uint64_t)K, (uint64_t)K * 2, sc.rows, BK, CU_TENSOR_MAP_SWIZZLE_128B))
      return rc;
    // operand "a" of the MMA = weights (bf16, from TMEM), "b" = activations (bf16, K-major)
    const uint32_t idesc_full = dev::make_idesc(/*c=f32*/ 1, /*bf16*/ 1, /*bf16*/ 1, 0, /*b K-major*/ 0, BNW, sc.rows);
    const uint32_t idesc_half = dev::make_idesc(1, 1, 1, 0, 0, BNW, sc.rows / 2);
    const bool parts = WBITS == 8 && 2 * sc.rows <= kMaxRows && (K + BK - 1) / BK > static_cast<int64_t>(kLeastPart) * sc.ks;
    if (sc.ks > 1) {
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute attr[2];
      cfg.gridDim = dim3(sc.ks, sc.tail_tiles * sc.tail_div);
      cfg.blockDim = dim3(kThreads);
      cfg.dynamicSmemBytes = kSmemBytes;
      cfg.stream = stream;
      split::set_attrs(cfg, attr, sc.ks);
      QMM_CUDA_TRY(cudaLaunchKernelEx(&cfg, split_kerns[parts], wmap, xmap, scale, gq, out, (int)rows, (int)N, (int)K, (long long)ldy, idesc_full,
                                      idesc_half, sc, flags, signal, arrive, device_status_word()));
      return QMM_OK;
    }
    const int grid = sc.full_waves > 0 ? sms : (sc.tail_tiles * sc.tail_div < sms ? sc.tail_tiles * sc.tail_div : sms);
    // Programmatic stream serialization: the CTAs of this launch may become resident while the
    // kernel ahead of it drains; they order themselves behind it inside the kernel (or not at all
    // when the caller states independence, which fills the last, partly idle round of one launch
    // with the first tiles of the next).
    QMM_CUDA_TRY(launch_pdl(kerns[parts], dim3(grid), dim3(kThreads), kSmemBytes, stream, wmap, xmap, scale, gq, out, (int)rows,
                            (int)N, (int)K, (long long)ldy, idesc_full, idesc_half, sc, flags, signal, arrive,
                            device_status_word()));
    return QMM_OK;
  };
  if (int rc = launch(sc, 0, first)) return rc;
  return first < M ? launch(rest, first, M - first) : QMM_OK;
}

int w8a16_tcgen05(const uint16_t* x, const int8_t* w, const float* scale, uint16_t* y, int64_t M,
                  int64_t N, int64_t K, int64_t ldy, uint32_t flags, uint32_t* signal, uint32_t* arrive,
                  cudaStream_t stream) {
  const tc::w8::GroupQuant none = {nullptr, nullptr, 0};
  return launch_weight_only<8>(x, w, scale, none, y, M, N, K, ldy, flags, signal, arrive, stream);
}

// int4 g128 weight-only GEMM for prefill-sized M: same pipeline, nibbles dequantised by the
// converter warps.  Requires K % 128 == 0 and N % 128 == 0 (checked by the caller).
int w4a16_tcgen05(const uint16_t* x, const uint8_t* wq, const uint16_t* scales, const uint8_t* zeros,
                  int zeros_packed, uint16_t* y, int64_t M, int64_t N, int64_t K, uint32_t flags,
                  cudaStream_t stream) {
  const tc::w8::GroupQuant gq = {scales, zeros, zeros_packed};
  return launch_weight_only<4>(x, wq, nullptr, gq, y, M, N, K, N, flags, nullptr, nullptr, stream);
}

}  // namespace qmm
