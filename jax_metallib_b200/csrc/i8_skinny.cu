// int8 x int8 -> int32 dot for few rows, and for rows that TMA cannot describe (sm_100a).
//
//   acc[M,N] = a[M,K] . b[K,N]      exact, wrapping like the int32 accumulator of the reference
//   out[M,N] = float(acc) * row[m] * col[n]
//
// The layout of the int8 weight-only kernel: a cluster of KS CTAs owns tiles of 128 columns x MT * 8 rows and splits K,
// the ring of 64-k stages runs on over the tiles, ldmatrix.trans turns b's rows into registers with four k of one
// column, and mma.sync.m16n8k32 takes b as its 16-row operand and a as its 8-column operand.  The partial tiles of the
// cluster meet in distributed shared memory.
//
// Row pitches that are no multiple of 16 bytes (K or N odd, a view at an odd offset) have no tensor map.  Where they and
// the addresses are multiples of 8, loader warps copy pieces of 8 or 16 bytes asynchronously to where TMA would have put
// them, a whole ring of stages ahead.  Elsewhere they fetch the aligned 32-bit words around each 16-byte piece, shift the
// bytes into place and store the piece, with the next stage's words on their way.  Only words that hold a byte of the tensor
// are read.
// Measured (shifted words, copies): 65 x 2048 x 1000 13.1, 11.4 us (9.8 with 1024 columns, by TMA); 1000 x 2056 x 2056 69, 53 us.
// Pieces of 4 bytes lost where there is more to do (33 x 4100 x 4100 19.9, 22.8 us).  Shifted words (one thread per result before, without the
// prefetch, now): 64 x 4095 x 4097 437, 63, 26 us; 4000 x 4097 x 4095 22.7 ms, 2.0 ms, 0.86 ms; bound by their loads: five
// per 16 bytes.
#include <cooperative_groups.h>

#include "split_k.cuh"

namespace cg = cooperative_groups;

namespace qmm {
namespace i8s {

using namespace split;

constexpr int kCols = 128;           // columns per tile
constexpr int kBK = 64;              // k per stage
constexpr int kConsumerWarps = 8;    // 4 column groups of 32 x 2 halves of a stage's k
constexpr int kLoaderWarps = 4;      // rows without a tensor map
constexpr int kWBytes = kBK * kCols;

template <int MT, bool TMA>
struct Smem {
  static constexpr int kX = MT * 8 * kBK;                  // a's part of a stage: [MT * 8 rows][64 bytes], TMA's 64-byte swizzle
  static constexpr int kStage = kWBytes + (kX < 1024 ? 1024 : kX);
  static constexpr int kPerSm = MT == 8 ? 1 : 2;           // 64 accumulators a thread at MT = 8
  static constexpr int kReducers = 3;                      // warps that add the partial tiles
  static constexpr int kProducers = TMA ? 1 : kLoaderWarps;
  static constexpr int kFirstReducer = kConsumerWarps + kProducers;
  static constexpr int kThreads = (kFirstReducer + kReducers) * 32;
  static constexpr int kStages = MT == 1 ? 8 : 6;
  static constexpr int kPartBufs = MT <= 2 ? 2 : 1;        // tiles whose partial results may be in flight
  static constexpr int kPart = MT * 8 * kCols * 4;         // partial tile of one k half
  static constexpr int kOffPart = kStages * kStage;
  static constexpr int kOffBar = kOffPart + kPartBufs * 2 * kPart;
  static constexpr int kTotal = kOffBar + (2 * kStages + 2 * kPartBufs) * 8 + 1024;  // + alignment slack
  static_assert(kPerSm * (kTotal + 1024) <= 228 * 1024, "resident CTAs");
};

template <bool AU, bool BU>
__device__ __forceinline__ void mma_i8(int (&d)[4], uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3, uint32_t x0, uint32_t x1) {
#define QMM_MMA_I8(TB, TA)                                                                                              \
  asm("mma.sync.aligned.m16n8k32.row.col.s32." TB "." TA ".s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};" \
      : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])                                                                  \
      : "r"(w0), "r"(w1), "r"(w2), "r"(w3), "r"(x0), "r"(x1))
  if (BU && AU) QMM_MMA_I8("u8", "u8");
  else if (BU) QMM_MMA_I8("u8", "s8");
  else if (AU) QMM_MMA_I8("s8", "u8");
  else QMM_MMA_I8("s8", "s8");
#undef QMM_MMA_I8
}

// The 16 bytes at p, of which only those before `end` are wanted, on their way: five aligned words, none of them without a
// wanted byte.  get() shifts them into place.
struct Piece {
  uint32_t w[5], shift;
  __device__ __forceinline__ void load(const uint8_t* p, const uint8_t* end) {
    const uint32_t off = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(p) & 3);
    const uint32_t* q = reinterpret_cast<const uint32_t*>(p - off);
    shift = off * 8;
#pragma unroll
    for (int i = 0; i < 5; ++i)
      w[i] = (reinterpret_cast<const uint8_t*>(q + i) < end && (i < 4 || off != 0)) ? __ldg(q + i) : 0u;
  }
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < 5; ++i) w[i] = 0u;
    shift = 0;
  }
  __device__ __forceinline__ uint4 get() const {
    return make_uint4(__funnelshift_r(w[0], w[1], shift), __funnelshift_r(w[1], w[2], shift), __funnelshift_r(w[2], w[3], shift),
                      __funnelshift_r(w[3], w[4], shift));
  }
};

// Copies a stage's [ROWS][BYTES] part in pieces of W bytes by the 128 loader threads: rows row0 + r, columns col0 + c of a
// tensor of `rows` x `cols` bytes whose pitch, address and col0 are multiples of W; zeros beyond its ends.  place(r, c): offset
// of a byte in the stage.
template <int W, int ROWS, int BYTES, typename Place>
__device__ __forceinline__ void copy_pieces(uint32_t dst, const uint8_t* src, int row0, int rows, int col0, int cols, int lt, Place place) {
  constexpr int kPer = BYTES / W, kStep = kLoaderWarps * 32 / kPer;
  const int c = (lt % kPer) * W;
#pragma unroll 4
  for (int r = lt / kPer; r < ROWS; r += kStep) {
    const bool in = row0 + r < rows && col0 + c < cols;
    const uint8_t* from = in ? src + static_cast<size_t>(row0 + r) * cols + col0 + c : src;
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst + place(r, c)), "l"(from), "n"(W), "r"(in ? W : 0) : "memory");
  }
}
template <int ROWS, int BYTES, typename Place>
__device__ __forceinline__ void copy_part(int w, uint32_t dst, const uint8_t* src, int row0, int rows, int col0, int cols, int lt, Place place) {
  if (w == 16) copy_pieces<16, ROWS, BYTES>(dst, src, row0, rows, col0, cols, lt, place);
  else copy_pieces<8, ROWS, BYTES>(dst, src, row0, rows, col0, cols, lt, place);
}

// LOAD: how a stage arrives.
enum Load { kWords, kPieces, kTma };
template <int MT, bool AU, bool BU, Load LOAD>
__global__ void __launch_bounds__(Smem<MT, LOAD == kTma>::kThreads, Smem<MT, LOAD == kTma>::kPerSm)
i8_skinny_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap, const uint8_t* __restrict__ a,
                 const uint8_t* __restrict__ b, int32_t* __restrict__ acc_out, float* __restrict__ out,
                 const float* __restrict__ row_scale, const float* __restrict__ col_scale, int M, int N, int K, int stages_total,
                 int pairs, int a_piece, int b_piece, int* status) {
  constexpr bool TMA = LOAD == kTma;
  using L = Smem<MT, TMA>;
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

  if (threadIdx.x == 0) {
    if (TMA) {
      dev::tma_prefetch_desc(&wmap);
      dev::tma_prefetch_desc(&xmap);
    }
    for (int s = 0; s < S; ++s) {
      dev::mbar_init(&full[s], TMA ? 1 : kLoaderWarps * (LOAD == kPieces ? 32 : 1));
      dev::mbar_init(&empty[s], kConsumerWarps);
    }
    for (int b = 0; b < PB; ++b) {
      dev::mbar_init(&ready[b], KS * kConsumerWarps);
      dev::mbar_init(&vacant[b], KS * L::kReducers);
    }
    dev::fence_mbar_init();
  }
  cluster.sync();   // barriers of every CTA are initialised before a peer arrives on them
  dev::pdl_wait();
  dev::pdl_launch_dependents();

  if (warp >= kConsumerWarps && warp < L::kFirstReducer) {
    // ------------------------------ producers -----------------------------
    int n = 0;   // stages issued
    bool ok = true;
    if (TMA) {
      if (lane == 0) {
        const uint64_t policy = dev::policy_evict_first();
        for (int t = blockIdx.y; ok && t < tiles; t += gridDim.y) {
          const int col0 = (t / row_tiles) * kCols, row0 = (t % row_tiles) * MT * 8;
          for (int it = it_begin; it < it_end; ++it, ++n) {
            const int s = n % S;
            if (!dev::mbar_wait_relaxed(&empty[s], ((n / S) & 1) ^ 1, status, 110)) { ok = false; break; }
            uint8_t* st = smem + s * L::kStage;
            dev::mbar_expect_tx(&full[s], kWBytes + L::kX);   // rows and columns past the ends arrive as zeros
            if (row_tiles == 1) dev::tma_load_2d_hint(st, &wmap, &full[s], col0, it * kBK, policy);
            else dev::tma_load_2d(st, &wmap, &full[s], col0, it * kBK);   // the next row tile reads them again
            dev::tma_load_2d(st + kWBytes, &xmap, &full[s], it * kBK, row0);
          }
        }
        // no copy may still be on its way into this CTA's shared memory when it leaves, whatever the consumers did
        for (int i = n > S ? n - S : 0; i < n; ++i)
          if (!dev::mbar_wait_relaxed(&full[i % S], (i / S) & 1, status, 111)) break;
      }
      __syncwarp();
    } else if (LOAD == kPieces) {
      const int lt = threadIdx.x - kConsumerWarps * 32;   // 0 .. 127
      for (int t = blockIdx.y; ok && t < tiles; t += gridDim.y) {
        const int col0 = (t / row_tiles) * kCols, row0 = (t % row_tiles) * MT * 8;
        for (int it = it_begin; it < it_end; ++it, ++n) {
          const int s = n % S;
          if (!dev::mbar_wait_relaxed_warp(&empty[s], ((n / S) & 1) ^ 1, status, 110)) { ok = false; break; }
          const uint32_t st = dev::smem_u32(smem + s * L::kStage);
          copy_part<kBK, kCols>(b_piece, st, b, it * kBK, K, col0, N, lt,
                                [](int r, int c) { return r * 128 + (((c >> 4) ^ (r & 7)) << 4) + (c & 15); });
          copy_part<MT * 8, kBK>(a_piece, st + kWBytes, a, row0, M, it * kBK, K, lt,
                                 [](int r, int c) { return r * 64 + (((c >> 4) ^ ((r >> 1) & 3)) << 4) + (c & 15); });
          asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(dev::smem_u32(&full[s])) : "memory");
        }
      }
      // no copy may still be on its way into this CTA's shared memory when it leaves
      asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
      const int lt = threadIdx.x - kConsumerWarps * 32;   // 0 .. 127
      const uint8_t* a_end = a + static_cast<size_t>(M) * K;
      const uint8_t* b_end = b + static_cast<size_t>(K) * N;
      // The words of the next stage are requested before this one is stored.
      constexpr int kXP = (MT * 32 + 127) / 128;
      const int len = it_end - it_begin;
      const int mine = blockIdx.y < tiles ? (tiles - 1 - static_cast<int>(blockIdx.y)) / static_cast<int>(gridDim.y) + 1 : 0;
      Piece v[4], x[kXP];
      auto request = [&](int t, int it) {
        const int col0 = (t / row_tiles) * kCols, row0 = (t % row_tiles) * MT * 8;
        // b: rows lt / 8 + 16 i, 16 columns each; rows past K are zeros, so that what a's rows hold past K does not count
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int k = it * kBK + (lt >> 3) + i * 16, c = col0 + (lt & 7) * 16;
          if (k < K && c < N) v[i].load(b + static_cast<size_t>(k) * N + c, b_end);
          else v[i].zero();
        }
#pragma unroll
        for (int i = 0; i < kXP; ++i) {
          const int r = (lt >> 2) + i * 32, k = it * kBK + (lt & 3) * 16;
          if (r < MT * 8 && row0 + r < M && k < K) x[i].load(a + static_cast<size_t>(row0 + r) * K + k, a_end);
          else x[i].zero();
        }
      };
      int t = blockIdx.y, it = it_begin;
      const int total = mine * len;
      if (total > 0) request(t, it);
      for (; n < total; ++n) {
        const int s = n % S;
        uint4 vs[4], xs[kXP];
#pragma unroll
        for (int i = 0; i < 4; ++i) vs[i] = v[i].get();
#pragma unroll
        for (int i = 0; i < kXP; ++i) xs[i] = x[i].get();
        if (++it == it_end) {
          it = it_begin;
          t += gridDim.y;
        }
        if (n + 1 < total) request(t, it);
        if (!dev::mbar_wait_relaxed_warp(&empty[s], ((n / S) & 1) ^ 1, status, 110)) break;
        uint8_t* st = smem + s * L::kStage;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = (lt >> 3) + i * 16;
          *reinterpret_cast<uint4*>(st + r * 128 + (((lt & 7) ^ (r & 7)) << 4)) = vs[i];
        }
#pragma unroll
        for (int i = 0; i < kXP; ++i) {
          const int r = (lt >> 2) + i * 32;
          if (r < MT * 8) *reinterpret_cast<uint4*>(st + kWBytes + r * 64 + (((lt & 3) ^ ((r >> 1) & 3)) << 4)) = xs[i];
        }
        __syncwarp();
        if (lane == 0) dev::mbar_arrive(&full[s]);
      }
    }
  } else if (warp < kConsumerWarps) {
    // ------------------------------ consumers -----------------------------
    const int cgrp = warp & 3, kh = warp >> 2;
    const int g8 = lane >> 2, t4 = lane & 3;
    // b: a thread's register holds four neighbouring k of one column, k = 4 t4 .. of the first and 16 + 4 t4 .. of the
    // second half of the warp's 32 k: matrix m of an ldmatrix has the k rows {4i, 4i + 1} or {4i + 2, 4i + 3} of one half
    const int w_k = kh * 32 + (lane >> 4) * 16 + ((lane & 7) >> 1) * 4 + (lane & 1) + ((lane >> 3) & 1) * 2;
    const uint32_t w_off0 = w_k * 128 + (((2 * cgrp) ^ (w_k & 7)) << 4);
    const uint32_t w_off1 = w_k * 128 + (((2 * cgrp + 1) ^ (w_k & 7)) << 4);
    // a: row g8, bytes 4 t4 of the two 16-byte chunks of the warp's k half (chunks XOR-swizzled by bits 1-2 of the row)
    const uint32_t x_row = kWBytes + g8 * 64 + t4 * 4;
    const uint32_t x_off0 = x_row + (((2 * kh) ^ ((g8 >> 1) & 3)) << 4), x_off1 = x_row + (((2 * kh + 1) ^ ((g8 >> 1) & 3)) << 4);
    const uint32_t ring = dev::smem_u32(smem);
    int s = 0;
    uint32_t ph = 0;
    int tile = 0;
    bool ok = true;
    const int never = stages_total < 0;   // false, but not to the compiler
    for (int t = blockIdx.y; t < tiles; t += gridDim.y, ++tile) {
      int acc[2][MT][4];
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[j][mt][i] = 0;
      for (int it = it_begin; it < it_end; ++it) {
        if (!dev::mbar_wait_relaxed_warp(&full[s], ph, status, 112)) { ok = false; break; }
        const uint32_t st = ring + s * L::kStage;
        uint32_t wr[2][4];
        ldmatrix_x4_trans(st + w_off0, wr[0]);
        ldmatrix_x4_trans(st + w_off1, wr[1]);
        uint32_t dep = wr[0][3] ^ wr[1][3];
        uint32_t xr[MT][2];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          asm volatile("ld.shared.u32 %0, [%1];" : "=r"(xr[mt][0]) : "r"(st + x_off0 + mt * 512));
          asm volatile("ld.shared.u32 %0, [%1];" : "=r"(xr[mt][1]) : "r"(st + x_off1 + mt * 512));
          dep ^= xr[mt][0] ^ xr[mt][1];
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          // registers 2h, 2h + 1: k 4t, 4t + 1 and 4t + 2, 4t + 3 of half h, columns 2 g8 (even bytes) and 2 g8 + 1
          const uint32_t w0 = __byte_perm(wr[j][0], wr[j][1], 0x6420), w1 = __byte_perm(wr[j][0], wr[j][1], 0x7531);
          const uint32_t w2 = __byte_perm(wr[j][2], wr[j][3], 0x6420), w3 = __byte_perm(wr[j][2], wr[j][3], 0x7531);
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) mma_i8<AU, BU>(acc[j][mt], w0, w1, w2, w3, xr[mt][0], xr[mt][1]);
        }
        release_slot(&empty[s], dep, never, lane);
        if (++s == S) { s = 0; ph ^= 1; }
      }
      if (!ok) break;
      // ---- hand the partial tile over to the reducers of the cluster
      const int b = tile % PB;
      if (tile >= PB && !wait_cluster_warp(&vacant[b], ((tile / PB) & 1) ^ 1, status, 113)) break;
      int* part = reinterpret_cast<int*>(smem + L::kOffPart + b * 2 * L::kPart);
      int* mine = part + kh * (L::kPart / 4);
      // rows 2 t4, 2 t4 + 1 of columns 2 g8, 2 g8 + 1 of each 16-column block
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int r = 0; r < 2; ++r)
            *reinterpret_cast<int2*>(mine + (mt * 8 + 2 * t4 + r) * kCols + cgrp * 32 + j * 16 + 2 * g8) =
                make_int2(acc[j][mt][r], acc[j][mt][2 + r]);
      __syncwarp();
      if (lane < KS) arrive_remote(&ready[b], lane);
    }
  } else {
    // ------------------------------ reducers ------------------------------
    // CTA `rank` adds every KS-th run of column pairs, in CTA order
    constexpr int kR = L::kReducers * 32;
    const int tid = threadIdx.x - L::kFirstReducer * 32;
    int tile = 0;
    for (int t = blockIdx.y; t < tiles; t += gridDim.y, ++tile) {
      const int b = tile % PB;
      const int* part = reinterpret_cast<const int*>(smem + L::kOffPart + b * 2 * L::kPart);
      if (!wait_cluster_warp(&ready[b], (tile / PB) & 1, status, 114)) break;
      const int col0 = (t / row_tiles) * kCols, row0 = (t % row_tiles) * MT * 8;
      const int rows = min(MT * 8, M - row0);
      for (int e = rank * kR + tid; e < rows * (kCols / 2); e += KS * kR) {
        const int m = e / (kCols / 2), c = (e % (kCols / 2)) * 2;
        if (col0 + c >= N) continue;
        int2 lo[kMaxCluster], hi[kMaxCluster];
#pragma unroll
        for (int r = 0; r < kMaxCluster; ++r)
          if (r < KS) {
            const int* p = cluster.map_shared_rank(part, r) + m * kCols + c;
            lo[r] = *reinterpret_cast<const int2*>(p);
            hi[r] = *reinterpret_cast<const int2*>(p + L::kPart / 4);
          }
        uint32_t v0 = 0, v1 = 0;   // wraps mod 2^32
#pragma unroll
        for (int r = 0; r < kMaxCluster; ++r)
          if (r < KS) {
            v0 += static_cast<uint32_t>(lo[r].x) + static_cast<uint32_t>(hi[r].x);
            v1 += static_cast<uint32_t>(lo[r].y) + static_cast<uint32_t>(hi[r].y);
          }
        const size_t i = static_cast<size_t>(row0 + m) * N + col0 + c;
        const bool second = col0 + c + 1 < N;
        if (acc_out) {
          if (pairs) *reinterpret_cast<int2*>(acc_out + i) = make_int2(static_cast<int>(v0), static_cast<int>(v1));
          else {
            acc_out[i] = static_cast<int>(v0);
            if (second) acc_out[i + 1] = static_cast<int>(v1);
          }
        }
        if (out) {
          const float rs = __ldg(row_scale + row0 + m);
          const float o0 = static_cast<float>(static_cast<int>(v0)) * rs * __ldg(col_scale + col0 + c);
          const float o1 = second ? static_cast<float>(static_cast<int>(v1)) * rs * __ldg(col_scale + col0 + c + 1) : 0.f;
          if (pairs) *reinterpret_cast<float2*>(out + i) = make_float2(o0, o1);
          else {
            out[i] = o0;
            if (second) out[i + 1] = o1;
          }
        }
      }
      __syncwarp();
      if (lane < KS) arrive_remote(&vacant[b], lane);
    }
  }
  cluster.sync();   // peers keep their shared memory alive until it has been read
}

struct Args {
  const uint8_t *a, *b;
  int32_t* acc;
  float* out;
  const float *rs, *cs;
  int M, N, K;
};

// The largest piece that a pitch and an address are made of, 8 or 16 bytes, or 0.
static int piece(const uint8_t* at, int pitch) {
  const uintptr_t bits = reinterpret_cast<uintptr_t>(at) | static_cast<uintptr_t>(pitch);
  return bits % 16 == 0 ? 16 : bits % 8 == 0 ? 8 : 0;
}

template <int MT, bool AU, bool BU, Load LOAD>
static int launch(const Args& p, cudaStream_t stream) {
  constexpr bool TMA = LOAD == kTma;
  using L = Smem<MT, TMA>;
  CUtensorMap wmap = {}, xmap = {};
  if (TMA) {
    if (int rc = make_tensor_map_2d(&wmap, p.b, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)p.K, (uint64_t)p.N, (uint64_t)p.N, kBK,
                                    kCols, CU_TENSOR_MAP_SWIZZLE_128B))
      return rc;
    if (int rc = make_tensor_map_2d(&xmap, p.a, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)p.M, (uint64_t)p.K, (uint64_t)p.K,
                                    MT * 8, kBK, CU_TENSOR_MAP_SWIZZLE_64B))
      return rc;
  }
  static std::atomic<uint64_t> configured{0};  // per device (one mask per template instance)
  static std::atomic<int> resident[kMaxDevices][kMaxCluster + 1];
  auto kern = i8_skinny_kernel<MT, AU, BU, LOAD>;
  if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), L::kTotal, configured)) return rc;
  const int stages_total = (p.K + kBK - 1) / kBK;
  // a limit leaves SMs to a collective: one CTA to each of the others
  const int limit = gemm_ctas() < num_sms() ? gemm_ctas() : INT_MAX;
  const Grid g = choose_grid(((p.N + kCols - 1) / kCols) * ((p.M + MT * 8 - 1) / (MT * 8)), stages_total, [&](int ks) {
    return resident_clusters(kern, L::kThreads, L::kTotal, L::kPerSm, ks, resident);
  }, limit);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  cfg.gridDim = dim3(g.ks, g.clusters);
  cfg.blockDim = dim3(L::kThreads);
  cfg.dynamicSmemBytes = L::kTotal;
  cfg.stream = stream;
  set_attrs(cfg, attr, g.ks);
  const int pairs = p.N % 2 == 0 && aligned(p.acc, 8) && aligned(p.out, 8);
  QMM_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, wmap, xmap, p.a, p.b, p.acc, p.out, p.rs, p.cs, p.M, p.N, p.K, stages_total, pairs,
                                  piece(p.a, p.K), piece(p.b, p.N), device_status_word()));
  return QMM_OK;
}

template <bool AU, bool BU, Load LOAD>
static int launch_rows(const Args& p, cudaStream_t stream) {
  if (p.M <= 8) return launch<1, AU, BU, LOAD>(p, stream);
  if (p.M <= 16) return launch<2, AU, BU, LOAD>(p, stream);
  if (p.M <= 32) return launch<4, AU, BU, LOAD>(p, stream);
  return launch<8, AU, BU, LOAD>(p, stream);
}
template <Load LOAD>
static int launch_types(const Args& p, int au, int bu, cudaStream_t stream) {
  if (au) return bu ? launch_rows<true, true, LOAD>(p, stream) : launch_rows<true, false, LOAD>(p, stream);
  return bu ? launch_rows<false, true, LOAD>(p, stream) : launch_rows<false, false, LOAD>(p, stream);
}

}  // namespace i8s

// Any M, N, K >= 1 and any alignment; aligned_rows: K and N multiples of 16, a and b 16-byte aligned.
int i8_skinny(const void* a, const void* b, int32_t* acc, const float* row_scale, const float* col_scale, float* out, int64_t M,
              int64_t N, int64_t K, int a_unsigned, int b_unsigned, bool aligned_rows, cudaStream_t stream) {
  const i8s::Args p = {static_cast<const uint8_t*>(a), static_cast<const uint8_t*>(b), acc, out, row_scale, col_scale,
                       static_cast<int>(M), static_cast<int>(N), static_cast<int>(K)};
  if (aligned_rows) return i8s::launch_types<i8s::kTma>(p, a_unsigned, b_unsigned, stream);
  // one operand without pieces: shifted words for both
  if (i8s::piece(p.a, p.K) && i8s::piece(p.b, p.N)) return i8s::launch_types<i8s::kPieces>(p, a_unsigned, b_unsigned, stream);
  return i8s::launch_types<i8s::kWords>(p, a_unsigned, b_unsigned, stream);
}

}  // namespace qmm
