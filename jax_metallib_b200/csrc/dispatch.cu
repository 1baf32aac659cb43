// Entry points whose work is routed between the tcgen05 GEMMs, the mma.sync
// kernels that split K (few rows; int8 dots of any alignment) and plain
// CUDA-core kernels, which are left for weight-only shapes that TMA cannot
// describe (16-byte row pitches) and for K = 0.
// Both routes are GPU code; there is no host fallback.
#include <stddef.h>
#include <stdlib.h>
#include <string.h>

#include "common.cuh"

namespace qmm {

int i8gemm_tcgen05(const void* a, const void* b, int32_t* acc, const float* row_scale,
                   const float* col_scale, float* out, int64_t M, int64_t N, int64_t K,
                   int a_unsigned, int b_unsigned, cudaStream_t stream);
int w8a16_tcgen05(const uint16_t* x, const int8_t* w, const float* scale, uint16_t* y, int64_t M,
                  int64_t N, int64_t K, int64_t ldy, uint32_t flags, uint32_t* signal, uint32_t* arrive,
                  cudaStream_t stream);
int i8_skinny(const void* a, const void* b, int32_t* acc, const float* row_scale, const float* col_scale, float* out, int64_t M,
              int64_t N, int64_t K, int a_unsigned, int b_unsigned, bool aligned_rows, cudaStream_t stream);
int w8a16_decode(const uint16_t* x, const int8_t* w, const float* scale, uint16_t* y, int64_t M, int64_t N, int64_t K,
                 int64_t ldy, uint32_t flags, cudaStream_t stream);

namespace simple {

template <bool AU, bool BU>
__global__ void i8dot_kernel(const uint8_t* __restrict__ a, const uint8_t* __restrict__ b,
                             int32_t* __restrict__ acc, float* __restrict__ out,
                             const float* __restrict__ rs, const float* __restrict__ cs, int M, int N,
                             int K) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  const int m = blockIdx.y;
  if (n >= N || m >= M) return;
  int32_t s = 0;  // wraps mod 2^32 like the reference's int32 accumulator
  for (int k = 0; k < K; ++k) {
    const int av = AU ? static_cast<int>(a[static_cast<size_t>(m) * K + k])
                      : static_cast<int>(static_cast<int8_t>(a[static_cast<size_t>(m) * K + k]));
    const int bv = BU ? static_cast<int>(b[static_cast<size_t>(k) * N + n])
                      : static_cast<int>(static_cast<int8_t>(b[static_cast<size_t>(k) * N + n]));
    s = static_cast<int32_t>(static_cast<uint32_t>(s) + static_cast<uint32_t>(av * bv));
  }
  if (acc) acc[static_cast<size_t>(m) * N + n] = s;
  if (out) out[static_cast<size_t>(m) * N + n] = static_cast<float>(s) * rs[m] * cs[n];
}

__global__ void w8a16_kernel(const uint16_t* __restrict__ x, const int8_t* __restrict__ w,
                             const float* __restrict__ scale, uint16_t* __restrict__ y, int M, int N,
                             int K, long long ldy) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  const int m = blockIdx.y;
  if (n >= N || m >= M) return;
  float s = 0.f;
  for (int k = 0; k < K; ++k)
    s = fmaf(dev::bf16_bits_to_float(x[static_cast<size_t>(m) * K + k]),
             static_cast<float>(w[static_cast<size_t>(k) * N + n]), s);
  y[static_cast<size_t>(m) * ldy + n] = dev::float_to_bf16_bits(s * scale[n]);
}

// One thread per word: wait (bounded) until words[i] >= expected.  The words are written by other
// GPUs (the completion signals of a sharded linear), never by a kernel sharing this GPU.
__global__ void wait_words_kernel(const uint32_t* words, int count, uint32_t expected, unsigned long long limit_ns,
                                  int* status) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const uint64_t t0 = dev::globaltimer_ns();
  while (true) {
    // counts wrap: "reached" means no more than 2^31 behind
    if (static_cast<int32_t>(dev::ld_acquire_sys_u32(words + i) - expected) >= 0) return;
    if (dev::globaltimer_ns() - t0 > limit_ns) break;
    __nanosleep(200);
  }
  if (status) atomicExch(status, (60 << 16) | QMM_ERR_TIMEOUT);
}

// Local block -> multicast address, 16 bytes per thread, four loads in flight per thread; the last CTA to finish
// publishes the completion count on every rank (tag of the bounded wait that reads it: 60).
__global__ void __launch_bounds__(512)
multicast_copy_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst_mc, size_t n16, uint32_t* signal_mc,
                      uint32_t* arrive) {
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  for (; i + 3 * stride < n16; i += 4 * stride) {
    uint4 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = src[i + j * stride];
#pragma unroll
    for (int j = 0; j < 4; ++j) dev::multimem_st_v4_b32(dst_mc + i + j * stride, v[j]);
  }
  for (; i < n16; i += stride) dev::multimem_st_v4_b32(dst_mc + i, src[i]);
  dev::fence_sys();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned prev = atomicInc(arrive, gridDim.x - 1);
    if (prev == gridDim.x - 1) {
      dev::fence_sys();
      dev::multimem_red_release_add_u32(signal_mc, 1u);
    }
  }
}

struct PeerList {
  uint4* dst[QMM_MAX_PEERS];
  uint32_t* signal[QMM_MAX_PEERS];
  int n;
};
// Local block -> the same block of every peer's buffer by plain stores over NVLink (no copy to this GPU).
__global__ void __launch_bounds__(512)
peer_copy_kernel(const uint4* __restrict__ src, PeerList peers, size_t n16, uint32_t* local_signal, uint32_t* arrive) {
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  for (; i + 3 * stride < n16; i += 4 * stride) {
    uint4 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = src[i + j * stride];
    for (int p = 0; p < peers.n; ++p) {
#pragma unroll
      for (int j = 0; j < 4; ++j) __stcg(peers.dst[p] + i + j * stride, v[j]);
    }
  }
  for (; i < n16; i += stride) {
    const uint4 v = src[i];
    for (int p = 0; p < peers.n; ++p) __stcg(peers.dst[p] + i, v);
  }
  dev::fence_sys();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned prev = atomicInc(arrive, gridDim.x - 1);
    if (prev == gridDim.x - 1) {
      dev::fence_sys();
      for (int p = 0; p < peers.n; ++p) dev::red_release_sys_add_u32(peers.signal[p], 1u);
      dev::red_release_sys_add_u32(local_signal, 1u);
    }
  }
}

}  // namespace simple

// QMM_FORCE_SIMPLE=1 routes every shape to the CUDA-core kernels (a cross-check of the tensor-core
// route on a GPU box); read once per process.
static int force_simple() {
  static std::atomic<int> cache{INT32_MIN};
  return env_int_once("QMM_FORCE_SIMPLE", 0, cache);
}

// Which int8 dots take the kernel that splits K, for few rows or rows that TMA cannot describe.  Measured in us (it, the
// kernel that would run otherwise), operands in L2:
static bool i8_skinny_covers(int64_t M, int64_t N, int64_t K, bool tma_ok) {
  if (M > 65535 || (N + 127) / 128 * ((M + 7) / 8) > (1ll << 30)) return false;
  if (force_split_k()) return true;
  const bool large = M * N >= 128 * 128;
  if (!tma_ok) {
    // else one thread per result: its time goes with K and, once the device is full, with M * N; this kernel has a start and
    // a hand-over of 4 to 12 us.  M = 8, N = 255, K = 64: 5.8, 4.2; 128: 5.4, 5.9.  M = 64, N = 1023, K = 128: 11.5, 6.8;
    // 256: 9.6, 11.3; N = 4095, K = 128: 11.7, 15.9.  M = 512, N = 4095, K = 32 25.2, 22.6; 64 25.6, 44.1.
    const int64_t results = M * N;
    if (K >= 256) return true;
    if (K >= 128) return M <= 8 || results >= (M <= 32 ? 100000 : 200000);
    return K >= 64 && results >= (M <= 32 ? 400000 : 900000);
  }
  if (!large) return K >= 256 || (K >= 128 && M <= 16);   // else one thread per result: M = 32, N = 256, K = 128 7.1, 6.1
  if (gemm_ctas() != num_sms()) return false;             // a limit keeps the GEMM
  // Both split K.  This kernel reads b once per 64 rows and hands over 64 x 128 results at a time, the GEMM once per 128 and
  // 128 x 256.  M = 16, 4096 x 4096 8.0, 9.1; 8192 x 8192 14.3, 12.4, M = 8 13.1, 15.4.
  // M = 32, K = 128, N = 4096 7.6, 7.4 (M = 20 6.5, 7.6); 64: 8.5, 7.5; 512 x 1024 6.2, 6.5; 512 x 4096 8.0, 6.7; 2048 x 1024
  // 7.0, 7.5; 2048 x 2048 7.9, 7.7; 4096 x 1024 7.6, 8.0; 4096 x 4096 9.8, 8.9; 8192 x 1024 9.6, 9.5.
  if (M <= 32) return M <= 16 || (K >= 128 && (K < 256 ? N <= 8192 : N <= 2048 && N * K <= 4 << 20));
  // M = 64, 512 x 512 8.1, 7.9; 2048 x 2048 10.9, 8.8; 8192 x 8192 30, 14.  With more rows, only few columns suit it: M = 128,
  // 512 x 512 8.2, 9.2; 2048 x 512 9.3, 10.0; 1024 x 1024 9.7, 9.7; M = 192, 2048 x 512 9.7, 10.1; M = 256, 1024 x 256 8.6, 9.5;
  // 2048 x 512 10.4, 10.2; M = 512, 1024 x 256 9.7, 9.7.
  return M > 64 && (M + 63) / 64 * ((N + 127) / 128 * 128) <= 1536 && K >= 512;
}

}  // namespace qmm

extern "C" {

int qmm_i8i8_i32(const void* a, const void* b, int32_t* acc, const float* row_scale,
                 const float* col_scale, float* out, int64_t M, int64_t N, int64_t K,
                 int a_unsigned, int b_unsigned, void* stream) {
  using namespace qmm;
  QMM_REQUIRE(M >= 0 && N >= 0 && K >= 0 && M < (1ll << 30) && N < (1ll << 30) && K < (1ll << 30),
              QMM_ERR_INVALID_ARGUMENT, "qmm_i8i8_i32: bad shape");
  if (M == 0 || N == 0) return QMM_OK;  // empty result
  QMM_REQUIRE(a && b, QMM_ERR_INVALID_ARGUMENT, "qmm_i8i8_i32: null operand");
  QMM_REQUIRE(acc || out, QMM_ERR_INVALID_ARGUMENT, "qmm_i8i8_i32: neither acc nor out requested");
  QMM_REQUIRE(!out || (row_scale && col_scale), QMM_ERR_INVALID_ARGUMENT,
              "qmm_i8i8_i32: out needs row_scale and col_scale");
  if (int st = read_device_status())
    return set_error(QMM_ERR_TIMEOUT, "a previous kernel gave up waiting (status word 0x%x)", st);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool tma_ok = K > 0 && K % 16 == 0 && N % 16 == 0 && aligned(a, 16) && aligned(b, 16) &&
                      (!acc || aligned(acc, 16)) && (!out || (aligned(out, 16) && aligned(col_scale, 16)));
  if (K > 0 && !force_simple() && i8_skinny_covers(M, N, K, tma_ok))
    return i8_skinny(a, b, acc, row_scale, col_scale, out, M, N, K, a_unsigned, b_unsigned, tma_ok, s);
  if (tma_ok && M * N >= 128 * 128 && !force_simple())
    return i8gemm_tcgen05(a, b, acc, row_scale, col_scale, out, M, N, K, a_unsigned, b_unsigned, s);
  QMM_REQUIRE(M <= 65535, QMM_ERR_UNSUPPORTED, "qmm_i8i8_i32: unaligned shape with M > 65535");
  dim3 grid(static_cast<unsigned>((N + 127) / 128), static_cast<unsigned>(M));
  const uint8_t* ap = static_cast<const uint8_t*>(a);
  const uint8_t* bp = static_cast<const uint8_t*>(b);
  const int m = (int)M, n = (int)N, k = (int)K;
  if (a_unsigned && b_unsigned)
    simple::i8dot_kernel<true, true><<<grid, 128, 0, s>>>(ap, bp, acc, out, row_scale, col_scale, m, n, k);
  else if (a_unsigned)
    simple::i8dot_kernel<true, false><<<grid, 128, 0, s>>>(ap, bp, acc, out, row_scale, col_scale, m, n, k);
  else if (b_unsigned)
    simple::i8dot_kernel<false, true><<<grid, 128, 0, s>>>(ap, bp, acc, out, row_scale, col_scale, m, n, k);
  else
    simple::i8dot_kernel<false, false><<<grid, 128, 0, s>>>(ap, bp, acc, out, row_scale, col_scale, m, n, k);
  QMM_CHECK_LAUNCH("i8dot_kernel");
  return QMM_OK;
}

static int w8a16_entry(const char* name, const uint16_t* x, const int8_t* w, const float* scale, uint16_t* y,
                       int64_t M, int64_t N, int64_t K, int64_t ldy, const qmm_gemm_ext* ext, void* stream) {
  using namespace qmm;
  QMM_REQUIRE(M >= 0 && N >= 0 && K >= 0 && M < (1ll << 30) && N < (1ll << 30) && K < (1ll << 30) &&
                  ldy >= N,
              QMM_ERR_INVALID_ARGUMENT, "%s: bad shape (ldy must be >= N)", name);
  uint32_t flags = 0;
  uint32_t* signal = nullptr;
  uint32_t* arrive = nullptr;
  if (ext) {
    // fields are read only as far as the caller's struct reaches
    QMM_REQUIRE(ext->struct_size >= offsetof(qmm_gemm_ext, flags) + sizeof(ext->flags), QMM_ERR_INVALID_ARGUMENT,
                "%s: qmm_gemm_ext.struct_size (%zu) is too small", name, ext->struct_size);
    flags = ext->flags;
    if (ext->struct_size >= offsetof(qmm_gemm_ext, arrive_counter) + sizeof(ext->arrive_counter)) {
      signal = ext->done_signal;
      arrive = ext->arrive_counter;
    }
    QMM_REQUIRE((flags & ~(QMM_GEMM_INDEPENDENT | QMM_GEMM_STORE_MULTIMEM)) == 0, QMM_ERR_INVALID_ARGUMENT,
                "%s: unknown flag bits 0x%x", name, flags);
    QMM_REQUIRE((signal == nullptr) == (arrive == nullptr), QMM_ERR_INVALID_ARGUMENT,
                "%s: done_signal and arrive_counter go together", name);
    QMM_REQUIRE(aligned(signal, 4) && aligned(arrive, 4), QMM_ERR_INVALID_ARGUMENT, "%s: misaligned signal word", name);
  }
  if (M == 0 || N == 0) {
    QMM_REQUIRE(signal == nullptr, QMM_ERR_UNSUPPORTED, "%s: an empty result cannot signal", name);
    return QMM_OK;  // empty result
  }
  QMM_REQUIRE(x && w && scale && y, QMM_ERR_INVALID_ARGUMENT, "%s: null pointer", name);
  if (int st = read_device_status())
    return set_error(QMM_ERR_TIMEOUT, "a previous kernel gave up waiting (status word 0x%x)", st);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool tma_ok = K > 0 && K % 8 == 0 && N % 16 == 0 && ldy % 2 == 0 && aligned(x, 16) &&
                      aligned(w, 16) && aligned(y, 4);
  // Few rows, results that stay on this GPU: the HBM-bound kernel, which reads the weights once per 32 rows and splits K over
  // clusters.  So does the GEMM where its tiles are few, and it reads them once: up to 16 rows the other one is ahead by its
  // shorter start and end (M = 16, 4096 x 4096 8.8 against 12.5 us, 14336 x 4096 16.4 against 23.5, 8192 x 57344 96 against
  // 117), with more rows while a call is short: while fewer than 15 M weights are read, over all passes (M = 32: 14336 x 1024
  // 16.1 against 17.8 us, 4096 x 4096 14.1 against 12.7, 8192 x 8192 25.8 against 22.0; M = 64: 4096 x 1024 10.9 against 11.0,
  // 2048 x 4096 11.9 against 11.5, 8192 x 8192 45 against 23.5), ...
  // ... and while its columns, over all passes, are fewer than 64 for each SM, or 32 where K is short (1024 x 8192, M = 32 9.8
  // against 10.0 us, M = 64 12.2 against 11.2; 512 x 16384, M = 32 9.8 against 9.1; 256 x 4096, M = 32 6.3 against 7.1, M = 64
  // 8.1 against 7.0); K = 64: 4096 columns, M = 32 6.9 against 6.0, none.
  // Results that are too few for the GEMM (M * N < 128 * 128) are one thread each otherwise, which is quicker for a short K:
  // M = 32, N = 128, K = 64 6.8 against 3.8 us; K = 128 6.8 against 6.8.
  // (A caller that limits the GEMM's CTAs keeps the GEMM: the kernel for few rows fills the device.)
  const int64_t columns = (M + 31) / 32 * N;
  const bool gemm = M * N >= 128 * 128;
  const bool brief = columns <= num_sms() * (K < 128 ? 0 : K < 512 ? 32 : 64) && columns * K < 15000000;
  const bool pays = gemm ? M <= 16 || brief : K >= 128;
  if (tma_ok && (pays || force_split_k()) && gemm_ctas() == num_sms() && !(flags & QMM_GEMM_STORE_MULTIMEM) && signal == nullptr &&
      !force_simple())
    return w8a16_decode(x, w, scale, y, M, N, K, ldy, flags, s);
  if (tma_ok && gemm && !force_simple())
    return w8a16_tcgen05(x, w, scale, y, M, N, K, ldy, flags, signal, arrive, s);
  QMM_REQUIRE(!(flags & QMM_GEMM_STORE_MULTIMEM) && signal == nullptr, QMM_ERR_UNSUPPORTED,
              "%s: multicast stores and completion signals need the tensor-core route "
              "(K %% 8 == 0, N %% 16 == 0, even ldy, 16-byte aligned x and w, M*N >= 16384)", name);
  QMM_REQUIRE(M <= 65535, QMM_ERR_UNSUPPORTED, "%s: unaligned shape with M > 65535", name);
  dim3 grid(static_cast<unsigned>((N + 127) / 128), static_cast<unsigned>(M));
  simple::w8a16_kernel<<<grid, 128, 0, s>>>(x, w, scale, y, (int)M, (int)N, (int)K, (long long)ldy);
  QMM_CHECK_LAUNCH("w8a16_kernel(simple)");
  return QMM_OK;
}

int qmm_w8a16_perchannel(const uint16_t* x, const int8_t* w, const float* scale, uint16_t* y,
                         int64_t M, int64_t N, int64_t K, int64_t ldy, void* stream) {
  return w8a16_entry("qmm_w8a16_perchannel", x, w, scale, y, M, N, K, ldy, nullptr, stream);
}

int qmm_w8a16_perchannel_ex(const uint16_t* x, const int8_t* w, const float* scale, uint16_t* y,
                            int64_t M, int64_t N, int64_t K, int64_t ldy, const qmm_gemm_ext* ext,
                            void* stream) {
  return w8a16_entry("qmm_w8a16_perchannel_ex", x, w, scale, y, M, N, K, ldy, ext, stream);
}

int qmm_wait_signals(const uint32_t* words, int count, uint32_t expected, uint64_t timeout_ns, void* stream) {
  using namespace qmm;
  QMM_REQUIRE(words != nullptr && count >= 1 && count <= 4096 && aligned(words, 4), QMM_ERR_INVALID_ARGUMENT,
              "qmm_wait_signals: bad arguments");
  if (int st = read_device_status())
    return set_error(QMM_ERR_TIMEOUT, "a previous kernel gave up waiting (status word 0x%x)", st);
  if (timeout_ns == 0 || timeout_ns > 10000000000ull) timeout_ns = dev::kWaitLimitNs;
  simple::wait_words_kernel<<<(count + 127) / 128, 128, 0, static_cast<cudaStream_t>(stream)>>>(
      words, count, expected, timeout_ns, device_status_word());
  QMM_CHECK_LAUNCH("wait_words_kernel");
  return QMM_OK;
}

int qmm_multicast_copy(const void* src, void* dst_multicast, size_t bytes, uint32_t* done_signal, uint32_t* arrive_counter,
                       int max_ctas, void* stream) {
  using namespace qmm;
  QMM_REQUIRE(src && dst_multicast && done_signal && arrive_counter, QMM_ERR_INVALID_ARGUMENT,
              "qmm_multicast_copy: null pointer");
  QMM_REQUIRE(bytes % 16 == 0 && aligned(src, 16) && aligned(dst_multicast, 16) && aligned(done_signal, 4) &&
                  aligned(arrive_counter, 4),
              QMM_ERR_INVALID_ARGUMENT, "qmm_multicast_copy: bytes and pointers must be multiples of 16");
  QMM_REQUIRE(max_ctas >= 0 && max_ctas <= 1024, QMM_ERR_INVALID_ARGUMENT, "qmm_multicast_copy: bad max_ctas");
  if (bytes == 0) return QMM_OK;
  const size_t n16 = bytes / 16;
  int ctas = max_ctas == 0 ? 16 : max_ctas;
  const size_t need = (n16 + 511) / 512;
  if (static_cast<size_t>(ctas) > need) ctas = static_cast<int>(need);
  simple::multicast_copy_kernel<<<ctas, 512, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(src), static_cast<uint4*>(dst_multicast), n16, done_signal, arrive_counter);
  QMM_CHECK_LAUNCH("multicast_copy_kernel");
  return QMM_OK;
}

int qmm_peer_copy(const void* src, void* const* dst_peers, uint32_t* const* signal_peers, int n_peers, size_t bytes,
                  uint32_t* local_signal, uint32_t* arrive_counter, int max_ctas, void* stream) {
  using namespace qmm;
  QMM_REQUIRE(src && dst_peers && signal_peers && local_signal && arrive_counter, QMM_ERR_INVALID_ARGUMENT,
              "qmm_peer_copy: null pointer");
  QMM_REQUIRE(n_peers >= 1 && n_peers <= QMM_MAX_PEERS, QMM_ERR_INVALID_ARGUMENT, "qmm_peer_copy: 1 to %d peers",
              QMM_MAX_PEERS);
  QMM_REQUIRE(bytes % 16 == 0 && aligned(src, 16) && aligned(local_signal, 4) && aligned(arrive_counter, 4),
              QMM_ERR_INVALID_ARGUMENT, "qmm_peer_copy: bytes and pointers must be multiples of 16");
  QMM_REQUIRE(max_ctas >= 0 && max_ctas <= 1024, QMM_ERR_INVALID_ARGUMENT, "qmm_peer_copy: bad max_ctas");
  simple::PeerList peers;
  peers.n = n_peers;
  for (int p = 0; p < n_peers; ++p) {
    QMM_REQUIRE(dst_peers[p] && signal_peers[p] && aligned(dst_peers[p], 16) && aligned(signal_peers[p], 4),
                QMM_ERR_INVALID_ARGUMENT, "qmm_peer_copy: peer %d: null or misaligned pointer", p);
    peers.dst[p] = static_cast<uint4*>(dst_peers[p]);
    peers.signal[p] = signal_peers[p];
  }
  if (bytes == 0) return QMM_OK;
  const size_t n16 = bytes / 16;
  int ctas = max_ctas == 0 ? 16 : max_ctas;
  const size_t need = (n16 + 511) / 512;
  if (static_cast<size_t>(ctas) > need) ctas = static_cast<int>(need);
  simple::peer_copy_kernel<<<ctas, 512, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const uint4*>(src), peers, n16,
                                                                              local_signal, arrive_counter);
  QMM_CHECK_LAUNCH("peer_copy_kernel");
  return QMM_OK;
}

}  // extern "C"
