// Dequantisation of the operator-API weight formats, one rule per format as the reference kernels state it
// (f32 throughout): shared by the CUDA-core kernels and by the exact path of the tensor-core GEMM.
#pragma once

#include "common.cuh"

namespace qmm {
namespace opapi {

static __device__ __constant__ float kE2M1[16] = {0.0f,  0.5f,  1.0f,  1.5f,  2.0f,  3.0f,  4.0f,  6.0f,
                                           -0.0f, -0.5f, -1.0f, -1.5f, -2.0f, -3.0f, -4.0f, -6.0f};

__device__ __forceinline__ float decode_e4m3(uint32_t b) {
  if ((b & 127u) == 127u) return __uint_as_float(0x7FC00000u);
  const __half h = __ushort_as_half(static_cast<unsigned short>((b & 127u) << 7));
  const float v = __half2float(h) * 256.0f;
  return (b & 128u) ? -v : v;
}
__device__ __forceinline__ float decode_e8m0(uint32_t b) {
  if (b == 0xFFu) return __uint_as_float(0x7FC00000u);
  return __uint_as_float(b == 0 ? 0x00400000u : (b << 23));
}

// Decoders: eight dequantised weights for column n, k = k8 .. k8+7.
struct Affine4 {
  const uint32_t* w; const float* s; const float* b; int K; int gs;
  __device__ __forceinline__ void operator()(int n, int k8, float (&o)[8]) const {
    const uint32_t word = __ldg(w + static_cast<size_t>(n) * (K / 8) + k8 / 8);
    const int g = k8 / gs;
    const float sc = __ldg(s + static_cast<size_t>(n) * (K / gs) + g);
    const float bi = __ldg(b + static_cast<size_t>(n) * (K / gs) + g);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = fmaf(sc, static_cast<float>((word >> (4 * j)) & 0xFu), bi);
  }
};
struct Affine8 {
  const uint8_t* w; const float* s; const float* b; int K; int gs;
  __device__ __forceinline__ void operator()(int n, int k8, float (&o)[8]) const {
    const uint2 words = __ldg(reinterpret_cast<const uint2*>(w + static_cast<size_t>(n) * K + k8));
    const int g = k8 / gs;
    const float sc = __ldg(s + static_cast<size_t>(n) * (K / gs) + g);
    const float bi = __ldg(b + static_cast<size_t>(n) * (K / gs) + g);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      o[j] = fmaf(sc, static_cast<float>((words.x >> (8 * j)) & 0xFFu), bi);
      o[4 + j] = fmaf(sc, static_cast<float>((words.y >> (8 * j)) & 0xFFu), bi);
    }
  }
};
template <int MODE>  // 0 mxfp4 (group 32, e8m0), 1 mxfp8 (group 32, e8m0), 2 nvfp4 (group 16, e4m3)
struct Mx {
  const uint8_t* w; const uint8_t* s; int K;
  __device__ __forceinline__ void operator()(int n, int k8, float (&o)[8]) const {
    constexpr int gs = (MODE == 2) ? 16 : 32;
    const uint32_t sb = __ldg(s + static_cast<size_t>(n) * (K / gs) + k8 / gs);
    const float sc = (MODE == 2) ? decode_e4m3(sb) : decode_e8m0(sb);
    if (MODE == 1) {
      const uint2 words = __ldg(reinterpret_cast<const uint2*>(w + static_cast<size_t>(n) * K + k8));
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        o[j] = sc * decode_e4m3((words.x >> (8 * j)) & 0xFFu);
        o[4 + j] = sc * decode_e4m3((words.y >> (8 * j)) & 0xFFu);
      }
    } else {
      const uint32_t word =
          __ldg(reinterpret_cast<const uint32_t*>(w + static_cast<size_t>(n) * (K / 2) + k8 / 2));
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = sc * kE2M1[(word >> (4 * j)) & 0xFu];
    }
  }
};

}  // namespace opapi
}  // namespace qmm
