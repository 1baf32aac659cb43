// What the tensor-core GEMMs of the operator API share: conversion of packed codes into 16-bit operands, packed f32
// arithmetic, and the dot product that takes over where an operand cannot hold the values.
#pragma once

#include "opapi_decode.cuh"

namespace qmm {
namespace opg {

enum { kAffine4 = 0, kAffine8 = 1, kMxfp4 = 2, kMxfp8 = 3, kNvfp4 = 4 };

__device__ __forceinline__ uint32_t lop_and_or(uint32_t a, uint32_t m, uint32_t o) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(m), "r"(o));
  return r;
}
template <bool BF16>
__device__ __forceinline__ uint32_t mul2(uint32_t a, uint32_t b) {
  uint32_t r;
  if (BF16) asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  else asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
template <bool BF16>
__device__ __forceinline__ uint32_t sub2(uint32_t a, uint32_t b) {
  uint32_t r;
  if (BF16) asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  else asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ void e2m1_to_f16(uint32_t w, uint32_t (&r)[4]) {
  asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\tmov.b32 {b0, b1, b2, b3}, %4;\n\t"
      "cvt.rn.f16x2.e2m1x2 %0, b0;\n\tcvt.rn.f16x2.e2m1x2 %1, b1;\n\t"
      "cvt.rn.f16x2.e2m1x2 %2, b2;\n\tcvt.rn.f16x2.e2m1x2 %3, b3;\n\t}"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
      : "r"(w));
}
__device__ __forceinline__ void e4m3_to_f16(uint32_t w, uint32_t& p01, uint32_t& p23) {
  asm("{\n\t.reg .b16 h0, h1;\n\tmov.b32 {h0, h1}, %2;\n\t"
      "cvt.rn.f16x2.e4m3x2 %0, h0;\n\tcvt.rn.f16x2.e4m3x2 %1, h1;\n\t}"
      : "=r"(p01), "=r"(p23)
      : "r"(w));
}
__device__ __forceinline__ uint32_t f16x2_to_bf16x2(uint32_t h) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
  return dev::pack_bf16x2(f.x, f.y);
}

// Eight codes of k .. k+7 -> eight 16-bit operand values in k order.  For 4-bit formats `lo` holds all eight.
//   integers:  128 + q or 1024 + q by OR-ing the code into a constant's mantissa, minus that constant.  An 8-bit code
//              in bf16 reads as q * 2^-133 where it stands (a subnormal up to 127, the first binade above) and is
//              multiplied by 2^127: q / 64, the group's scale makes up for it.  Against f32 results a code may go in
//              centred (centred(): q - 8 or q - 128).
//   e2m1:      cvt to f16; for bf16 the code's exponent and mantissa are moved into place (worth 2^-126 of the
//              element) and multiplied by 2^126
//   e4m3:      cvt to f16, then to bf16 (4 significant bits: exact)
template <int FMT, bool BF16>
__device__ __forceinline__ uint4 convert8(uint32_t lo, uint32_t hi, uint32_t scale2, bool centre) {
  uint32_t r[4];
  if (FMT == kAffine8) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t sel = (i & 1) ? 0x4342 : 0x4140;
      if (BF16) {   // q * 2^-133 * 2^127, minus 2 for a centred code
        const uint32_t c = centre ? 0xC000C000u : 0u;
        asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r[i]) : "r"(__byte_perm(i < 2 ? lo : hi, 0u, sel)), "r"(0x7F007F00u), "r"(c));
      } else r[i] = sub2<false>(__byte_perm(i < 2 ? lo : hi, 0x64646464u, sel), 0x64006400u);
    }
  } else if (FMT == kMxfp8) {
    e4m3_to_f16(lo, r[0], r[1]);
    e4m3_to_f16(hi, r[2], r[3]);
    if (BF16) {
#pragma unroll
      for (int i = 0; i < 4; ++i) r[i] = f16x2_to_bf16x2(r[i]);
    }
  } else if (!BF16 && (FMT == kMxfp4 || FMT == kNvfp4)) {
    e2m1_to_f16(lo, r);
  } else {
    const uint32_t e = lo & 0x0F0F0F0Fu, o = (lo >> 4) & 0x0F0F0F0Fu;  // even and odd k
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      // byte 0 = e[i], byte 2 = o[i]; bytes 1 and 3 are e[0] and are masked off
      const uint32_t p = __byte_perm(e, o, static_cast<uint32_t>(i) | (4u + i) << 8);
      if (FMT == kAffine4) {
        const uint32_t t = lop_and_or(p, 0x000F000Fu, BF16 ? 0x43004300u : 0x64006400u);
        r[i] = sub2<BF16>(t, BF16 ? (centre ? 0x43084308u : 0x43004300u) : 0x64006400u);
      } else {
        const uint32_t mag = (p & 0x00070007u) << 6, sgn = (p & 0x00080008u) << 12;
        r[i] = mul2<true>(mag | sgn, 0x7E807E80u);                       // times 2^126
      }
    }
  }
  if (FMT == kNvfp4) {
#pragma unroll
    for (int i = 0; i < 4; ++i) r[i] = mul2<BF16>(r[i], scale2);
  }
  return make_uint4(r[0], r[1], r[2], r[3]);
}

// Whether a group's integer codes go in centred (f32 results).  scale * q + bias = scale * (q - c) + (bias + c * scale):
// the usual group spans zero, its bias is about -c * scale, and the two parts of its sum would cancel to half their
// size.  A flat group has scale 1, code 0 and its value as bias: centring it would make the parts large instead.
template <int FMT>
__device__ __forceinline__ bool centred(float s, float b, float& shifted) {
  shifted = fmaf(FMT == kAffine4 ? 8.f : 128.f, s, b);
  return fabsf(shifted) < fabsf(b);
}

// e4m3 scale byte -> (s, s) in f16 or bf16
template <bool BF16>
__device__ __forceinline__ uint32_t e4m3_pair(uint32_t b) {
  uint32_t p, unused;
  e4m3_to_f16(b | (b << 8), p, unused);
  return BF16 ? f16x2_to_bf16x2(p) : p;
}

__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

__device__ __forceinline__ uint64_t fmul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ void add2(uint64_t& acc, uint64_t a) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(acc) : "l"(a)); }

// sum_{k in [k0, k1)} x[m,k] * weight[n,k], as the CUDA-core kernels compute it
template <int FMT, bool XF32>
__device__ __forceinline__ float exact_dot_here(const void* x, const uint8_t* w, const void* scales, const float* biases, int K, int gs,
                                        int m, int n, int k0, int k1) {
  float acc = 0.f;
  for (int k = k0; k < k1; k += 8) {
    float wv[8];
    if constexpr (FMT == kAffine4) {
      opapi::Affine4 d{reinterpret_cast<const uint32_t*>(w), static_cast<const float*>(scales), biases, K, gs};
      d(n, k, wv);
    } else if constexpr (FMT == kAffine8) {
      opapi::Affine8 d{w, static_cast<const float*>(scales), biases, K, gs};
      d(n, k, wv);
    } else {
      opapi::Mx<FMT - kMxfp4> d{w, static_cast<const uint8_t*>(scales), K};
      d(n, k, wv);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const size_t i = static_cast<size_t>(m) * K + k + j;
      const float xv = XF32 ? __ldg(static_cast<const float*>(x) + i) : __half2float(static_cast<const __half*>(x)[i]);
      acc = fmaf(xv, wv[j], acc);
    }
  }
  return acc;
}
// The same as a call: it is rare, and its registers are not to weigh on the code around it.
template <int FMT, bool XF32>
__device__ __noinline__ float exact_dot(const void* x, const uint8_t* w, const void* scales, const float* biases, int K, int gs,
                                        int m, int n, int k0, int k1) {
  return exact_dot_here<FMT, XF32>(x, w, scales, biases, K, gs, m, n, k0, k1);
}

}  // namespace opg
}  // namespace qmm
