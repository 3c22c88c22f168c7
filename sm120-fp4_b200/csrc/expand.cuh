// W4A16 on an FP4 x FP4 tensor-core instruction: a 16-bit activation block is written as a short sum of NVFP4 blocks,
//     x = q1*s1/g1 + q2*s2/g2 + q3*s3/g3 + q4*s4/g4 + r,   g_t = g1 * 6^(t-1),   |r| <= blockmax(x) * 6^-4,
// each term the NVFP4 quantisation (E2M1 codes, E4M3 scale per 16 values) of the residual left by the terms before it.
// Shared by the decode kernel, its activation-expansion kernel and the W4A16 grouped GEMM of mid-sized batches.
#pragma once
#include "ptx.cuh"

namespace b200 {

constexpr int kTerms = 4;

__device__ __forceinline__ uint8_t tc_e4m3(float v) {   // RNE, saturating at 448, subnormals kept
  uint16_t r;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(0.0f), "f"(v));
  return (uint8_t)(r & 0xff);
}
__device__ __forceinline__ float rcp_approx(float v) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
// two lanes of one instruction: (oa, ob) = (a, b) * s; (ra, rb) += (a, b) * s
__device__ __forceinline__ void mul_f32x2(float a, float b, float s, float& oa, float& ob) {
  asm("{\n .reg .b64 x, y;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %4};\n mul.rn.f32x2 x, x, y;\n mov.b64 {%0, %1}, x;\n}\n" : "=f"(oa), "=f"(ob) : "f"(a), "f"(b), "f"(s));
}
__device__ __forceinline__ void fma_f32x2(float a, float b, float s, float& ra, float& rb) {
  asm("{\n .reg .b64 x, y, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %4};\n mov.b64 z, {%0, %1};\n fma.rn.f32x2 z, x, y, z;\n mov.b64 {%0, %1}, z;\n}\n"
      : "+f"(ra), "+f"(rb) : "f"(a), "f"(b), "f"(s));
}

// 8 floats -> 8 E2M1 codes in one word (element 2j in the low nibble of byte j), hardware round-to-nearest-even,
// saturating. cvt.rn.satfinite.e2m1x2.f32 d, a, b puts a into the high and b into the low nibble of d. (The bytes are put together
// with shifts: where the word is taken apart again into .b8 registers right after, as here, the assembler of CUDA 12.9 drops the
// upper two bytes of a word built by mov.b32 from four .b8 registers.)
__device__ __forceinline__ uint32_t cvt_f32x8_e2m1(const float* v) {
  uint32_t b[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    asm("{\n .reg .b8 t;\n cvt.rn.satfinite.e2m1x2.f32 t, %1, %2;\n cvt.u32.u8 %0, t;\n}\n" : "=r"(b[i]) : "f"(v[2 * i + 1]), "f"(v[2 * i]));
  return (b[0] | (b[1] << 8)) | ((b[2] << 16) | (b[3] << 24));
}

// One 16-value block -> kTerms NVFP4 terms (residual expansion). g1: global scale of the first term; term t uses g1*6^t.
// codes[t] = 8 packed bytes (element 2j in the low nibble), sf[t] = E4M3 scale byte. The residual is taken against the
// codes and the scale actually emitted, so any rounding on the way (approximate reciprocal included) is absorbed by the
// next term.
// Returns true when the block's maximum lies beyond what the first term can hold (its scale clamps at 448, i.e. values
// above 2688 / g1): the later terms, with their larger global scales, cannot absorb the clipped part.
// Each term is handed to `put(t, codes, scale byte)` as it is formed. kLoop: the terms as a loop of about a hundred instructions
// rather than four copies of it, for kernels that run through their code only a few times per launch - an instruction line
// that is not yet in the SM's cache costs more than the loop does.
// K blocks at a time share the latency of the chain (900 cycles for one block, 1,300 for two; put also gets the block's index).
template <bool kLoop, int K, class F>
__device__ __forceinline__ bool expand_blocks16(float (&r)[K][16], const float (&g1)[K], F&& put) {
  float g[K], ginv[K];
#pragma unroll
  for (int k = 0; k < K; ++k) g[k] = g1[k], ginv[k] = __frcp_rn(g1[k]);
  bool clipped = false;
#pragma unroll(kLoop ? 1 : kTerms)
  for (int t = 0; t < kTerms; ++t) {
    uint8_t sb[K];
    uint2 codes[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      float m[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) m[i] = fmaxf(fabsf(r[k][i]), fabsf(r[k][i + 8]));
#pragma unroll
      for (int i = 0; i < 4; ++i) m[i] = fmaxf(m[i], m[i + 4]);
      const float amax = fmaxf(fmaxf(m[0], m[2]), fmaxf(m[1], m[3]));
      const float want = amax * (1.0f / 6.0f) * g[k];
      if (t == 0) clipped |= want > 464.0f;   // 464 is the first value that no longer rounds down to 448
      sb[k] = tc_e4m3(fminf(want, 448.0f));
      const uint32_t svh = cvt_e4m3x2_f16x2(sb[k]);
      const float sv = __low2float(*reinterpret_cast<const __half2*>(&svh));
      const float scale = sv > 0.f ? g[k] * rcp_approx(sv) : 0.f, back = -sv * ginv[k];
      float sc[16];
#pragma unroll
      for (int i = 0; i < 16; i += 2) mul_f32x2(r[k][i], r[k][i + 1], scale, sc[i], sc[i + 1]);
      const uint32_t lo = cvt_f32x8_e2m1(sc), hi = cvt_f32x8_e2m1(sc + 8);
      uint32_t dl[4], dh[4];
      cvt_e2m1x8_f16x2(lo, dl);
      cvt_e2m1x8_f16x2(hi, dh);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&dl[i]));
        const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&dh[i]));
        fma_f32x2(a.x, a.y, back, r[k][2 * i], r[k][2 * i + 1]);
        fma_f32x2(b.x, b.y, back, r[k][8 + 2 * i], r[k][8 + 2 * i + 1]);
      }
      codes[k] = make_uint2(lo, hi);
      g[k] *= 6.0f;
      ginv[k] *= (1.0f / 6.0f);
    }
#pragma unroll
    for (int k = 0; k < K; ++k) put(k, t, codes[k], sb[k]);
  }
  return clipped;
}
template <bool kLoop, class F>
__device__ __forceinline__ bool expand_block16(float (&r)[16], float g1, F&& put) {
  const float g[1] = {g1};
  return expand_blocks16<kLoop, 1>(reinterpret_cast<float(&)[1][16]>(r), g, [&](int, int t, uint2 codes, uint8_t sf) { put(t, codes, sf); });
}

// One block spread over the four lanes 4i..4i+3 of a warp, four values each (all lanes of the warp call it): half the latency of the
// whole block in one lane. put(t, two bytes of codes, scale byte).
template <class F>
__device__ __forceinline__ bool expand_quad(float (&r)[4], float g1, F&& put) {
  float g = g1, ginv = __frcp_rn(g1);
  bool clipped = false;
#pragma unroll 1
  for (int t = 0; t < kTerms; ++t) {
    float amax = fmaxf(fmaxf(fabsf(r[0]), fabsf(r[1])), fmaxf(fabsf(r[2]), fabsf(r[3])));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    const float want = amax * (1.0f / 6.0f) * g;
    if (t == 0) clipped = want > 464.0f;   // 464 is the first value that no longer rounds down to 448
    const uint8_t sb = tc_e4m3(fminf(want, 448.0f));
    const uint32_t svh = cvt_e4m3x2_f16x2(sb);
    const float sv = __low2float(*reinterpret_cast<const __half2*>(&svh));
    const float scale = sv > 0.f ? g * rcp_approx(sv) : 0.f, back = -sv * ginv;
    float sc[4];
    mul_f32x2(r[0], r[1], scale, sc[0], sc[1]);
    mul_f32x2(r[2], r[3], scale, sc[2], sc[3]);
    uint32_t c0, c1, d0, d1;
    asm("{\n .reg .b8 t;\n cvt.rn.satfinite.e2m1x2.f32 t, %1, %2;\n cvt.u32.u8 %0, t;\n}\n" : "=r"(c0) : "f"(sc[1]), "f"(sc[0]));
    asm("{\n .reg .b8 t;\n cvt.rn.satfinite.e2m1x2.f32 t, %1, %2;\n cvt.u32.u8 %0, t;\n}\n" : "=r"(c1) : "f"(sc[3]), "f"(sc[2]));
    asm("{\n .reg .b8 t;\n cvt.u8.u32 t, %1;\n cvt.rn.f16x2.e2m1x2 %0, t;\n}\n" : "=r"(d0) : "r"(c0));
    asm("{\n .reg .b8 t;\n cvt.u8.u32 t, %1;\n cvt.rn.f16x2.e2m1x2 %0, t;\n}\n" : "=r"(d1) : "r"(c1));
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&d0)), b = __half22float2(*reinterpret_cast<const __half2*>(&d1));
    fma_f32x2(a.x, a.y, back, r[0], r[1]);
    fma_f32x2(b.x, b.y, back, r[2], r[3]);
    put(t, (uint16_t)(c0 | (c1 << 8)), sb);
    g *= 6.0f;
    ginv *= (1.0f / 6.0f);
  }
  return clipped;
}

}  // namespace b200
