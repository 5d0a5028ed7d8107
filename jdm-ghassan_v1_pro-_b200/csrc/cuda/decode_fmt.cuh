// Stored weight rows of the decode kernels: how eight consecutive values of a row are expanded into floats, per
// storage format (formats and block layouts in gb_decode.h), and the router's choice by one warp.  Shared by the per-kernel token step
// (decode.cu) and the single-kernel token step (decode_mega.cu).
#pragma once
#include "sm100_common.cuh"
#include "gb_decode.h"

namespace gb {

__device__ __forceinline__ float h2f(uint16_t h) { return __half2float(__ushort_as_half(h)); }
__device__ __forceinline__ uint16_t ld_u16(const uint8_t* p) { return *reinterpret_cast<const uint16_t*>(p); }

// Expand unit u (values 8u .. 8u+7) of one stored row into floats.
template <int FMT>
__device__ __forceinline__ void load8(const uint8_t* __restrict__ row, int u, float (&w)[8]) {
  if constexpr (FMT == GB_W_F16) {
    const uint4 q = *reinterpret_cast<const uint4*>(row + 16 * (size_t)u);
    const __half2* h = reinterpret_cast<const __half2*>(&q);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 f = __half22float2(h[i]); w[2 * i] = f.x; w[2 * i + 1] = f.y; }
  } else if constexpr (FMT == GB_W_BF16) {
    const uint4 q = *reinterpret_cast<const uint4*>(row + 16 * (size_t)u);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(h[i]); w[2 * i] = f.x; w[2 * i + 1] = f.y; }
  } else if constexpr (FMT == GB_W_GGML_Q8_0) {
    const uint8_t* p = row + (size_t)(u >> 2) * 34;
    const float d = h2f(ld_u16(p));
    const uint8_t* q = p + 2 + (u & 3) * 8;           // 2-byte aligned: blocks are 34 bytes
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint16_t v = ld_u16(q + 2 * i);
      w[2 * i] = d * (float)(int8_t)(v & 0xFF);
      w[2 * i + 1] = d * (float)(int8_t)(v >> 8);
    }
  } else if constexpr (FMT == GB_W_Q4_0) {
    const uint8_t* p = row + (size_t)(u >> 2) * 18;
    const float d = h2f(ld_u16(p));
    const uint8_t* q = p + 2 + (u & 3) * 4;
    const uint32_t v = (uint32_t)ld_u16(q) | ((uint32_t)ld_u16(q + 2) << 16);
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = d * (float)((int)((v >> (4 * i)) & 0xF) - 8);   // byte i: low nibble = value 2i
  } else if constexpr (FMT == GB_W_Q8_64) {
    const uint8_t* p = row + (size_t)(u >> 3) * 68;
    const float d = *reinterpret_cast<const float*>(p);
    // blocks are 68 bytes: the quants are 4-byte aligned but not 8-byte aligned, so two 32-bit loads
    const uint32_t* qp = reinterpret_cast<const uint32_t*>(p + 4 + (u & 7) * 8);
    const uint32_t vx = qp[0], vy = qp[1];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      w[i] = d * (float)(int8_t)((vx >> (8 * i)) & 0xFF);
      w[4 + i] = d * (float)(int8_t)((vy >> (8 * i)) & 0xFF);
    }
  } else {   // GB_W_Q4_1
    const uint8_t* p = row + (size_t)(u >> 2) * 20;
    const float d = h2f(ld_u16(p)), m = h2f(ld_u16(p + 2));
    const uint32_t v = *reinterpret_cast<const uint32_t*>(p + 4 + (u & 3) * 4);
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = d * (float)((v >> (4 * i)) & 0xF) + m;
  }
}

// Soft-max over ne <= 64 logits, lane e holding experts e (l0) and e + 32 (l1; -inf where there is none), and the top_k picks by
// probability + bias (ties: the lower index), their probabilities renormalised.  Lane k < top_k gets pick k: expert my_e, weight my_w.
__device__ __forceinline__ void warp_route(float l0, float l1, const float* __restrict__ bias, int ne, int top_k, int& my_e, float& my_w) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  if (ne <= 8) {                        // eight lanes do: three steps instead of five, nothing in a second register
    float mx = lane < ne ? l0 : -INFINITY;
#pragma unroll
    for (int o = 4; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(full, mx, o));
    const float p0 = lane < ne ? __expf(l0 - mx) : 0.f;
    float sum = p0;
#pragma unroll
    for (int o = 4; o; o >>= 1) sum += __shfl_xor_sync(full, sum, o);
    const float p = p0 * (1.f / sum), score = lane < ne ? p + (bias ? bias[lane] : 0.f) : -INFINITY;
    int place = 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float v = __shfl_sync(full, score, e);
      place += e < ne && (v > score || (v == score && e < lane)) ? 1 : 0;
    }
    float psum = 0.f;
    my_w = 0.f;
    my_e = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const unsigned who = __ballot_sync(full, lane < ne && place == k);
      const int e = who ? __ffs(who) - 1 : 0;
      const float w = __shfl_sync(full, p, e);
      if (k < top_k) {
        if (lane == k) { my_e = e; my_w = w; }
        psum += w;
      }
    }
    my_w *= psum > 1e-8f ? 1.f / psum : 0.f;
    return;
  }
  const bool h0 = lane < ne, h1 = lane + 32 < ne;
  const float mx = warp_max(fmaxf(l0, l1));
  float p0 = h0 ? __expf(l0 - mx) : 0.f, p1 = h1 ? __expf(l1 - mx) : 0.f;
  const float inv = 1.f / warp_sum(p0 + p1);
  p0 *= inv;
  p1 *= inv;
  float s0 = h0 ? p0 + (bias ? bias[lane] : 0.f) : -INFINITY;
  float s1 = h1 ? p1 + (bias ? bias[lane + 32] : 0.f) : -INFINITY;
  // An expert's place is the number of experts ahead of it: independent shuffles, where picking the best top_k times was a chain of ten
  // shuffles a pick.
  int r0 = 0, r1 = 0;
#pragma unroll 8
  for (int e = 0; e < ne; ++e) {
    const float v = __shfl_sync(full, e < 32 ? s0 : s1, e & 31);
    r0 += v > s0 || (v == s0 && e < lane) ? 1 : 0;
    r1 += v > s1 || (v == s1 && e < lane + 32) ? 1 : 0;
  }
  float psum = 0.f;
  my_w = 0.f;
  my_e = 0;
#pragma unroll 4
  for (int k = 0; k < top_k; ++k) {
    const unsigned b0 = __ballot_sync(full, h0 && r0 == k), b1 = __ballot_sync(full, h1 && r1 == k);
    const int e = b0 ? __ffs(b0) - 1 : b1 ? __ffs(b1) + 31 : 0;
    const float w = __shfl_sync(full, b0 ? p0 : p1, e & 31);
    if (lane == k) { my_e = e; my_w = w; }
    psum += w;
  }
  my_w *= psum > 1e-8f ? 1.f / psum : 0.f;
}

}  // namespace gb
