// Per-head RMS norm with weight + partial rotary embedding of one row, 8 channels per thread,
// D/8 consecutive lanes per row (shared by the stand-alone producer kernel and the exchange's
// stores).  Formula and canonical arithmetic: see producer.cu.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

namespace nr {

template <typename T>
__device__ __forceinline__ float to_float(T v);
template <>
__device__ __forceinline__ float to_float<__half>(__half v) {
  return __half2float(v);
}
template <>
__device__ __forceinline__ float to_float<__nv_bfloat16>(__nv_bfloat16 v) {
  return __bfloat162float(v);
}
// Two results rounded to T, in one register.
template <typename T>
__device__ __forceinline__ uint32_t pack2(float a, float b);
template <>
__device__ __forceinline__ uint32_t pack2<__half>(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
template <>
__device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// The steps of one row.  Every lane of the warp must call them (they shuffle inside groups of D/8
// lanes); `raw` holds the thread's 8 channels (lane * 8 ...) of the row, zeros for a row that is not live.

// Sum of the row's squares, in every lane of its group.
template <typename T, int D>
__device__ __forceinline__ float square_sum(uint4 raw) {
  const T* e = reinterpret_cast<const T*>(&raw);
  float sum = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float v = to_float<T>(e[i]);
    sum = __fmaf_rn(v, v, sum);
  }
#pragma unroll
  for (int off = D / 16; off > 0; off >>= 1) sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, off));
  return sum;
}

// (D is a power of two: the product with 1/D is the quotient)
template <int D>
__device__ __forceinline__ float inverse_rms(float sum, float eps) {
  return __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fmul_rn(sum, 1.0f / D), eps)));
}

// Where a lane's channels stand in the rotary span; partner channels live half/8 lanes away
// (rotary_dim is a multiple of 16).
struct Rotary {
  bool in, first;
  int partner;
  __device__ __forceinline__ Rotary(int lane, int rotary_dim) {
    const int half = rotary_dim / 2, c0 = lane * 8;
    in = c0 < rotary_dim;
    first = c0 < half;
    partner = in ? (first ? lane + half / 8 : lane - half / 8) : lane;
  }
};

// 8 consecutive table entries of a token's row: two 16-byte loads each.  The first half's sines change
// sign here: -pn * sn and pn * -sn are the same number.
__device__ __forceinline__ void load_tables(const float* cos_row, const float* sin_row, int lane, bool first,
                                            float (&cs)[8], float (&sn)[8]) {
  const float4* ct = reinterpret_cast<const float4*>(cos_row + lane * 8);
  const float4* st = reinterpret_cast<const float4*>(sin_row + lane * 8);
  *reinterpret_cast<float4*>(cs) = __ldg(ct);
  *reinterpret_cast<float4*>(cs + 4) = __ldg(ct + 1);
  *reinterpret_cast<float4*>(sn) = __ldg(st);
  *reinterpret_cast<float4*>(sn + 4) = __ldg(st + 1);
  if (first)
#pragma unroll
    for (int i = 0; i < 8; ++i) sn[i] = -sn[i];
}

// Norm, weight and rotation; cs / sn: the table entries of the thread's channels, only read inside
// the span.  Returns the 8 results rounded to T.
template <typename T, int D>
__device__ __forceinline__ uint4 norm_rope_row(uint4 raw, uint4 wraw, float r, const Rotary& rot,
                                               const float (&cs)[8], const float (&sn)[8]) {
  const T* e = reinterpret_cast<const T*>(&raw);
  const T* w = reinterpret_cast<const T*>(&wraw);
  float o[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float n = __fmul_rn(__fmul_rn(to_float<T>(e[i]), r), to_float<T>(w[i]));
    // every lane takes part in the shuffle; lanes outside the span read themselves
    const float pn = __shfl_sync(0xffffffffu, n, rot.partner, D / 8);
    o[i] = rot.in ? __fmaf_rn(pn, sn[i], __fmul_rn(n, cs[i])) : n;
  }
  return make_uint4(pack2<T>(o[0], o[1]), pack2<T>(o[2], o[3]), pack2<T>(o[4], o[5]), pack2<T>(o[6], o[7]));
}

// One row at once.  `cos_row` / `sin_row` point at the row's token in the fp32 tables ([rotary_dim]
// entries); they are only read by live lanes inside the rotary span.
template <typename T, int D>
__device__ __forceinline__ uint4 norm_rope8(uint4 raw, const T* weight, const float* cos_row,
                                            const float* sin_row, int rotary_dim, float eps, int lane,
                                            bool live) {
  const Rotary rot(lane, rotary_dim);
  float cs[8] = {}, sn[8] = {};
  if (rot.in && live) load_tables(cos_row, sin_row, lane, rot.first, cs, sn);
  const float r = inverse_rms<D>(square_sum<T, D>(raw), eps);
  return norm_rope_row<T, D>(raw, *reinterpret_cast<const uint4*>(weight + lane * 8), r, rot, cs, sn);
}

}  // namespace nr
