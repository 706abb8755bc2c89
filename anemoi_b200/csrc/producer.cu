// Producer-side fusion in front of the attention path: per-head RMS norm with weight, then
// partial rotary embedding, in place on Q or K ([tokens][heads][D], 16-bit).  One pass over HBM
// (read + write) instead of the six of an eager implementation.
//
// Follows the reference's fused kernel
// (anemoi/models/minimax_h3/solengine/models/minimax_h3/optimized/fusions.py:208-274):
//   variance = sum_j x_j^2 / D;  r = 1/sqrt(variance + eps);  n_j = (x_j * r) * w_j
//   inside the rotary span [0, rotary_dim), half = rotary_dim/2, channel j pairs with j +- half:
//     out_j = n_j * cos_j + rot_j * sin_j,  rot_j = -n_{j+half} (j < half), +n_{j-half} (j >= half)
//   outside it out_j = n_j; cos/sin are fp32 tables [tokens][rotary_dim] shared by the heads.
// The reference leaves the summation order and the contraction of the last line to its
// compiler; here they are fixed so that a CPU restatement reproduces every bit: each thread
// sums its 8 channels with a sequential FMA chain, the D/8 threads of a row combine with an
// xor butterfly (largest offset first), r is an IEEE division by an IEEE square root, and
// out_j = fma(rot_j, sin_j, round(n_j * cos_j)).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include "../../include/anemoi_sm100.h"
#include "norm_rope.cuh"

namespace {

// A group of D/8 consecutive lanes takes kRows heads of one token, 8 channels per thread.  HBM bound
// (read + write of x), which takes loads in flight: with one row per group (a 16-byte load per
// thread, then the whole arithmetic) 33,272 tokens x 56 heads x 128 take 289 us = 3.3 TB/s.  Four rows
// give four loads in flight, one read of the token's cos / sin entries and of the weights for all four,
// and the square root and division of a row, which every lane of the group would repeat, are
// done once, by lane i for row i: 180 us (two rows: 206; eight: 321).  With two results per conversion and
// the sines' sign turned once, and 80 registers, so that nothing spills, in CTAs of two warps: 166-170 us = 5.7 TB/s
// over one tensor again and again (of 128 threads 169, of 256 175; at 64 registers 205; with packed multiplications
// 188); Q and K of a model in turn, 333-360 us, 82-88 % of a plain copy's rate.  One row per group where a token
// has no more than two heads.
constexpr int kThreads = 64;
template <typename T, int D, int kRows>
__global__ void __launch_bounds__(kThreads, 12) qknorm_rope_kernel(T* x, const T* weight, const float* cos_table,
                                                             const float* sin_table, uint32_t units, int quads,
                                                             int heads, int rotary_dim, float eps,
                                                             int64_t token_stride, int64_t head_stride) {
  constexpr int kLanes = D / 8;
  // (in units, not threads: 32 bits hold every unit that the launcher admits, threads are 8 or 16 times as many)
  const uint32_t unit = blockIdx.x * (uint32_t)(kThreads / kLanes) + threadIdx.x / kLanes;
  const int lane = threadIdx.x % kLanes;
  const bool in = unit < units;
  const uint32_t token = in ? unit / (uint32_t)quads : 0u;
  const int head0 = in ? (int)(unit - token * (uint32_t)quads) * kRows : 0;
  T* p = x + (int64_t)token * token_stride + (int64_t)head0 * head_stride + lane * 8;
  uint4 raw[kRows];
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    raw[i] = make_uint4(0, 0, 0, 0);
    if (in && head0 + i < heads) raw[i] = *reinterpret_cast<const uint4*>(p + i * head_stride);
  }
  const nr::Rotary rot(lane, rotary_dim);
  float cs[8], sn[8];
  if (rot.in && in)
    nr::load_tables(cos_table + (int64_t)token * rotary_dim, sin_table + (int64_t)token * rotary_dim, lane, rot.first,
                    cs, sn);
  const uint4 wraw = __ldg(reinterpret_cast<const uint4*>(weight + lane * 8));
  float mine = 0.0f;
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    const float sum = nr::square_sum<T, D>(raw[i]);
    if ((lane & (kRows - 1)) == i) mine = sum;
  }
  const float r_mine = nr::inverse_rms<D>(mine, eps);
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    const float r = __shfl_sync(0xffffffffu, r_mine, i, kLanes);
    const uint4 out = nr::norm_rope_row<T, D>(raw[i], wraw, r, rot, cs, sn);
    if (in && head0 + i < heads) *reinterpret_cast<uint4*>(p + i * head_stride) = out;
  }
}

template <typename T, int D, int kRows>
int launch_rows(void* x, const void* weight, const float* c, const float* s, int64_t tokens, int heads, int rotary,
                float eps, const int64_t* strides, cudaStream_t st) {
  const int64_t quads = (heads + kRows - 1) / kRows, units = tokens * quads;
  constexpr int64_t kUnits = kThreads / (D / 8);
  if (tokens * heads > 0x7fffffffLL) return ANEMOI_SM100_ELIMIT;
  qknorm_rope_kernel<T, D, kRows><<<(unsigned)((units + kUnits - 1) / kUnits), kThreads, 0, st>>>(
      static_cast<T*>(x), static_cast<const T*>(weight), c, s, (uint32_t)units, (int)quads, heads, rotary, eps,
      strides[0], strides[1]);
  return cudaGetLastError() == cudaSuccess ? ANEMOI_SM100_OK : ANEMOI_SM100_ELAUNCH;
}

template <typename T>
int launch(void* x, const void* weight, const float* c, const float* s, int64_t tokens, int heads, int d,
           int rotary, float eps, const int64_t* strides, cudaStream_t st) {
  if (d == 64)
    return heads > 2 ? launch_rows<T, 64, 4>(x, weight, c, s, tokens, heads, rotary, eps, strides, st)
                     : launch_rows<T, 64, 1>(x, weight, c, s, tokens, heads, rotary, eps, strides, st);
  return heads > 2 ? launch_rows<T, 128, 4>(x, weight, c, s, tokens, heads, rotary, eps, strides, st)
                   : launch_rows<T, 128, 1>(x, weight, c, s, tokens, heads, rotary, eps, strides, st);
}

}  // namespace

extern "C" int anemoi_sm100_qknorm_rope(void* x, const void* weight, const float* cos_table,
                                        const float* sin_table, int64_t tokens, int32_t heads,
                                        int32_t head_dim, int32_t rotary_dim, float eps, int32_t is_bf16,
                                        const int64_t* strides, void* stream) {
  if (!x || !weight || !strides || tokens < 0 || heads <= 0) return ANEMOI_SM100_EINVAL;
  if (rotary_dim > 0 && (!cos_table || !sin_table)) return ANEMOI_SM100_EINVAL;
  if (head_dim != 64 && head_dim != 128) return ANEMOI_SM100_EINVAL;
  // the pairing j <-> j + rotary_dim/2 must move whole 8-channel vectors
  if (rotary_dim < 0 || rotary_dim > head_dim || rotary_dim % 16) return ANEMOI_SM100_EINVAL;
  if (strides[0] % 8 || strides[1] % 8 || !(eps >= 0.0f)) return ANEMOI_SM100_EINVAL;
  // every load and store takes 16 bytes
  for (const void* p : {static_cast<const void*>(x), weight, static_cast<const void*>(cos_table),
                        static_cast<const void*>(sin_table)})
    if (reinterpret_cast<uintptr_t>(p) % 16) return ANEMOI_SM100_EINVAL;
  if (tokens == 0) return ANEMOI_SM100_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return is_bf16 ? launch<__nv_bfloat16>(x, weight, cos_table, sin_table, tokens, heads, head_dim, rotary_dim,
                                         eps, strides, st)
                 : launch<__half>(x, weight, cos_table, sin_table, tokens, heads, head_dim, rotary_dim, eps,
                                  strides, st);
}
