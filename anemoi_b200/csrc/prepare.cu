// Gather + narrow + pool + quantise: one pass over raw Q/K/V that fills the
// operand store (tile records) every later kernel consumes.  HBM-bandwidth bound.
//
// One CTA = one (task, head).  A task is a video query tile, a video key/value
// block (QB rows = QB/64 stages), a prefix key/value stage, or a prefix query
// tile.  The CTA gathers the tile's rows with 16-byte loads into shared memory
// (narrowed to fp16), derives pools / amax / scales from shared memory, and
// streams the tile records out with 16-byte coalesced stores.
//
// Between HBM and issue bound: maxima are taken two halves at a time, V is read two channels
// at a time (lanes side by side; single halves 16 rows apart met in four banks), codes are
// packed by the converting instructions, and the quotients, sums and products are packed fp32 instructions (one value
// per instruction / two, with the maxima of V, us: 56 heads of D = 128 and S = 85,184, all cells, 11.5 GB, 2,281 / 2,230; S =
// 33,272 914 / 907, INT8 + FP16 with max pools 730 / 731; Q64 INT8, S = 38,247 601 / 588; NVFP4 D = 64, 4 heads of 84,672
// 58.1 / 55.0; 8 heads of 4,109 19.0 / 18.9).
//
// Numeric contract (reference: csrc/attention/cuda/sm120/q128_microscaling_preparation.cu):
//   narrow  bf16 -> f32 -> f16 rn (:227-232); invalid slots and prefix padding are +0 (:369-374)
//   mean    f16( sum_slots f32 in slot order / count ), IEEE division (:375-377,511-517)
//   max     over valid slots (:378-381)
//   INT8    scale = amax/127 + 1e-7; code = trunc(x/scale +- 0.5) (:458,503-506)
//   V E4M3  code = e4m3_satfinite(v * (2.25/amax_channel)); scale = amax/2.25 (:744-748,784-794)
//   NVFP4   scale = e4m3_satfinite((amax16/6)/gs); code = e2m1_rn(x/(e4m3(scale)*gs)) (:43-62)
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp4.h>
#include <cuda_fp8.h>

#include "layer.cuh"
#include "packed.cuh"
#include "records.cuh"

namespace {

using sm100::fadd2;
using sm100::ffma2;
using sm100::fmul2;

constexpr int kThreads = 256;
// CTAs per SM: 51 registers per thread for 128-row blocks, 32 for 64-row ones; fewer CTAs
// with more registers are slower (56 heads x 33,272 tokens: 759 us at four, 728 at five, 821 at six).
// Four where the CTAs of values find the maxima themselves: such grids are small, and the maxima's loads in flight need
// registers (with a query block's own limit 12 heads x 768 tokens of D = 128, Q64, 29.3 us a call, now 27.7; 2 x 1,040 of
// D = 64 25.4 and 23.7).
__host__ __device__ constexpr int min_ctas(int qb, bool own_maxima) { return own_maxima ? 4 : qb == 128 ? 5 : 8; }
constexpr int kPad = 8;  // halves of padding per shared-memory row

struct PrepParams {
  anemoi_sm100_shape s;
  anemoi_sm100_operands o;
  const void* q;
  const void* k;
  const void* v;
  const int32_t* indices;
  const int32_t* counts;
  int prefix_stages, stages, prefix_q_tiles;
  int64_t stride[6];  // token and head stride (elements) of q, k, v
};

// 8 raw 16-bit elements -> 8 fp16 (bf16 through fp32, round to nearest even; fp16 unchanged)
template <typename InT>
__device__ __forceinline__ uint4 narrow8(uint4 raw);
template <>
__device__ __forceinline__ uint4 narrow8<__half>(uint4 raw) {
  return raw;
}
template <>
__device__ __forceinline__ uint4 narrow8<__nv_bfloat16>(uint4 raw) {
  const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&raw);
  uint4 out;
  __half2* h = reinterpret_cast<__half2*>(&out);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 f = __bfloat1622float2(b[i]);
    h[i] = __floats2half2_rn(f.x, f.y);
  }
  return out;
}

__device__ __forceinline__ float block_max(float v, float* red) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = red[0];
#pragma unroll
  for (int w = 1; w < kThreads / 32; ++w) r = fmaxf(r, red[w]);
  return r;
}

__device__ __forceinline__ uint8_t nv_scale_byte(float amax, float gs) {
  return __nv_cvt_float_to_fp8(__fdiv_rn(__fdiv_rn(amax, 6.0f), gs), __NV_SATFINITE, __NV_E4M3);
}
__device__ __forceinline__ float e4m3_to_float(uint8_t bits) {
  __half_raw h = __nv_cvt_fp8_to_halfraw(bits, __NV_E4M3);
  return __half2float(*reinterpret_cast<__half*>(&h));
}
// Correctly rounded x / y, two at a time, from the correctly rounded reciprocal `inv` = 1/y shared by a
// whole group: q0 = x*inv, residual r = x - q0*y (exact in an FMA), q = q0 + r*inv.  For the
// normal-range operands here this equals IEEE division bit for bit at a third of its cost.
__device__ __forceinline__ float2 div_rn(float2 x, float y, float inv) {
  const float2 inv2 = make_float2(inv, inv);
  const float2 q0 = fmul2(x, inv2);
  const float2 r = ffma2(q0, make_float2(-y, -y), x);
  return ffma2(r, inv2, q0);
}
__device__ __forceinline__ uint8_t e2m1_pair(float2 x, float dq, float inv_dq) {
  if (dq == 0.0f) return 0;
  return __nv_cvt_float2_to_fp4x2(div_rn(x, dq, inv_dq), __NV_E2M1, cudaRoundNearest);
}
// trunc(x / scale +- 0.5); |result| <= 127
__device__ __forceinline__ int2 int8_codes(__half2 h, float scale, float inv_scale) {
  const float2 t = div_rn(__half22float2(h), scale, inv_scale);
  const auto half = [](float v) { return __int_as_float((__float_as_int(v) & 0x80000000) | 0x3f000000); };
  const float2 u = fadd2(t, make_float2(half(t.x), half(t.y)));
  return make_int2(__float2int_rz(u.x), __float2int_rz(u.y));
}
// Four codes as bytes, the first one lowest.
__device__ __forceinline__ uint32_t pack_s8(int2 lo, int2 hi) {
  uint32_t r;
  asm("{\n\t.reg .b32 t;\n\tcvt.pack.sat.s8.s32.b32 t, %4, %3, 0;\n\tcvt.pack.sat.s8.s32.b32 %0, %2, %1, t;\n\t}"
      : "=r"(r)
      : "r"(lo.x), "r"(lo.y), "r"(hi.x), "r"(hi.y));
  return r;
}
// The larger of two magnitudes, both halves at once.
__device__ __forceinline__ __half2 max_abs2(__half2 m, __half2 x) { return __hmax2(m, __habs2(x)); }

// Gathers ROWS rows into `tile` ([ROWS][D + kPad] halves), zero for invalid slots.  The trip
// count is a compile-time constant and the loop is split into a load pass and a store pass, so
// every thread has all of its 16-byte loads (and the slot-index loads before them) in flight at
// once: the kernel is bound by memory latency per CTA, not by arithmetic.
template <typename InT, int D, int ROWS>
__device__ __forceinline__ void gather_tile(__half* tile, const InT* src, const PrepParams& p,
                                            int head, bool video, int first_slot, int first_token,
                                            int valid_rows, int64_t token_stride,
                                            int64_t head_stride) {
  constexpr int kVec = D / 8;
  constexpr int kIter = ROWS * kVec / kThreads;
  static_assert(ROWS * kVec % kThreads == 0, "tile must be a multiple of the CTA's vector width");
  int64_t token[kIter];
#pragma unroll
  for (int i = 0; i < kIter; ++i) {
    const int r = (threadIdx.x + i * kThreads) / kVec;
    token[i] = r < valid_rows
                   ? (video ? (int64_t)p.s.prefix_tokens + __ldg(p.indices + first_slot + r)
                            : (int64_t)first_token + r)
                   : -1;
  }
  uint4 raw[kIter];
#pragma unroll
  for (int i = 0; i < kIter; ++i) {
    const int c8 = (threadIdx.x + i * kThreads) % kVec;
    raw[i] = make_uint4(0, 0, 0, 0);
    if (token[i] >= 0)
      raw[i] = __ldg(reinterpret_cast<const uint4*>(src + token[i] * token_stride +
                                                    (int64_t)head * head_stride + c8 * 8));
  }
#pragma unroll
  for (int i = 0; i < kIter; ++i) {
    const int idx = threadIdx.x + i * kThreads;
    const int r = idx / kVec, c8 = idx % kVec;
    *reinterpret_cast<uint4*>(tile + r * (D + kPad) + c8 * 8) = narrow8<InT>(raw[i]);
  }
}

// fp16 tile record (K-major image of `rows` x D; also used for the MN-major V tile).
template <int D>
__device__ __forceinline__ void write_fp16_tile(uint8_t* dst, const __half* tile, int row0,
                                                int rows) {
  constexpr int kChunks = D / 8;
  for (int idx = threadIdx.x; idx < rows * kChunks; idx += kThreads) {
    const int r = (idx / (8 * kChunks)) * 8 + (idx & 7), j = (idx >> 3) % kChunks;
    *reinterpret_cast<uint4*>(dst + (size_t)idx * 16) =
        *reinterpret_cast<const uint4*>(tile + (row0 + r) * (D + kPad) + j * 8);
  }
}

template <int D>
__device__ __forceinline__ float tile_amax(const __half* tile, int row0, int rows, float* red) {
  constexpr int kVec = D / 8;
  __half2 m2 = __half2(__half(0.0f), __half(0.0f));
  for (int idx = threadIdx.x; idx < rows * kVec; idx += kThreads) {
    const int r = idx / kVec, c8 = idx % kVec;
    const uint4 raw = *reinterpret_cast<const uint4*>(tile + (row0 + r) * (D + kPad) + c8 * 8);
    const __half2* h = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) m2 = max_abs2(m2, h[i]);
  }
  const float m = __half2float(__hmax(m2.x, m2.y));
  return block_max(m, red);
}

template <int D>
__device__ __forceinline__ void write_int8_tile(uint8_t* dst, const __half* tile, int row0,
                                                int rows, float scale) {
  constexpr int kChunks = D / 16;
  const float inv_scale = __frcp_rn(scale);
  for (int idx = threadIdx.x; idx < rows * kChunks; idx += kThreads) {
    const int r = (idx / (8 * kChunks)) * 8 + (idx & 7), j = (idx >> 3) % kChunks;
    const __half* src = tile + (row0 + r) * (D + kPad) + j * 16;
    uint4 a = *reinterpret_cast<const uint4*>(src), b = *reinterpret_cast<const uint4*>(src + 8);
    const __half2* ha = reinterpret_cast<const __half2*>(&a);
    const __half2* hb = reinterpret_cast<const __half2*>(&b);
    const auto four = [&](__half2 lo, __half2 hi) {
      return pack_s8(int8_codes(lo, scale, inv_scale), int8_codes(hi, scale, inv_scale));
    };
    const uint4 out = make_uint4(four(ha[0], ha[1]), four(ha[2], ha[3]), four(hb[0], hb[1]), four(hb[2], hb[3]));
    *reinterpret_cast<uint4*>(dst + (size_t)idx * 16) = out;
  }
}

// NVFP4 K-major tile (rows x D, groups of 16 channels) + scale blocks.
template <int D>
__device__ __forceinline__ void write_nvfp4_rows(uint8_t* codes, uint8_t* sf, const __half* tile,
                                                 int row0, int rows, float gs) {
  constexpr int kChunks = D / 32;
  for (int idx = threadIdx.x; idx < rows * kChunks; idx += kThreads) {
    const int r = (idx / (8 * kChunks)) * 8 + (idx & 7), j = (idx >> 3) % kChunks;
    const __half* src = tile + (row0 + r) * (D + kPad) + j * 32;
    uint4 out;
    uint8_t* c = reinterpret_cast<uint8_t*>(&out);
    uint8_t sb[2];
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      uint4 a = *reinterpret_cast<const uint4*>(src + g * 16);
      uint4 b = *reinterpret_cast<const uint4*>(src + g * 16 + 8);
      float2 x[8];
      const __half2* ha = reinterpret_cast<const __half2*>(&a);
      const __half2* hb = reinterpret_cast<const __half2*>(&b);
      __half2 m2 = __hmax2(__habs2(ha[0]), __habs2(hb[0]));
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        x[i] = __half22float2(ha[i]);
        x[4 + i] = __half22float2(hb[i]);
        if (i > 0) m2 = max_abs2(max_abs2(m2, ha[i]), hb[i]);
      }
      // (a group of NaNs alone has maximum zero, like one with no values: its scale byte and codes are zero)
      const float amax = fmaxf(__half2float(__hmax(m2.x, m2.y)), 0.0f);
      sb[g] = nv_scale_byte(amax, gs);
      const float dq = __fmul_rn(e4m3_to_float(sb[g]), gs);
      const float inv_dq = __frcp_rn(dq);
#pragma unroll
      for (int i = 0; i < 8; ++i) c[g * 8 + i] = e2m1_pair(x[i], dq, inv_dq);
    }
    *reinterpret_cast<uint4*>(codes + (size_t)idx * 16) = out;
    uint8_t* s = sf + (j >> 1) * 512 + rec::sf_offset(r, (j & 1) * 2);
    *reinterpret_cast<uint16_t*>(s) = (uint16_t)sb[0] | ((uint16_t)sb[1] << 8);
  }
}

// V^T tiles of one 64-key stage: channels x keys, keys contiguous.  A thread takes two neighbouring
// channels of 16 keys: 4-byte reads, lanes side by side along the channels.
template <int D>
__device__ __forceinline__ void write_v_e4m3(uint8_t* dst, const __half* tile, int row0,
                                             const float* recip) {
  for (int idx = threadIdx.x; idx < D * 2; idx += kThreads) {
    const int c = idx % (D / 2) * 2, jj = idx / (D / 2);
    const float2 rc = *reinterpret_cast<const float2*>(recip + c);
    const __half* src = tile + (row0 + jj * 16) * (D + kPad) + c;
    uint4 out[2];
    uint16_t* o0 = reinterpret_cast<uint16_t*>(&out[0]);
    uint16_t* o1 = reinterpret_cast<uint16_t*>(&out[1]);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 a = __half22float2(*reinterpret_cast<const __half2*>(src + 2 * i * (D + kPad)));
      const float2 b = __half22float2(*reinterpret_cast<const __half2*>(src + (2 * i + 1) * (D + kPad)));
      // (a channel whose factor is zero holds zeros only)
      const float2 sa = fmul2(a, rc), sb = fmul2(b, rc);
      o0[i] = __nv_cvt_float2_to_fp8x2(make_float2(sa.x, sb.x), __NV_SATFINITE, __NV_E4M3);
      o1[i] = __nv_cvt_float2_to_fp8x2(make_float2(sa.y, sb.y), __NV_SATFINITE, __NV_E4M3);
    }
    if (rc.x == 0.0f) out[0] = make_uint4(0, 0, 0, 0);
    if (rc.y == 0.0f) out[1] = make_uint4(0, 0, 0, 0);
    uint4* to = reinterpret_cast<uint4*>(dst + rec::tile_offset(c, jj, 4));
    to[0] = out[0];
    to[1] = out[1];
  }
}

template <int D>
__device__ __forceinline__ void write_v_nvfp4(uint8_t* codes, uint8_t* sf, const __half* tile,
                                              int row0, float gs) {
  // a thread: two neighbouring channels, 16 of the 64 keys
  for (int idx = threadIdx.x; idx < D * 2; idx += kThreads) {
    const int c = idx % (D / 2) * 2, jg = idx / (D / 2);
    const __half* src = tile + (row0 + jg * 16) * (D + kPad) + c;
    float2 x[16];
    __half2 m2 = __half2(__half(0.0f), __half(0.0f));
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const __half2 h = *reinterpret_cast<const __half2*>(src + i * (D + kPad));
      m2 = max_abs2(m2, h);
      x[i] = __half22float2(h);
    }
    const float2 amax = __half22float2(m2);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const uint8_t sb = nv_scale_byte(k ? amax.y : amax.x, gs);
      const float dq = __fmul_rn(e4m3_to_float(sb), gs);
      const float inv_dq = __frcp_rn(dq);
      uint2 out;
      uint8_t* o = reinterpret_cast<uint8_t*>(&out);
#pragma unroll
      for (int i = 0; i < 8; ++i)
        o[i] = e2m1_pair(k ? make_float2(x[2 * i].y, x[2 * i + 1].y) : make_float2(x[2 * i].x, x[2 * i + 1].x), dq, inv_dq);
      *reinterpret_cast<uint2*>(codes + rec::tile_offset(c + k, jg >> 1, 2) + (jg & 1) * 8) = out;
      sf[rec::sf_offset(c + k, jg)] = sb;
    }
  }
}

template <int D>
// `second`: the extra pool holds the second moments (mean of the squares, one FMA per row in
// row order; padding rows are zero) instead of the maxima - the diag-Jensen draft map's input.
__device__ __forceinline__ void write_pools(const __half* tile, int rows, int count, __half* mean,
                                            __half* maxp, bool second) {
  // a thread: two neighbouring channels, all rows in order
  if (threadIdx.x < D / 2) {
    const int c = threadIdx.x * 2;
    const __half* src = tile + c;
    float2 sum = make_float2(0.0f, 0.0f);
    if (maxp == nullptr) {
#pragma unroll 16
      for (int r = 0; r < rows; ++r) {
        const float2 x = __half22float2(*reinterpret_cast<const __half2*>(src + r * (D + kPad)));
        sum = fadd2(sum, x);
      }
    } else {
      float2 sq = make_float2(0.0f, 0.0f), mx = make_float2(-INFINITY, -INFINITY);
#pragma unroll 8
      for (int r = 0; r < rows; ++r) {
        const float2 x = __half22float2(*reinterpret_cast<const __half2*>(src + r * (D + kPad)));
        sum = fadd2(sum, x);
        if (second) {
          sq = ffma2(x, x, sq);
        } else if (r < count) {
          mx.x = fmaxf(mx.x, x.x);
          mx.y = fmaxf(mx.y, x.y);
        }
      }
      if (second) mx = make_float2(__fdiv_rn(sq.x, (float)count), __fdiv_rn(sq.y, (float)count));
      *reinterpret_cast<__half2*>(maxp + c) = __floats2half2_rn(mx.x, mx.y);
    }
    *reinterpret_cast<__half2*>(mean + c) =
        __floats2half2_rn(__fdiv_rn(sum.x, (float)count), __fdiv_rn(sum.y, (float)count));
  }
}

// Two 16-bit magnitudes at a time; a NaN never wins (as fmaxf).
template <typename InT>
struct Abs2;
template <>
struct Abs2<__half> {
  using T = __half2;
};
template <>
struct Abs2<__nv_bfloat16> {
  using T = __nv_bfloat162;
};

// max |v| of channel threadIdx.x over every token of a short sequence (as v_amax_kernel finds it); `part`: 4 KB.
template <typename InT, int D>
__device__ __forceinline__ float channel_maximum(const InT* v, const PrepParams& p, int head, void* part) {
  using T2 = typename Abs2<InT>::T;
  constexpr int kVec = D / 8, kLanes = kThreads / kVec;
  const int x = threadIdx.x % kVec, y = threadIdx.x / kVec;
  const InT* src = v + (int64_t)head * p.stride[5] + x * 8;
  T2 m[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) m[i] = T2(InT(0.0f), InT(0.0f));
#pragma unroll 8
  for (int t = y; t < p.s.seq_tokens; t += kLanes) {
    const uint4 raw = __ldg(reinterpret_cast<const uint4*>(src + (int64_t)t * p.stride[4]));
    const T2* h = reinterpret_cast<const T2*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) m[i] = __hmax2(m[i], __habs2(h[i]));
  }
  T2* own = static_cast<T2*>(part) + threadIdx.x * 4;
#pragma unroll
  for (int i = 0; i < 4; ++i) own[i] = m[i];
  __syncthreads();
  float found = 0.0f;
  if (threadIdx.x < D) {
    const int c = threadIdx.x;
    const T2* all = static_cast<const T2*>(part) + (c / 8) * 4 + c % 8 / 2;
    T2 r = all[0];
    for (int k = 1; k < kLanes; ++k) r = __hmax2(r, all[k * kVec * 4]);
    found = __half2float(__float2half_rn(static_cast<float>(c & 1 ? r.y : r.x)));
  }
  __syncthreads();
  return found;
}

// Tasks of a head, in grid order: query tiles (video, prefix), then key/value blocks (R video blocks
// of QB rows = QB/64 stages each, then the 64-row prefix stages).  With kSplit keys and values of a
// block are separate CTAs (all keys first).  kOwnMaxima: of a short sequence's V, by every CTA of values, with no
// kernel before this one.
// kCells: a kernel holds the quantisers of the cells that its call may have.  They need the most registers, and what
// is live around them is spilled for every call of the kernel (at 32 and 48 registers).  Of all cells / of the
// call's, 16 heads x 33,272 tokens of D = 64, fp16, us: FP16 alone Q64 80.0 / 77.3, with max pools 100.5 / 79.8,
// Q128 87.1 / 84.7; INT8 Q64 102 / 98.5, with max pools 132.5 / 102.
enum Cells { kFp16Alone, kNoNvfp4, kAllCells };
template <typename InT, int QB, int D, bool kSplit, bool kOwnMaxima, Cells kCells>
__global__ void __launch_bounds__(kThreads, min_ctas(QB, kOwnMaxima)) prepare_kernel(PrepParams p) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  __half* tile = reinterpret_cast<__half*>(smem_raw);
  __shared__ float red[kThreads / 32];
  __shared__ float recip[D];

  // (read anew where they are asked for: kept, they take the registers that this is about)
  const auto has_int8 = [&] { return kCells != kFp16Alone && p.s.has_int8; };
  const auto has_nvfp4 = [&] { return kCells == kAllCells && p.s.has_nvfp4; };

  layer::grid_dependency_trigger();
  const int R = p.s.video_blocks;
  // heads vary fastest across concurrently running CTAs: neighbours read adjacent 2*D-byte
  // pieces of the same token rows
  const int task = blockIdx.x / p.s.heads, head = blockIdx.x - task * p.s.heads;
  constexpr int kF = QB / 64;
  const int64_t qtiles_i8 = R + p.prefix_q_tiles;

  if (task < qtiles_i8) {
    // ---------------- query tile (video or prefix) ----------------
    // (after the maxima's kernel, whose CTAs all began when what was before it in the stream was
    // complete; without INT8 there is no such kernel)
    if (kOwnMaxima || !has_int8()) layer::grid_dependency_wait();
    const bool video = task < R;
    const int t = video ? task : task - R;
    const int valid = video ? p.counts[t] : min(QB, p.s.prefix_tokens - t * QB);
    gather_tile<InT, D, QB>(tile, static_cast<const InT*>(p.q), p, head, video, t * QB, t * QB, valid, p.stride[0],
                            p.stride[1]);
    __syncthreads();
    if (video) {
      __half* mean = static_cast<__half*>(p.o.q_pool) + ((int64_t)head * R + t) * D;
      __half* mx = p.s.has_maxpool
                       ? static_cast<__half*>(p.o.q_max_pool) + ((int64_t)head * R + t) * D
                       : nullptr;
      write_pools<D>(tile, QB, valid, mean, mx, p.s.has_maxpool == 2);
      if (p.s.has_fp16) {
        write_fp16_tile<D>(static_cast<uint8_t*>(p.o.q_fp16) +
                               ((int64_t)head * R + t) * rec::q_fp16_bytes(QB, D),
                           tile, 0, QB);
      }
      if (has_nvfp4()) {
        uint8_t* r4 = static_cast<uint8_t*>(p.o.q_nvfp4) +
                      ((int64_t)head * R + t) * rec::q_nvfp4_bytes(QB, D);
        write_nvfp4_rows<D>(r4, r4 + QB * D / 2, tile, 0, QB, p.s.q_global_scale);
      }
    }
    if (has_int8()) {
      const int64_t slot = (int64_t)head * qtiles_i8 + task;
      const float amax = tile_amax<D>(tile, 0, QB, red);
      const float scale = __fadd_rn(__fdiv_rn(amax, 127.0f), 1.0e-7f);
      if (threadIdx.x == 0) p.o.q_int8_scale[slot] = scale;
      write_int8_tile<D>(static_cast<uint8_t*>(p.o.q_int8) + slot * rec::q_int8_bytes(QB, D), tile,
                         0, QB, scale);
    }
    return;
  }

  // ---------------- key or value block (video) or stage (prefix) ----------------
  const int blocks = R + p.prefix_stages;
  const bool second_half = kSplit && task >= qtiles_i8 + blocks;
  const int block = task - (int)qtiles_i8 - (second_half ? blocks : 0);
  const bool video = block < R;
  const int b = video ? block : block - R;
  const int nst = video ? kF : 1;
  const int stage0 = video ? p.prefix_stages + b * kF : b;
  if (kOwnMaxima || !has_int8()) layer::grid_dependency_wait();  // (the layout's tables, too, may be new)
  const int valid = video ? p.counts[b] : min(64, p.s.prefix_tokens - b * 64);
  const int64_t rec0 = (int64_t)head * p.stages + stage0;
  auto gather = [&](const void* src, int64_t token_stride, int64_t head_stride) {
    if (video) {
      gather_tile<InT, D, QB>(tile, static_cast<const InT*>(src), p, head, true, b * QB, 0, valid, token_stride,
                              head_stride);
    } else {
      gather_tile<InT, D, 64>(tile, static_cast<const InT*>(src), p, head, false, 0, b * 64, valid, token_stride,
                              head_stride);
    }
  };
  if (!second_half) {
    gather(p.k, p.stride[2], p.stride[3]);
    __syncthreads();
    if (video) {
      __half* mean = static_cast<__half*>(p.o.k_pool) + ((int64_t)head * R + b) * D;
      __half* mx = p.s.has_maxpool
                       ? static_cast<__half*>(p.o.k_max_pool) + ((int64_t)head * R + b) * D
                       : nullptr;
      write_pools<D>(tile, QB, valid, mean, mx, p.s.has_maxpool == 2);
    }
    for (int g = 0; g < nst; ++g) {
      if (p.s.has_fp16) {
        write_fp16_tile<D>(static_cast<uint8_t*>(p.o.kv_fp16) + (rec0 + g) * rec::kv_fp16_bytes(D),
                           tile, g * 64, 64);
      }
      if (has_nvfp4()) {
        uint8_t* r4 = static_cast<uint8_t*>(p.o.kv_nvfp4) + (rec0 + g) * rec::kv_nvfp4_bytes(D);
        write_nvfp4_rows<D>(r4, r4 + rec::kv_nvfp4_ksf_offset(D), tile, g * 64, 64,
                            p.s.k_global_scale);
      }
      if (has_int8()) {
        const float amax = tile_amax<D>(tile, g * 64, 64, red);
        const float scale = __fadd_rn(__fdiv_rn(amax, 127.0f), 1.0e-7f);
        if (threadIdx.x == 0) p.o.k_int8_scale[rec0 + g] = scale;
        write_int8_tile<D>(static_cast<uint8_t*>(p.o.kv_int8) + (rec0 + g) * rec::kv_int8_bytes(D),
                           tile, g * 64, 64, scale);
      }
    }
    if (kSplit) return;
    __syncthreads();
  }

  // ---- values of the same rows ----
  float maximum = 0.0f;
  if constexpr (kOwnMaxima) {
    maximum = channel_maximum<InT, D>(static_cast<const InT*>(p.v), p, head, tile);
    if (block == 0 && threadIdx.x < D) p.o.v_amax[(int64_t)head * D + threadIdx.x] = maximum;
  }
  gather(p.v, p.stride[4], p.stride[5]);
  if (has_int8()) {
    if (!kOwnMaxima) layer::grid_dependency_wait();
    if (threadIdx.x < D) {
      const float amax =
          kOwnMaxima ? maximum : __half2float(__float2half_rn(p.o.v_amax[(int64_t)head * D + threadIdx.x]));
      recip[threadIdx.x] = amax == 0.0f ? 0.0f : __fdiv_rn(2.25f, amax);
      if (block == 0) p.o.v_e4m3_scale[(int64_t)head * D + threadIdx.x] = __fdiv_rn(amax, 2.25f);
    }
  }
  __syncthreads();
  for (int g = 0; g < nst; ++g) {
    if (p.s.has_fp16) {
      write_fp16_tile<D>(static_cast<uint8_t*>(p.o.kv_fp16) + (rec0 + g) * rec::kv_fp16_bytes(D) +
                             64 * D * 2,
                         tile, g * 64, 64);
    }
    if (has_int8()) {
      write_v_e4m3<D>(static_cast<uint8_t*>(p.o.kv_int8) + (rec0 + g) * rec::kv_int8_bytes(D) +
                          64 * D,
                      tile, g * 64, recip);
    }
    if (has_nvfp4()) {
      uint8_t* r4 = static_cast<uint8_t*>(p.o.kv_nvfp4) + (rec0 + g) * rec::kv_nvfp4_bytes(D);
      write_v_nvfp4<D>(r4 + rec::kv_nvfp4_v_offset(D), r4 + rec::kv_nvfp4_vsf_offset(D), tile,
                       g * 64, p.s.v_global_scale);
    }
  }
}

// max |v| per (head, channel) over every token, as the bit pattern of a non-negative float
// (integer max == float max).  The token ranges' maxima meet in global atomics (`out` must be zeroed
// first) or, kCluster, in one cluster's shared memory.  A pure read of V, so HBM bound; the
// maximum is taken in the input's own type (rounding to fp16 is monotonic and happens once at
// the end).  One CTA = 32 vectors of 8 channels x 8 token lanes, four 16-byte loads in flight per
// thread, and about three CTAs per SM whatever the number of heads: with one thread per vector
// walking 128 tokens alone, V of 7 heads x 33,272 tokens (60 MB) took 60 us, now 15.
constexpr int kAmaxLanes = 8;
template <typename InT, bool kCluster>
__global__ void __launch_bounds__(32 * kAmaxLanes) v_amax_kernel(const InT* v, int* out, int64_t tokens,
                                                                 int heads, int d8, int64_t token_stride,
                                                                 int64_t head_stride, int tokens_per_block) {
  using T2 = typename Abs2<InT>::T;
  __shared__ T2 part[kAmaxLanes][32][4 + 1];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int col8 = blockIdx.x * 32 + x;
  const bool live = col8 < heads * d8;
  layer::grid_dependency_wait();
  layer::grid_dependency_trigger();
  T2 m[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) m[i] = T2(InT(0.0f), InT(0.0f));
  if (live) {
    const InT* src = v + (int64_t)(col8 / d8) * head_stride + (col8 % d8) * 8;
    const int64_t t0 = (int64_t)blockIdx.y * tokens_per_block;
    const int64_t t1 = min(tokens, t0 + tokens_per_block);
    int64_t t = t0 + y;
    for (; t + 3 * kAmaxLanes < t1; t += 4 * kAmaxLanes) {
      uint4 raw[4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        raw[k] = __ldg(reinterpret_cast<const uint4*>(src + (t + k * kAmaxLanes) * token_stride));
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const T2* h = reinterpret_cast<const T2*>(&raw[k]);
#pragma unroll
        for (int i = 0; i < 4; ++i) m[i] = __hmax2(m[i], __habs2(h[i]));
      }
    }
    for (; t < t1; t += kAmaxLanes) {
      const uint4 raw = __ldg(reinterpret_cast<const uint4*>(src + t * token_stride));
      const T2* h = reinterpret_cast<const T2*>(&raw);
#pragma unroll
      for (int i = 0; i < 4; ++i) m[i] = __hmax2(m[i], __habs2(h[i]));
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) part[y][x][i] = m[i];
  __syncthreads();
  // thread (x, y) finishes channel y of vector x
  T2 r = part[0][x][y >> 1];
#pragma unroll
  for (int k = 1; k < kAmaxLanes; ++k) r = __hmax2(r, part[k][x][y >> 1]);
  const int found = __float_as_int(__half2float(__float2half_rn(static_cast<float>(y & 1 ? r.y : r.x))));
  if (kCluster) {
    namespace cg = cooperative_groups;
    __shared__ int mine[32 * kAmaxLanes];
    cg::cluster_group cluster = cg::this_cluster();
    mine[threadIdx.x] = found;
    cluster.sync();
    if (cluster.block_rank() == 0 && live) {
      int all = found;
      for (int c = 1; c < (int)cluster.num_blocks(); ++c) all = max(all, cluster.map_shared_rank(mine, c)[threadIdx.x]);
      out[col8 * 8 + y] = all;
    }
    cluster.sync();  // no CTA leaves while its maxima are read
  } else if (live) {
    atomicMax(out + col8 * 8 + y, found);
  }
}

// The maxima start at zero: a kernel and not a memset, which would wait for all before it and hold up what follows.  Calls
// with the memset / with this, us: 8 heads x 4,109 tokens 77.2 / 75.4, 13 x 2,892 65.4 / 62.0, 1 x 3,276 42.8 / 40.0, 6 x 2,420
// 35.8 / 33.0, 14 x 3,760 141.7 / 139.2.
constexpr int kZeroThreads = 512;
__global__ void __launch_bounds__(kZeroThreads) zero_kernel(int* out, int n) {
  layer::grid_dependency_trigger();
  layer::grid_dependency_wait();
  for (int i = blockIdx.x * kZeroThreads + threadIdx.x; i < n; i += gridDim.x * kZeroThreads) out[i] = 0;
}

// Values of a head up to which every CTA of values finds the maxima of V itself: reading 192 KB from L2 takes 1-2 us, a
// kernel for them 4 and its launch 2.5 on the host.  Every such CTA reads all of its head's V, so their number is
// bounded, too.  Calls of INT8, us, with the kernel / without, one after another: D = 64 Q64 4 heads x 1,024 tokens 25.1 /
// 23.5, 6 x 1,536 (144 CTAs) 30.2 / 27.7, Q128 12 x 1,536 30.8 / 27.9; D = 128 Q64 12 x 768 28.0 / 27.7, Q128 24 x 768 30.8 / 28.7;
// with 256 prefix tokens Q64 6 x 1,536 of D = 64 37.3 / 37.1, Q128 18 x 768 of D = 128 35.8 / 35.1.  Alone each gains 1-4; the
// worst is 5 x 1,480 with 200 prefix tokens, Q64 D = 64: 35.9 / 36.9 one after another, 57.2 / 54.9 alone.  Past the lines, in an
// earlier form: 3 x 2,040 of D = 64 33.4 / 33.1, 30 x 2,040 (960 CTAs) 61 / 68, 40 x 2,040 of D = 128 93 / 119.
constexpr int64_t kOwnMaximaValues = 96 * 1024;
inline bool own_maxima(const anemoi_sm100_shape& s) {
  return s.has_int8 && (int64_t)s.seq_tokens * s.head_dim <= kOwnMaximaValues &&
         ((int64_t)s.video_blocks + rec::prefix_stages(s)) * s.heads <= 148;
}

// The grid of the kernel of the maxima: about three CTAs per SM, each with at least sixteen loads per thread: every CTA
// ends in 256 atomics (8 heads x 4,109 tokens with eight per SM and two loads: the preparation took 40 us, now 24).
inline int maxima_chunks(const anemoi_sm100_shape& s) { return (s.heads * s.head_dim / 8 + 31) / 32; }
inline int maxima_tokens(const anemoi_sm100_shape& s) {
  const int rows = max(1, 3 * 148 / maxima_chunks(s));
  return max(16 * kAmaxLanes, (s.seq_tokens + rows - 1) / rows);
}
// Up to eight token ranges are one cluster, which needs no zeroed memory: a launch less, and nothing
// between this kernel and what was before it (1,024 tokens x 4 heads: the call 36.5 -> 34.4 us).
inline bool zeroes_maxima(const anemoi_sm100_shape& s) {
  return s.has_int8 && !own_maxima(s) && (s.seq_tokens + maxima_tokens(s) - 1) / maxima_tokens(s) > 8;
}
// With FP16 prefix queries by a memset, for those that torch's attention computes on another stream: its wait lets their few
// long CTAs in first, each on an SM of its own.  Calls of INT8 cells, us, memset / kernel: 14 heads x 10,872 tokens with 512 of
// prefix 370 / 377, 14 x 6,940 with 700 203 / 214, 3 x 18,940 with 700 230 / 238.  Beside dense rows of this library the two are
// alike: 8 x 2,542 with 62 49.1 / 50.2, 1 x 3,990 with 150 49.2 / 48.4, 30 x 18,782 with 62 1,639 / 1,647, 5 x 19,302 with 62
// 305.0 / 304.5.
inline bool zeroes_by_memset(const anemoi_sm100_shape& s) { return s.prefix_tokens > 0 && !s.has_prefix_query_int8; }

template <typename InT, int QB, int D, bool kSplit, bool kOwnMaxima, Cells kCells>
int launch(const PrepParams& p, cudaStream_t stream) {
  const size_t smem = (size_t)QB * (D + kPad) * sizeof(__half);
  auto kernel = prepare_kernel<InT, QB, D, kSplit, kOwnMaxima, kCells>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
      cudaSuccess)
    return ANEMOI_SM100_ELAUNCH;
  if (p.s.has_int8 && !kOwnMaxima) {
    const int tokens_per_block = maxima_tokens(p.s);
    dim3 grid(maxima_chunks(p.s), (p.s.seq_tokens + tokens_per_block - 1) / tokens_per_block);
    cudaError_t err;
    if (!zeroes_maxima(p.s)) {
      err = layer::launch_cluster(v_amax_kernel<InT, true>, grid, dim3(1, grid.y), dim3(32 * kAmaxLanes), 0, stream,
                                  static_cast<const InT*>(p.v), reinterpret_cast<int*>(p.o.v_amax), p.s.seq_tokens,
                                  p.s.heads, D / 8, p.stride[4], p.stride[5], tokens_per_block);
    } else {
      const int n = p.s.heads * D;
      if (zeroes_by_memset(p.s))
        err = cudaMemsetAsync(p.o.v_amax, 0, sizeof(float) * n, stream);
      else
        err = layer::launch(zero_kernel, dim3(min(148, (n + kZeroThreads - 1) / kZeroThreads)), dim3(kZeroThreads), 0, stream,
                          reinterpret_cast<int*>(p.o.v_amax), n);
      if (err == cudaSuccess)
        err = layer::launch(v_amax_kernel<InT, false>, grid, dim3(32 * kAmaxLanes), 0, stream,
                            static_cast<const InT*>(p.v), reinterpret_cast<int*>(p.o.v_amax), p.s.seq_tokens,
                            p.s.heads, D / 8, p.stride[4], p.stride[5], tokens_per_block);
    }
    if (err != cudaSuccess) return ANEMOI_SM100_ELAUNCH;
  }
  const int64_t blocks = (int64_t)p.s.video_blocks + p.prefix_stages;
  const int64_t tasks = p.s.video_blocks + p.prefix_q_tiles + (kSplit ? 2 : 1) * blocks;
  if (tasks * p.s.heads > INT32_MAX) return ANEMOI_SM100_ELIMIT;
  const dim3 grid((unsigned)(tasks * p.s.heads));
  return layer::launch(kernel, grid, dim3(kThreads), smem, stream, p) == cudaSuccess ? ANEMOI_SM100_OK
                                                                                    : ANEMOI_SM100_ELAUNCH;
}

}  // namespace

extern "C" int anemoi_sm100_arch(void) { return 100; }

extern "C" int anemoi_sm100_prepare_kernels(const anemoi_sm100_shape* shape) {
  return rec::validate_shape(shape) == ANEMOI_SM100_OK ? 1 + (shape->has_int8 && !own_maxima(*shape)) : 0;
}

extern "C" int anemoi_sm100_prepare_zero_kernels(const anemoi_sm100_shape* shape) {
  return rec::validate_shape(shape) == ANEMOI_SM100_OK && zeroes_maxima(*shape) && !zeroes_by_memset(*shape);
}

extern "C" int64_t anemoi_sm100_operand_bytes(const anemoi_sm100_shape* s, int which) {
  if (rec::validate_shape(s) != ANEMOI_SM100_OK) return ANEMOI_SM100_EINVAL;
  const int64_t H = s->heads, D = s->head_dim, QB = s->query_block, R = s->video_blocks;
  const int64_t NS = rec::stages(*s), PQ = rec::prefix_query_tiles(*s);
  switch (which) {
    case ANEMOI_SM100_BUF_Q_FP16: return s->has_fp16 ? H * R * rec::q_fp16_bytes(QB, D) : 0;
    case ANEMOI_SM100_BUF_KV_FP16: return s->has_fp16 ? H * NS * rec::kv_fp16_bytes(D) : 0;
    case ANEMOI_SM100_BUF_Q_INT8: return s->has_int8 ? H * (R + PQ) * rec::q_int8_bytes(QB, D) : 0;
    case ANEMOI_SM100_BUF_KV_INT8: return s->has_int8 ? H * NS * rec::kv_int8_bytes(D) : 0;
    case ANEMOI_SM100_BUF_Q_NVFP4: return s->has_nvfp4 ? H * R * rec::q_nvfp4_bytes(QB, D) : 0;
    case ANEMOI_SM100_BUF_KV_NVFP4: return s->has_nvfp4 ? H * NS * rec::kv_nvfp4_bytes(D) : 0;
    case ANEMOI_SM100_BUF_Q_INT8_SCALE: return s->has_int8 ? H * (R + PQ) * 4 : 0;
    case ANEMOI_SM100_BUF_K_INT8_SCALE: return s->has_int8 ? H * NS * 4 : 0;
    case ANEMOI_SM100_BUF_V_E4M3_SCALE: return s->has_int8 ? H * D * 4 : 0;
    case ANEMOI_SM100_BUF_V_AMAX: return s->has_int8 ? H * D * 4 : 0;
    case ANEMOI_SM100_BUF_POOL: return H * R * D * 2;
    default: return ANEMOI_SM100_EINVAL;
  }
}

extern "C" int anemoi_sm100_prepare(const anemoi_sm100_shape* shape, const void* q, const void* k,
                                    const void* v, const int64_t* strides, const int32_t* indices,
                                    const int32_t* counts, const anemoi_sm100_operands* out,
                                    void* stream) {
  if (rec::validate_shape(shape) != ANEMOI_SM100_OK || !q || !k || !v || !indices || !counts || !out)
    return ANEMOI_SM100_EINVAL;
  const anemoi_sm100_shape& s = *shape;
  if (!out->q_pool || !out->k_pool) return ANEMOI_SM100_EINVAL;
  if (s.has_maxpool && (!out->q_max_pool || !out->k_max_pool)) return ANEMOI_SM100_EINVAL;
  if (s.has_fp16 && (!out->q_fp16 || !out->kv_fp16)) return ANEMOI_SM100_EINVAL;
  if (s.has_int8 && (!out->q_int8 || !out->kv_int8 || !out->q_int8_scale || !out->k_int8_scale ||
                     !out->v_e4m3_scale || !out->v_amax))
    return ANEMOI_SM100_EINVAL;
  if (s.has_nvfp4 && (!out->q_nvfp4 || !out->kv_nvfp4)) return ANEMOI_SM100_EINVAL;
  PrepParams p;
  p.s = s;
  p.o = *out;
  p.q = q;
  p.k = k;
  p.v = v;
  p.indices = indices;
  p.counts = counts;
  for (int i = 0; i < 6; ++i) {
    p.stride[i] = strides ? strides[i] : (i & 1 ? (int64_t)s.head_dim : (int64_t)s.heads * s.head_dim);
    if (p.stride[i] <= 0 || p.stride[i] % 8) return ANEMOI_SM100_EINVAL;
  }
  p.prefix_stages = rec::prefix_stages(s);
  p.stages = rec::stages(s);
  p.prefix_q_tiles = rec::prefix_query_tiles(s);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // Keys and values of a block in CTAs of their own: half the serial chain, which is quicker for
  // 128-row blocks (sweep's 4 heads 71 -> 64 us, 56 heads x 85,184 tokens 2,178 -> 2,128) and for small grids; for
  // many 64-row blocks a CTA's fixed cost weighs more (620 -> 687).
  const bool own = own_maxima(s);  // (a grid that small is split)
  const bool split = s.query_block == 128 || ((int64_t)2 * s.video_blocks + p.prefix_stages) * s.heads <= 4 * 148;
#define ANEMOI_DIM(T, QB, SPLIT, OWN, CELLS) \
  (s.head_dim == 64 ? launch<T, QB, 64, SPLIT, OWN, CELLS>(p, st) : launch<T, QB, 128, SPLIT, OWN, CELLS>(p, st))
#define ANEMOI_CELLS(T, QB, SPLIT)                                                                        \
  (s.has_nvfp4  ? (own ? ANEMOI_DIM(T, QB, true, true, kAllCells) : ANEMOI_DIM(T, QB, SPLIT, false, kAllCells)) \
   : s.has_int8 ? (own ? ANEMOI_DIM(T, QB, true, true, kNoNvfp4) : ANEMOI_DIM(T, QB, SPLIT, false, kNoNvfp4))   \
                : ANEMOI_DIM(T, QB, SPLIT, false, kFp16Alone))
#define ANEMOI_DISPATCH(T) \
  (s.query_block == 128 ? ANEMOI_CELLS(T, 128, true) : split ? ANEMOI_CELLS(T, 64, true) : ANEMOI_CELLS(T, 64, false))
  return s.input_is_bf16 ? ANEMOI_DISPATCH(__nv_bfloat16) : ANEMOI_DISPATCH(__half);
#undef ANEMOI_DISPATCH
#undef ANEMOI_CELLS
#undef ANEMOI_DIM
}
