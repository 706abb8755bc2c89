// Draft probability: pooled-QK logits (fp32 accumulate, rounded to fp16), row
// softmax in fp32, optional mean/max blend, fp16 result [H][R][R].
//
// Reference: csrc/attention/cuda/sm120/h3_draft_probability.cu:131-222 (softmax
// and blend) and :427-465 (cuBLAS pooled GEMM, fp16 logits).  The reference
// leaves the accumulation order to cuBLAS and uses a fast-math expf, so its own
// map is only reproducible to ~5e-4; the routing that follows ranks these values
// globally, so here every operation is fixed and individually rounded:
//   dot     acc = fma(q[c], k[c], acc) for c = 0..D-1 (products of fp16 values are
//           exact in fp32, so this equals a separately rounded add)
//   logit   f16_rn(acc * f32(1/sqrt(D)))
//   exp     y = max(t*log2e, -125); n = rint(y); f = y - n;
//           p = Horner degree 7 of 2^f with rounded multiplies and adds; e = p * 2^n
//   sum     lane l adds columns l, l+32, ... ascending; lanes are folded with an
//           xor butterfly 16, 8, 4, 2, 1
//   prob    f16_rn(e * (1/sum)), IEEE reciprocal; blend f16_rn((1-w)*pm + w*px)
// A CPU restatement with the same sequence reproduces the map bit for bit.
//
// Bound by the FMA pipe (56 heads x 672 blocks x 128 channels: 90 us of FMAs) and, as it is read here, as much again
// of shared memory and conversions; the softmax takes some 60 us.  So a key tile holds all channels (half the barriers
// of 64 at a time), as fp16 (half the bytes of floats), both maps go in one walk, and the exponentials are packed, without
// conversion instructions, and kept between the sum and the quotients.  us, 64 channels of floats and scalar
// exponentials / so: that map 312 / 260, 56 x 592 266 / 213, 7 x 672 51 / 38.5, 4 x 672 x 64 31.4 / 24.1, 7 x 273 with two maps
// 35.0 / 26.4, 8 x 33 with two 11.3 / 7.8.
#include <cuda_fp16.h>

#include "canonical.cuh"
#include "layer.cuh"
#include "packed.cuh"
#include "records.cuh"

namespace {

using canonical::exp_canonical;
using sm100::fadd2;
using sm100::ffma2;

constexpr int kWarps = 8;
constexpr int kChunk = 128;                   // key blocks per pass: 4 per lane
constexpr int kSlab = 64;                     // channels of the key tile held at a time
constexpr int kMaxBlocks = 4096;              // rows per head the shared-memory buffers allow

// Columns l, l + 32, ... of a row, lane l's share of the canonical sum, follow one another in shared memory as `fours`
// 8-byte words.  Where four or more divide their number, as many lanes of sixteen would meet in a bank: there word k
// lies at k ^ column_swizzle (no conflicts).  Elsewhere two meet at most, and the exclusive-or costs more (56 heads x 592
// blocks x 128 213 us plain, 220 with it).  Padding instead of it takes the shared memory of four rows per warp: 56 x 448
// with two maps 273 us, 327 padded, 56 x 1,024 618 and 791.
__host__ __device__ constexpr int column_fours(int R) { return (R + 127) / 128; }
template <bool kSwizzle>
__device__ __forceinline__ int column_swizzle(int lane, int fours) {
  if (!kSwizzle) return 0;
  const int n = min(fours & -fours, 16);
  return (lane >> (__clz(n) - 27)) & (n - 1);
}

// fp16 logits of kWarps * RPW query blocks against every key block of the head, for one pair of pools or two.
// Each warp owns RPW (1, 2 or 4) rows, each lane four key columns of the 128-column pass.  The key tile holds
// all channels, as it comes (fp16, two channels of a column in a word, so that one 16-byte load
// serves two channels of four columns); query values are floats, read by broadcasts.  Every logit is still
// the plain channel-ordered FMA chain (the canonical order).
template <int D, int RPW, int kMaps, bool kSwizzle>
__device__ __forceinline__ void row_logits(const __half* const (&q_pool)[2], const __half* const (&k_pool)[2], int head,
                                           int R, int row0, uint32_t* kc, float* qs, __half* lg, int fours) {
  constexpr int kRows = kWarps * RPW, kThreads = kWarps * 32;
  constexpr int kLoads = kChunk * (D / 8) / kThreads;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float scale = D == 64 ? 0.125f : __int_as_float(0x3db504f3);
  const int chunks = (R + kChunk - 1) / kChunk;
  // the next tile is on its way while this one is multiplied
  uint4 raw[kLoads];
  const auto fetch = [&](int piece) {
    const __half* src = (kMaps == 2 && piece >= chunks ? k_pool[1] : k_pool[0]) + (int64_t)head * R * D;
    const int c0 = (kMaps == 2 && piece >= chunks ? piece - chunks : piece) * kChunk;
#pragma unroll
    for (int i = 0; i < kLoads; ++i) {
      const int idx = threadIdx.x + i * kThreads, col = c0 + idx % kChunk;
      raw[i] = make_uint4(0, 0, 0, 0);
      if (col < R) raw[i] = __ldg(reinterpret_cast<const uint4*>(src + (int64_t)col * D) + idx / kChunk);
    }
  };
  fetch(0);
  const float* qw = qs + warp * D * RPW;
  for (int piece = 0; piece < kMaps * chunks; ++piece) {
    const int map = kMaps == 2 && piece >= chunks, c0 = (piece - map * chunks) * kChunk;
    if (piece > 0) __syncthreads();
    if (c0 == 0) {
      // the rows of a warp interleaved: qs[warp][channel][RPW]
      const __half* pools = (kMaps == 2 && map ? q_pool[1] : q_pool[0]) + (int64_t)head * R * D;
      if ((reinterpret_cast<uintptr_t>(pools) & 15) == 0) {
        for (int idx = threadIdx.x; idx < kRows * (D / 8); idx += kThreads) {
          const int r = idx % kRows, c8 = idx / kRows, row = row0 + r;
          uint4 v = make_uint4(0, 0, 0, 0);
          if (row < R) v = __ldg(reinterpret_cast<const uint4*>(pools + (int64_t)row * D) + c8);
          const __half* h = reinterpret_cast<const __half*>(&v);
#pragma unroll
          for (int j = 0; j < 8; ++j) qs[((r / RPW) * D + c8 * 8 + j) * RPW + r % RPW] = __half2float(h[j]);
        }
      } else {  // query pools may start at any half
#pragma unroll 1
        for (int idx = threadIdx.x; idx < kRows * D; idx += kThreads) {
          const int r = idx / D, c = idx % D, row = row0 + r;
          qs[((r / RPW) * D + c) * RPW + r % RPW] = row < R ? __half2float(pools[(int64_t)row * D + c]) : 0.0f;
        }
      }
    }
#pragma unroll
    for (int i = 0; i < kLoads; ++i) {
      const int idx = threadIdx.x + i * kThreads;
      uint32_t* dst = kc + idx / kChunk * 4 * kChunk + idx % kChunk;
      dst[0] = raw[i].x;
      dst[kChunk] = raw[i].y;
      dst[2 * kChunk] = raw[i].z;
      dst[3 * kChunk] = raw[i].w;
    }
    __syncthreads();
    if (piece + 1 < kMaps * chunks) fetch(piece + 1);
    float acc[RPW][4];
#pragma unroll
    for (int r = 0; r < RPW; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[r][j] = 0.0f;
#pragma unroll 4
    for (int c2 = 0; c2 < D / 2; ++c2) {
      const uint4 kv = *reinterpret_cast<const uint4*>(kc + c2 * kChunk + lane * 4);
      float2 k[4];
      k[0] = __half22float2(*reinterpret_cast<const __half2*>(&kv.x));
      k[1] = __half22float2(*reinterpret_cast<const __half2*>(&kv.y));
      k[2] = __half22float2(*reinterpret_cast<const __half2*>(&kv.z));
      k[3] = __half22float2(*reinterpret_cast<const __half2*>(&kv.w));
      float qv[2 * RPW];
      if (RPW == 1) {
        *reinterpret_cast<float2*>(qv) = *reinterpret_cast<const float2*>(qw + c2 * 2);
      } else {
#pragma unroll
        for (int r = 0; r < 2 * RPW; r += 4)
          *reinterpret_cast<float4*>(qv + r) = *reinterpret_cast<const float4*>(qw + c2 * 2 * RPW + r);
      }
#pragma unroll
      for (int r = 0; r < RPW; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[r][j] = __fmaf_rn(qv[r], k[j].x, acc[r][j]);
#pragma unroll
      for (int r = 0; r < RPW; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[r][j] = __fmaf_rn(qv[RPW + r], k[j].y, acc[r][j]);
    }
    // (columns from R on are written, too, and left out by the reader)
    __half* dst = lg + ((map * kRows + warp * RPW) * 32 + (lane & 7) * 4) * 4 * fours + (lane >> 3);
    if (!kSwizzle) dst += c0 >> 5;
#pragma unroll
    for (int r = 0; r < RPW; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int word = kSwizzle ? (c0 >> 7) ^ column_swizzle<true>((lane & 7) * 4 + j, fours) : 0;
        dst[((r * 32 + j) * fours + word) * 4] = __float2half_rn(__fmul_rn(acc[r][j], scale));
      }
  }
  __syncwarp();
}

// Four values of exp_canonical(x - m), packed arithmetic of the same roundings.  round(y) is a pair of
// additions (|y| <= 125, half to even as rintf), 2^n an addition to the exponent: the product is normal.  The
// conversion instructions of the plain form run at 1/8 of the rate of an addition.
// A product is a * b + zero with zero = -0, a value that the compiler does not know (an argument of the kernel): a
// packed mul, or one with a constant zero, comes back fused with the addition after it, .rn or not.
__device__ __forceinline__ void exp_four(const uint2& raw, float m, float zero, float (&e)[4]) {
  const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&raw.x));
  const float2 hi = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
  const auto both = [](float v) { return make_float2(v, v); };
  const auto bits = [&](int v) { return both(__int_as_float(v)); };
  const auto fmul2 = [&](float2 a, float2 b) { return ffma2(a, b, both(zero)); };
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float2 y = fmul2(fadd2(h ? hi : lo, both(-m)), bits(0x3fb8aa3b));
    y = make_float2(fmaxf(y.x, -125.0f), fmaxf(y.y, -125.0f));
    const float2 t = fadd2(y, both(12582912.0f));
    const float2 f = fadd2(y, ffma2(t, both(-1.0f), both(12582912.0f)));
    float2 p = bits(0x377fe5fe);
    p = fadd2(fmul2(p, f), bits(0x39218489));
    p = fadd2(fmul2(p, f), bits(0x3aaec3ff));
    p = fadd2(fmul2(p, f), bits(0x3c1d955b));
    p = fadd2(fmul2(p, f), bits(0x3d635847));
    p = fadd2(fmul2(p, f), bits(0x3e75fdf0));
    p = fadd2(fmul2(p, f), bits(0x3f317218));
    p = fadd2(fmul2(p, f), both(1.0f));
    e[2 * h] = __int_as_float(__float_as_int(p.x) + (__float_as_int(t.x) << 23));
    e[2 * h + 1] = __int_as_float(__float_as_int(p.y) + (__float_as_int(t.y) << 23));
  }
}

// One row of the map.  Up to kKept * 128 columns its exponentials stay in registers between the sum and
// the quotients; a longer row forms them twice.
constexpr int kKept = 6;
struct RowMap {
  float m, inv;
  float e[kKept][4];
};
template <bool kKeep, bool kSwizzle>
__device__ __forceinline__ void row_map(const __half* lg, int R, int fours, float zero, RowMap& row) {
  const int lane = threadIdx.x & 31;
  const int swizzle = column_swizzle<kSwizzle>(lane, fours);
  const auto load = [&](int k) { return reinterpret_cast<const uint2*>(lg)[k ^ swizzle]; };
  const int mine = (R - lane + 31) >> 5;  // the lane's values before the padding
  float m = -INFINITY;
  const auto fold = [&](int k) {
    const uint2 raw = load(k);
    const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&raw.x));
    const float2 hi = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
    const float v[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (4 * k + j < mine) m = fmaxf(m, v[j]);
  };
  float s = 0.0f;
  const auto add = [&](int k, float (&e)[4]) {
    exp_four(load(k), m, zero, e);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (4 * k + j < mine) s = __fadd_rn(s, e[j]);
  };
  if (kKeep) {
#pragma unroll
    for (int k = 0; k < kKept; ++k)
      if (k < fours) fold(k);
  } else {
    for (int k = 0; k < fours; ++k) fold(k);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
  if (kKeep) {
#pragma unroll
    for (int k = 0; k < kKept; ++k)
      if (k < fours) add(k, row.e[k]);
  } else {
    float e[4];
    for (int k = 0; k < fours; ++k) add(k, e);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, off));
  row.m = m;
  row.inv = __fdiv_rn(1.0f, s);
}
template <bool kBlend, bool kKeep, bool kSwizzle>
__device__ __forceinline__ void write_row(const __half* lg, const __half* lgx, float w, int R, float zero,
                                          __half* out) {
  const int lane = threadIdx.x & 31, fours = column_fours(R);
  const float wm = __fsub_rn(1.0f, w);
  lg += lane * 4 * fours;
  lgx += lane * 4 * fours;
  RowMap mean, most;
  row_map<kKeep, kSwizzle>(lg, R, fours, zero, mean);
  if (kBlend) row_map<kKeep, kSwizzle>(lgx, R, fours, zero, most);
  const auto put = [&](int k, const float (&e)[4], const float (&ex)[4]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int col = lane + 32 * (4 * k + j);
      const float p = __fmul_rn(e[j], mean.inv);
      if (col < R)
        out[col] =
            __float2half_rn(kBlend ? __fadd_rn(__fmul_rn(wm, p), __fmul_rn(w, __fmul_rn(ex[j], most.inv))) : p);
    }
  };
  if (kKeep) {
#pragma unroll
    for (int k = 0; k < kKept; ++k)
      if (k < fours) put(k, mean.e[k], kBlend ? most.e[k] : mean.e[k]);
  } else {
    const int swizzle = column_swizzle<kSwizzle>(lane, fours);
    for (int k = 0; k < fours; ++k) {
      float e[4], ex[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      exp_four(reinterpret_cast<const uint2*>(lg)[k ^ swizzle], mean.m, zero, e);
      if (kBlend) exp_four(reinterpret_cast<const uint2*>(lgx)[k ^ swizzle], most.m, zero, ex);
      put(k, e, ex);
    }
  }
}

// ---- diag-Jensen variant (an experimental routing proxy of the reference,
// anemoi/layers/attention/mpa/routing.py:87-103) -------------------------------------------
//   logit = q.k/sqrt(D) + 0.5 * max((q2.k2 - (q*q).(k*k)) / D, 0)   in fp32, not rounded to fp16
// q2, k2: per-channel second moments of the blocks.  Three dot products per pair, each the same
// channel-ordered FMA chain as above (two rows per warp, four key columns per lane); the third
// one's inputs are the fp32 squares of the pools.  kStep 0: base = round(acc * scale) stored;
// 1: v = acc stored in the second buffer; 2: logit = fma(0.5, max((v - acc) / D, 0), base).
template <int D, int kStep>
__device__ __forceinline__ void jensen_pass(const __half* q_src, const __half* k_src, int head, int R,
                                            int row0, float* kc, float* qs, float* lg, float* var,
                                            int stride) {
  constexpr int kRows = kWarps * 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float scale = D == 64 ? 0.125f : __int_as_float(0x3db504f3);
  __syncthreads();
  for (int idx = threadIdx.x; idx < kRows * D; idx += kWarps * 32) {
    const int r = idx / D, c = idx % D;
    const int row = row0 + r;
    float x = row < R ? __half2float(q_src[((int64_t)head * R + row) * D + c]) : 0.0f;
    if (kStep == 2) x = __fmul_rn(x, x);
    qs[((r >> 1) * D + c) * 2 + (r & 1)] = x;
  }
  for (int c0 = 0; c0 < R; c0 += kChunk) {
    float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    const float* qw = qs + warp * D * 2;
    for (int s0 = 0; s0 < D; s0 += kSlab) {
      __syncthreads();
      for (int idx = threadIdx.x; idx < kChunk * (kSlab / 8); idx += kWarps * 32) {
        const int col = idx % kChunk, c8 = idx / kChunk;
        uint4 raw = make_uint4(0, 0, 0, 0);
        if (c0 + col < R)
          raw = __ldg(reinterpret_cast<const uint4*>(k_src + ((int64_t)head * R + c0 + col) * D + s0) + c8);
        const __half* h = reinterpret_cast<const __half*>(&raw);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float x = __half2float(h[i]);
          if (kStep == 2) x = __fmul_rn(x, x);
          kc[(c8 * 8 + i) * kChunk + col] = x;
        }
      }
      __syncthreads();
      // (sixteen channels' loads ahead: with four the kernel of D = 64 has 32 registers, 24 heads x 672 blocks 453 us, so 388)
#pragma unroll 16
      for (int c = 0; c < kSlab; ++c) {
        const float2 qv = *reinterpret_cast<const float2*>(qw + (s0 + c) * 2);
        const float4 kv = *reinterpret_cast<const float4*>(kc + c * kChunk + lane * 4);
        acc[0][0] = __fmaf_rn(qv.x, kv.x, acc[0][0]);
        acc[0][1] = __fmaf_rn(qv.x, kv.y, acc[0][1]);
        acc[0][2] = __fmaf_rn(qv.x, kv.z, acc[0][2]);
        acc[0][3] = __fmaf_rn(qv.x, kv.w, acc[0][3]);
        acc[1][0] = __fmaf_rn(qv.y, kv.x, acc[1][0]);
        acc[1][1] = __fmaf_rn(qv.y, kv.y, acc[1][1]);
        acc[1][2] = __fmaf_rn(qv.y, kv.z, acc[1][2]);
        acc[1][3] = __fmaf_rn(qv.y, kv.w, acc[1][3]);
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int col = c0 + lane * 4 + j;
        if (col >= R) continue;
        const int at = (warp * 2 + r) * stride + col;
        if (kStep == 0) {
          lg[at] = __fmul_rn(acc[r][j], scale);
        } else if (kStep == 1) {
          var[at] = acc[r][j];
        } else {
          const float t = fmaxf(__fmul_rn(__fsub_rn(var[at], acc[r][j]), 1.0f / D), 0.0f);
          lg[at] = __fmaf_rn(0.5f, t, lg[at]);
        }
      }
  }
  __syncwarp();
}

template <int D>
__global__ void __launch_bounds__(kWarps * 32) draft_jensen_kernel(const __half* q_pool,
                                                                   const __half* k_pool,
                                                                   const __half* q_second,
                                                                   const __half* k_second, int R,
                                                                   __half* prob) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  constexpr int kRows = kWarps * 2;
  const int stride = (R + 3) & ~3;
  float* kc = reinterpret_cast<float*>(smem_raw);  // [kSlab][kChunk]
  float* qs = kc + kSlab * kChunk;                 // [kWarps][D][2]
  float* lg = qs + kRows * D;                      // [kRows][stride] fp32 logits
  float* var = lg + kRows * stride;                // [kRows][stride]
  const int head = blockIdx.y, row0 = blockIdx.x * kRows;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  jensen_pass<D, 0>(q_pool, k_pool, head, R, row0, kc, qs, lg, var, stride);
  jensen_pass<D, 1>(q_second, k_second, head, R, row0, kc, qs, lg, var, stride);
  jensen_pass<D, 2>(q_pool, k_pool, head, R, row0, kc, qs, lg, var, stride);
  for (int r = 0; r < 2; ++r) {
    const int row = row0 + warp * 2 + r;
    if (row >= R) break;
    const float* mine = lg + (warp * 2 + r) * stride;
    float m = -INFINITY;
    for (int j = lane; j < R; j += 32) m = fmaxf(m, mine[j]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
    float sum = 0.0f;
    for (int j = lane; j < R; j += 32) sum = __fadd_rn(sum, exp_canonical(__fsub_rn(mine[j], m)));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, off));
    const float inv = __fdiv_rn(1.0f, sum);
    __half* out = prob + ((int64_t)head * R + row) * R;
    for (int j = lane; j < R; j += 32)
      out[j] = __float2half_rn(__fmul_rn(exp_canonical(__fsub_rn(mine[j], m)), inv));
  }
}

template <int D, bool kBlend, int RPW, bool kSwizzle>
__global__ void __launch_bounds__(kWarps * 32, 2)
    draft_kernel(const __half* q_pool, const __half* k_pool, const __half* q_max, const __half* k_max, float w, int R,
                 float zero, __half* prob) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  constexpr int kRows = kWarps * RPW;
  const int fours = column_fours(R);
  uint32_t* kc = reinterpret_cast<uint32_t*>(smem_raw);         // [D / 2][kChunk], two channels a word
  float* qs = reinterpret_cast<float*>(kc + D / 2 * kChunk);    // [kWarps][D][RPW]
  __half* lg = reinterpret_cast<__half*>(qs + kRows * D);       // [kRows][32][4 * fours], twice when blending
  const int head = blockIdx.y, row0 = blockIdx.x * kRows;
  const int warp = threadIdx.x >> 5;

  layer::grid_dependency_wait();
  layer::grid_dependency_trigger();
  const __half* const q[2] = {q_pool, q_max};
  const __half* const k[2] = {k_pool, k_max};
  row_logits<D, RPW, kBlend ? 2 : 1, kSwizzle>(q, k, head, R, row0, kc, qs, lg, fours);
  for (int r = warp * RPW; r < warp * RPW + RPW; ++r) {
    if (row0 + r >= R) break;
    __half* out = prob + ((int64_t)head * R + row0 + r) * R;
    const __half *mean = lg + r * 128 * fours, *most = mean + kRows * 128 * fours;  // most: blend only
    if (R <= kKept * 128)
      write_row<kBlend, true, kSwizzle>(mean, most, w, R, zero, out);
    else
      write_row<kBlend, false, kSwizzle>(mean, most, w, R, zero, out);
  }
}

// Shared memory of one CTA: key tile, query rows, the logits of its rows (twice when blending).
template <int D, bool kBlend, int RPW>
size_t smem_bytes(int R) {
  constexpr size_t kRows = kWarps * RPW;
  return (size_t)D / 2 * kChunk * 4 + kRows * D * 4 + kRows * 128 * column_fours(R) * 2 * (kBlend ? 2 : 1);
}

template <int D, bool kBlend, int RPW>
int launch_rows(const __half* qp, const __half* kp, const __half* qx, const __half* kx, float w, int R,
                int H, __half* prob, cudaStream_t st) {
  const size_t smem = smem_bytes<D, kBlend, RPW>(R);
  auto kernel = column_fours(R) % 4 == 0 ? draft_kernel<D, kBlend, RPW, true> : draft_kernel<D, kBlend, RPW, false>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
      cudaSuccess)
    return ANEMOI_SM100_ELAUNCH;
  constexpr int kRows = kWarps * RPW;
  dim3 grid((R + kRows - 1) / kRows, H);
  return layer::launch(kernel, grid, dim3(kWarps * 32), smem, st, qp, kp, qx, kx, w, R, -0.0f, prob) == cudaSuccess
             ? ANEMOI_SM100_OK
             : ANEMOI_SM100_ELAUNCH;
}

// Rows per warp.  Four while two CTAs still fit an SM's shared memory, else two: a key tile read serves
// more rows.  But while a grid of fewer rows has no more CTAs than there are SMs, every CTA has one to
// itself and the shorter one wins.  One / two / four rows, us: 8 heads x 33 blocks, two maps (40 CTAs of one row)
// 7.7 / 10.6 / 16.4, 5 x 247 (80 of two) 8.5 / 7.0 / 10.5, 7 x 273, two maps (126 of two) 35.8 / 26.9 / 39.1, 4 x 672
// (168 of two) 29.8 / 27.0 / 24.2, 16 x 225 (240) 25.8 / 18.6 / 15.7, 56 x 672 541 / 354 / 260; two / four, two maps, 56 x 512
// (the last size of four) 396 / 324, 12 x 512 96.5 / 98.4.
constexpr int kSms = 148;
template <int D, bool kBlend>
int launch(const __half* qp, const __half* kp, const __half* qx, const __half* kx, float w, int R,
           int H, __half* prob, cudaStream_t st) {
  auto ctas = [&](int rpw) { return (int64_t)((R + kWarps * rpw - 1) / (kWarps * rpw)) * H; };
  if (ctas(1) <= kSms) return launch_rows<D, kBlend, 1>(qp, kp, qx, kx, w, R, H, prob, st);
  if (ctas(2) <= kSms || smem_bytes<D, kBlend, 4>(R) > 113 * 1024)
    return launch_rows<D, kBlend, 2>(qp, kp, qx, kx, w, R, H, prob, st);
  return launch_rows<D, kBlend, 4>(qp, kp, qx, kx, w, R, H, prob, st);
}

// Key pools are read 16 bytes at a time, query pools and the map by halves where they are not aligned.
bool aligned(const void* ptr, int bytes) { return reinterpret_cast<uintptr_t>(ptr) % bytes == 0; }

}  // namespace

extern "C" int anemoi_sm100_draft_probability(const anemoi_sm100_shape* shape, const void* q_pool,
                                              const void* k_pool, const void* q_max_pool,
                                              const void* k_max_pool, float maxpool_weight,
                                              void* probability, void* stream) {
  if (rec::validate_shape(shape) != ANEMOI_SM100_OK || !q_pool || !k_pool || !probability)
    return ANEMOI_SM100_EINVAL;
  if (!(maxpool_weight >= 0.0f && maxpool_weight <= 1.0f)) return ANEMOI_SM100_EINVAL;
  if (maxpool_weight != 0.0f && (!q_max_pool || !k_max_pool)) return ANEMOI_SM100_EINVAL;
  const int R = shape->video_blocks, H = shape->heads, D = shape->head_dim;
  if (R > kMaxBlocks || (maxpool_weight != 0.0f && maxpool_weight != 1.0f && R > 2400))
    return ANEMOI_SM100_ELIMIT;  // shared-memory row buffers
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __half* qp = static_cast<const __half*>(q_pool);
  const __half* kp = static_cast<const __half*>(k_pool);
  const __half* qx = static_cast<const __half*>(q_max_pool);
  const __half* kx = static_cast<const __half*>(k_max_pool);
  __half* prob = static_cast<__half*>(probability);
  if (maxpool_weight == 1.0f) {  // max pools only
    qp = qx;
    kp = kx;
    maxpool_weight = 0.0f;
  }
  const bool blend = maxpool_weight != 0.0f;
  if (!aligned(kp, 16) || !aligned(qp, 2) || !aligned(prob, 2) || (blend && (!aligned(kx, 16) || !aligned(qx, 2))))
    return ANEMOI_SM100_EINVAL;
  if (D == 64)
    return blend ? launch<64, true>(qp, kp, qx, kx, maxpool_weight, R, H, prob, st)
                 : launch<64, false>(qp, kp, qx, kx, maxpool_weight, R, H, prob, st);
  return blend ? launch<128, true>(qp, kp, qx, kx, maxpool_weight, R, H, prob, st)
               : launch<128, false>(qp, kp, qx, kx, maxpool_weight, R, H, prob, st);
}

extern "C" int anemoi_sm100_draft_probability_jensen(const anemoi_sm100_shape* shape,
                                                     const void* q_pool, const void* k_pool,
                                                     const void* q_second, const void* k_second,
                                                     void* probability, void* stream) {
  if (rec::validate_shape(shape) != ANEMOI_SM100_OK || !q_pool || !k_pool || !q_second || !k_second ||
      !probability)
    return ANEMOI_SM100_EINVAL;
  if (!aligned(k_pool, 16) || !aligned(k_second, 16) || !aligned(q_pool, 2) || !aligned(q_second, 2) ||
      !aligned(probability, 2))
    return ANEMOI_SM100_EINVAL;
  const int R = shape->video_blocks, H = shape->heads, D = shape->head_dim;
  const size_t smem = (size_t)kSlab * kChunk * 4 + (size_t)kWarps * 2 * D * 4 +
                      (size_t)kWarps * 2 * ((R + 3) & ~3) * 4 * 2;
  if (smem > 227 * 1024) return ANEMOI_SM100_ELIMIT;  // two fp32 row buffers: R up to about 1,400
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  dim3 grid((R + kWarps * 2 - 1) / (kWarps * 2), H);
  const __half* qp = static_cast<const __half*>(q_pool);
  const __half* kp = static_cast<const __half*>(k_pool);
  const __half* q2 = static_cast<const __half*>(q_second);
  const __half* k2 = static_cast<const __half*>(k_second);
  __half* prob = static_cast<__half*>(probability);
  if (D == 64) {
    if (cudaFuncSetAttribute(draft_jensen_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem) != cudaSuccess)
      return ANEMOI_SM100_ELAUNCH;
    draft_jensen_kernel<64><<<grid, kWarps * 32, smem, st>>>(qp, kp, q2, k2, R, prob);
  } else {
    if (cudaFuncSetAttribute(draft_jensen_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem) != cudaSuccess)
      return ANEMOI_SM100_ELAUNCH;
    draft_jensen_kernel<128><<<grid, kWarps * 32, smem, st>>>(qp, kp, q2, k2, R, prob);
  }
  return cudaGetLastError() == cudaSuccess ? ANEMOI_SM100_OK : ANEMOI_SM100_ELAUNCH;
}
