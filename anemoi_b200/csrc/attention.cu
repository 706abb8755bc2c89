// Block-sparse mixed-precision flash attention for sm_100a.
//
// One CTA owns one query tile (QB rows of one head, padded to the 128-row MMA
// shape) and walks that tile's ragged list of 64-key stages in the order
// NVFP4 -> INT8 -> FP16 with one online-softmax state.
//
// Roles (512 threads = four warpgroups, two CTAs per SM; registers move between them with setmaxnreg):
//   warps 0-3, 4-7  softmax of the even and of the odd stages: warp w owns TMEM lanes 32*(w%4)..
//                   (query rows), one thread per row with the row's 64 scores in registers
//   warps 8-11      rescale of O: when a stage moved some row's maximum, or at a phase change
//                   (where O also moves between the phases' value domains); they also move the
//                   FP16 phase's Q into tensor memory
//   warp 12         loader: one lane issues 1-D bulk copies (TMA engine) of the Q record of each
//                   phase and of one K|V record per stage into a ring of shared-memory slots
//   warp 13         S[128x64]  = Q K^T   kind::mxf4nvf4 / kind::i8 / kind::f16
//   warp 14         O[128xD]  += P V     kind::mxf4nvf4 / kind::f8f6f4 / kind::f16
//   warp 15         idle
// TMEM columns: S0 [0,64), O [64,64+D), from 192 on the NVFP4 scale factors or the INT8 and FP16 phases'
// Q; D = 64 has a second score buffer S1 behind O.
//
// Why this split.  A stage needs 8,192 exponentials = 512 cycles of the special-function unit and
// 130-580 cycles of the tensor core per SM, but one warp's chain through a stage (wait for S, load
// it, maximum, exponentials, conversion, store, fence, arrive) is over 2,000 cycles long, and with
// one softmax warp per row quadrant and CTA (8 per SM, all that tensor memory and two query tiles
// allow) latency set the pace: 1,250-1,400 cycles per stage and SM.  So two warpgroups share a tile
// and run alternate stages.  P is quantised against the running maximum of a strictly sequential
// walk, so the maximum is handed from stage to stage through shared memory as soon as it is known,
// and the exponentials of two stages overlap.  O's rescale, which waits for the previous PV, is
// off the softmax warps' path; QK and PV are issued by different warps so that QK of a stage waits
// for nothing but its key tile and its score buffer.
// Measured per stage and SM at D = 128, cycles, one softmax warpgroup / two: NVFP4 1,282 / 791,
// INT8 1,394 / 835, FP16 1,332 / 1,050, the mixed layer of S = 85,184 (8 heads) 1,250 / 900.  Bound
// by issue slots and the special-function unit (each 66 % busy: 520 of INT8's 790 cycles at the clock it
// ran at) and the waits around them - moving exponentials to the FMA pipe only adds issue slots -; FP16 by
// shared memory, which moves 96 KB = 768 cycles' worth per stage, and, in long runs, by the power limit.
//
// P is stored over the stage's K tile, which the tensor core has finished reading when the scores
// arrive; that leaves the ring all of the shared memory that Q does not take.
//
// Numerics follow the reference's phases
// (csrc/attention/cuda/sm120/q64_attention_phase_composer.inl:1-146, 506-932,
// 934-1331; primitives/qattn/attn_utils.cuh:363-389, 470-625):
//   base-2 online softmax, sigma = log2(e)/sqrt(D), m0 = -5e6, keys >= valid_k masked,
//   denominator accumulated from the unquantised P,
//   NVFP4: score scale sigma*q_gs*k_gs, P -> e2m1(6P) with a constant 448 block scale,
//          O_true = O * v_gs/(6*448)
//   INT8 : exact s32 scores, scale sigma*q_scale*k_scale[stage], P -> e4m3(P*2^8.807),
//          O_true[c] = O[c] * v_scale[c] * 2^-8.807
//   FP16 : P -> f16
// Accumulation is fp32 in TMEM (the reference accumulates a stage in fp16 for the
// INT8 and FP16 cells).
#include <cuda.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "bounded_wait.cuh"
#include "layer.cuh"
#include "packed.cuh"
#include "records.cuh"
#include "sm100_primitives.cuh"

namespace {

using namespace sm100;
using layer::TokenRows;

// Four warpgroups: softmax of the even stages, softmax of the odd stages, rescale of O, and
// loader / QK / PV (one warp each, the fourth idle).
constexpr int kThreads = 512;
constexpr int kCorrWarp = 8;
constexpr int kLoaderWarp = 12;
constexpr int kQkWarp = 13;
constexpr int kPvWarp = 14;
enum WaitRole : int { kSoftmaxRole = 0, kRescaleRole = 1, kMmaRole = 2 };
constexpr int kTmemCols = 256;
constexpr int kColS = 0;
constexpr int kColO = 64;
constexpr int kColQ = 192;     // INT8: D / 4 columns, FP16: D / 2
constexpr int kColSfaQ = 192;  // 2 k-steps x 4 columns
constexpr int kColSfbK = 200;  // 2 k-steps x 4 columns
constexpr int kColSfaP = 208;
constexpr int kColSfbV = 212;
constexpr int kRing = 8;       // entries of the per-stage rings, and the most key/value slots
constexpr int kSplitKeys = 4, kSplitValues = 2;  // key and value buffers of phases that keep them apart
constexpr int kMostParts = 8;    // CTAs that share the stages of a tile of dense rows: a portable cluster
constexpr float kFp8Offset = 8.807f;
constexpr float kLowest = -3.0e38f;  // maximum before the first stage of dense rows
constexpr float kNoPart = -1.0f;     // denominator of a part that its CTA did not walk
constexpr uint64_t kDrainNs = 100000000;  // limit of the waits for copies and MMAs in flight after a give-up

// log2(e) / sqrt(D)
__host__ __device__ constexpr float sigma(int d) { return (d == 64 ? 0.125f : 0.08838834764831845f) * 1.4426950408889634f; }

enum Cell : int { kNv = 0, kI8 = 1, kF16 = 2 };
// Which cells a kernel is built for: one, all, or two.
enum Cells : int { kAny = 3, kNvI8 = 4, kI8F16 = 5, kNvF16 = 6 };
__host__ __device__ constexpr bool mixed(int cells) { return cells >= kAny; }
__host__ __device__ constexpr bool has_cell(int cells, int cell) {
  return cells == cell || cells == kAny || (cells == kNvI8 && cell != kF16) || (cells == kI8F16 && cell != kNv) ||
         (cells == kNvF16 && cell != kI8);
}
// Whether the stage is of `which`, in a kernel built for `CELLS` (code of cells that it is not built for drops out).
template <int CELLS, int WHICH>
__device__ __forceinline__ bool is(int cell) {
  if constexpr (!has_cell(CELLS, WHICH)) return false;
  else if constexpr (!mixed(CELLS)) return true;
  else return cell == WHICH;
}

// What the roles keep in registers, kernel by kernel.  A loop that lacks registers is the better for a parity that follows
// from the stage's number, or for a pointer formed anew; one that has them loses by it.  Same results bit for bit.  us at
// 16 heads x 14,040, 9 x 6,528 and 30 x 8,415 tokens, the GPU kept busy for 40 ms per time:
// - FP16 D = 128 Q64, parity of the scores from the number 540 / 117 / 431, kept 514 / 114 / 404 (Q128 475 / 92 / 378 and 467 /
//   92 / 378); mixed kernels the other way (NVFP4 + INT8 D = 128 Q128 kept 454 / 119 / 403, from the number 445 / 115 / 389),
//   and dense rows (NVFP4 + FP16 40 x 8,056, 256 prefix rows 597 and 594).
__host__ __device__ constexpr bool keeps_s_parity(int d, int cells, bool raw) { return d == 128 && cells == kF16 && !raw; }
// - three cells D = 128 Q128, parities of the QK warp from the number 552 / 129 / 454, kept 548 / 129 / 451; others 0 to 1 %
//   slower if kept.
__host__ __device__ constexpr bool keeps_free_parity(int d, int cells, bool q64) { return d == 128 && cells == kAny && !q64; }
// - pointer kept / anew: INT8 D = 128 Q128 393 / 95 / 330 and 394 / 94 / 334, D = 64 Q64 378 / 98 / 307 and 367 / 98 / 300; FP16
//   D = 64 Q64 364 / 94 / 294 and 360 / 92 / 292; NVFP4 + INT8 D = 128 Q128 445 / 115 / 389 and 442 / 113 / 388, D = 64 Q128 (with
//   88 registers; with 96 it loses 1 %) 380 / 92 / 316 and 372 / 91 / 310; INT8 + FP16 D = 64 Q64 455 / 117 / 430 and 449 /
//   115 / 425; three cells D = 128 Q64 665 / 158 / 621 and 661 / 158 / 615, Q128 552 / 129 / 454 and 561 / 130 / 465.  INT8
//   D = 64 Q128 goes both ways: 338 / 79 / 272 and 340 / 77 / 274, 14 x 32,760 1,292 / 1,303, 8 x 15,400 255 / 240, 7 x 7,200
//   67.5 / 68.6.  The others that form it anew, at the same sizes: D = 64 Q64 NVFP4 + INT8 494 / 116 / 420 and 491 / 116 / 418,
//   NVFP4 + FP16 503 / 114 / 425 and 502 / 114 / 425, three cells 546 / 129 / 467 and 542 / 128 / 465; D = 64 Q128 FP16 315 / 66 /
//   269 and 317 / 66 / 273 (6 x 3,120 25.2 / 25.1, 1 x 25,600 115.1 / 114.5), INT8 + FP16 375 / 86 / 342 and 371 / 85 / 337,
//   NVFP4 + FP16 336 / 76 / 309 and 334 / 76 / 308; D = 128 Q128 INT8 + FP16 493 / 108 / 447 and 493 / 108 / 448.  Over 110
//   calls with a prefix of INT8 queries 1 % from it, over 130 without a prefix nothing beyond the runs' spread.
__host__ __device__ constexpr bool pointer_anew(int d, int cells, bool q64) {
  if (d == 64) return q64 ? cells != kNv : cells != kNv && cells != kI8 && cells != kAny;
  return q64 ? cells == kAny : cells == kNvI8 || cells == kI8F16;
}

// Registers per thread: 128 * (2 * softmax + rescale + other) == 512 * 64 (two CTAs per SM).  With 96 a
// softmax thread spills nothing, but rescales then go 16 columns at a time.  That is the better
// trade at D = 64 (where O is half as wide: the mixed Q64 kernel 834 -> 778 cycles per stage, FP16
// 930 -> 846) and for NVFP4 (821 -> 796); at D = 128 FP16 and mixed lose (1,005 -> 1,071, 863 -> 899).
// NVFP4 + INT8 D = 64 Q128, with the pointer formed anew, goes with 88: us, 96 / 88, 16 heads x 14,040 tokens 379 / 372,
// 30 x 8,415 318 / 310, 48 x 2,442 102 / 97, 14 x 32,760 1,373 / 1,362; with 200 prefix rows 426 / 419, 369 / 361, 137 / 131,
// 1,480 / 1,468 and, where the prefix tiles' walk is what a call takes, 2 x 11,380 163.2 / 163.6.  INT8 + FP16 and three cells
// gain up to 7 % there too, but lose up to 3 % where prefix tiles are few and long.
constexpr int kOtherRegs = 32;
template <int D, int CELLS, bool kQ64>
struct Regs {
  static constexpr bool kWide = D == 64 ? kQ64 || CELLS != kNvI8 : CELLS == kNv;
  static constexpr int kSoftmax = kWide ? 96 : 88, kRescale = kWide ? 32 : 48;
  static constexpr int kRescaleColumns = kWide ? 16 : 32;
};

// Kernels for dense rows of the caller's own tensors (prefix queries kept out of the cells), and their type.
enum Raw : int { kNone = 0, kRawF16 = 1, kRawBf16 = 2 };

constexpr int kColS1 = 128;    // D = 64: second score buffer

struct AttnParams {
  anemoi_sm100_shape s;
  anemoi_sm100_operands o;
  const int32_t* row_offset;
  const int32_t* row_counts;
  const int32_t* stage_ids;
  int64_t capacity;
  const int32_t* valid_k;
  // Q64 pairs: query blocks 2t and 2t+1 of a head share one CTA (rows 0-63 and 64-127 of the
  // 128-row MMA shape) and walk the union of their lists; bits 30 / 31 of a list entry say which
  // of the two blocks the stage belongs to.  Null: one query block per CTA.
  const int32_t* pair_counts;  // [H][ceil(R/2)][4]
  const int32_t* pair_ids;     // [H][capacity], a pair's list starts at row_offset of block 2t
  // Pairs of any two blocks, in launch order: [H][ceil(R/2)][8] first block, second or -1, start of the list in
  // pair_ids, its stages, those of each phase.  Null: the pairs above.
  const int4* pair_table;
  __half* out;       // [H][tiles*QB][D], or null:
  void* tokens;      // [S][H][D] in the caller's type: rows go straight to their tokens
  int tokens_bf16;
  const int32_t* indices;  // raster token of a packed slot
  const int32_t* counts;   // real tokens of a block
  int32_t* status;
  uint64_t wait_ns;  // limit of every mbarrier wait
  int dense_prefix;  // 1: prefix query tiles, INT8 cell over every stage
  int prefix_tiles;  // prefix query tiles of such a launch
  int stages;        // 64-key stages per head
  int q_tiles_int8;  // records per head in q_int8 (R + prefix query tiles)
  int out_rows;      // rows per head in `out`
  int ring_bytes;    // key/value ring; re-partitioned into equal slots at every phase
  int q_region;      // bytes
  int turn;          // a head's lists before this place in the order start shortest first
  int first_place;   // of a launch's tiles
};

// Dense rows (prefix queries kept out of the cells): 128 queries per tile, every row attends to every token, operands
// straight from the caller's tensors by tiled TMA.  Bound, as the FP16 cell, by shared memory (96 KB per stage of
// D = 128) where there are tiles for every SM, which few calls have: a prefix is some tiles per head, each as long as the
// head's keys, so the CTAs of a cluster (the grid's x) share a tile's stages and add up their parts through each other's
// shared memory.  Alone, us, torch's attention (cuDNN for bf16) / one CTA per tile / parts: bf16 D = 128 3 heads x 7,159
// tokens, 517 rows 82 / 83 / 44, 16 x 14,296, 256 rows 158 / 163 / 86, 53 x 13,093, 37 rows 258 / 153 / 71, 1 x 85,000, 30 rows
// 1,271 / 845 / 109; fp16 D = 64 6 x 33,178, 58 rows 564 / 282 / 44.  Where rows and heads fill the GPU the library is ahead
// (56 x 33,272, 512 rows 408 / 603 / 597), and long prefixes of long sequences are left to it.  Whole calls, of which these
// rows are a part beside the others: small ones 113 -> 37-58 us (its host work alone took 90), 48 x 2,474 with 74 rows 136 -> 122,
// 8 x 3,360 with 210 rows 108 -> 44.
struct alignas(64) RawParams : AttnParams {
  CUtensorMap q, k, v;  // [tokens][heads][D] as they lie in memory: 64 channels x 1 head x 64 tokens (Q: 128), swizzled
  int rows, tokens_in, parts;
  int64_t out_token, out_head;  // distances in `tokens`, in elements
};
template <int RAW>
using Params = std::conditional_t<RAW == kNone, AttnParams, RawParams>;

// Entry g % kRing of a ring belongs to stage g, in phase g / kRing of the barrier.  Stage
// g + kRing cannot begin before PV of stage g is complete (it needs a key/value slot and there are
// at most kRing), so no entry is reused while a role still needs it, and no waiter can miss a phase.
struct Shared {
  uint64_t kv_full[kRing];    // key/value record landed
  uint64_t pv_done[kRing];    // PV complete: slot free, O may be touched
  uint64_t p_full[kRing];     // per quadrant: P stored (softmax warp), O in the right scale (rescale warp)
  uint64_t m_full[4][kRing];  // running maxima of the quadrant's rows up to this stage published
  uint64_t v_full[kSplitValues];  // value tile landed (phases with buffers of their own for keys and values)
  uint64_t q_moved;               // INT8, FP16: Q in tensor memory
  uint64_t q_full, q_free;
  uint64_t s_full[2];  // scores ready, per softmax warpgroup (a waiter has to see every phase)
  uint64_t s_free[2];  // scores read, per score buffer
  uint64_t nv_done;    // every PV of the NVFP4 phase complete
  uint64_t all_done;   // every PV of the tile complete
  uint64_t qk_done;    // unwinding only
  WaitContext wc;
  int cnt[3], first_of[3];  // the tile's stages per phase, where each phase starts inside the list
  // per block of the tile: which factors move O into the INT8, FP16 phase's domain (kStays: none), the domain at the end
  int move[2][2], last[2];
  // which tile it is: read by the roles where they need it, or kept in registers from the start (kReread)
  volatile int head, block[2], tile_blocks;
  const int32_t* volatile list;
  uint32_t tmem_base;
  // per stage and query block of the tile: score scale, real keys (negative: not a stage of this block)
  float2 meta[kRing][2];
  // per stage and row: running maximum m(g), denominator d(g - 2)
  float2 rec[kRing][128];
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// Four fp32 -> four e4m3, eight fp32 -> eight e2m1, in element order (one register, no byte shuffles).
__device__ __forceinline__ uint32_t e4m3x4(float a, float b, float c, float d) {
  uint32_t v;
  asm("{\n\t.reg .b16 lo, hi;\n\tcvt.rn.satfinite.e4m3x2.f32 lo, %2, %1;\n\t"
      "cvt.rn.satfinite.e4m3x2.f32 hi, %4, %3;\n\tmov.b32 %0, {lo, hi};\n\t}"
      : "=r"(v)
      : "f"(a), "f"(b), "f"(c), "f"(d));
  return v;
}
__device__ __forceinline__ uint32_t e2m1x8(const float* e) {
  uint32_t v;
  asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\tcvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n\tcvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n\tmov.b32 %0, {b0, b1, b2, b3};\n\t}"
      : "=r"(v)
      : "f"(e[0]), "f"(e[1]), "f"(e[2]), "f"(e[3]), "f"(e[4]), "f"(e[5]), "f"(e[6]), "f"(e[7]));
  return v;
}
__device__ __forceinline__ uint32_t f16x2(float a, float b) {
  uint32_t v;
  asm("cvt.rn.f16x2.f32 %0, %2, %1;" : "=r"(v) : "f"(a), "f"(b));
  return v;
}

// Every thread of the cluster: what was written to shared memory before is visible after, across its CTAs.
__device__ __forceinline__ void cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Shared memory of the cluster's CTA `rank` at the place that is `addr` in this one's.
__device__ __forceinline__ uint32_t peer_smem(uint32_t addr, int rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
  return a;
}
__device__ __forceinline__ float2 peer_float2(uint32_t addr, int rank) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(peer_smem(addr, rank)) : "memory");
  return v;
}
__device__ __forceinline__ float4 peer_float4(uint32_t addr, int rank) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(peer_smem(addr, rank))
               : "memory");
  return v;
}

__device__ __forceinline__ uint32_t bf16x2(float a, float b) {
  uint32_t v;
  asm("cvt.rn.bf16x2.f32 %0, %2, %1;" : "=r"(v) : "f"(a), "f"(b));
  return v;
}
// 64 channels of 64 or 128 tokens of one head, rows of 128 bytes whose 16-byte pieces are swizzled (by TMA).
__device__ __forceinline__ void tensor_g2s(uint8_t* dst, const CUtensorMap* map, int channel, int head, int token,
                                           uint64_t* bar, uint32_t issue) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %6, 0;\n\t"
      "@q cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      "\n\t}" ::"r"(smem_u32(dst)),
      "l"(map), "r"(channel), "r"(head), "r"(token), "r"(smem_u32(bar)), "r"(issue)
      : "memory");
}
// Operand of 128-byte rows swizzled in groups of eight (1,024 bytes); `lbo`: between blocks of 64 channels where these
// are the operand's rows.
__device__ __forceinline__ uint64_t swizzled_desc(uint32_t addr, uint32_t lbo) {
  return smem_desc(addr, lbo, 1024) | (2ull << 61);
}

// Two fp32 -> fp16 (the result's precision) -> bf16, as the assembly of packed rows rounds.
__device__ __forceinline__ uint32_t bf16x2_of_f16x2(uint32_t h) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
  uint32_t v;
  asm("cvt.rn.bf16x2.f32 %0, %2, %1;" : "=r"(v) : "f"(f.x), "f"(f.y));
  return v;
}

__device__ __forceinline__ void tmem_st4(uint32_t taddr, uint32_t v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(v),
               "r"(v), "r"(v), "r"(v)
               : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(r));
  return r != 0;
}
// `issue` == 0 turns the arrival into a no-op (predicated, no branch).
__device__ __forceinline__ void mbar_arrive_if(uint64_t* bar, uint32_t issue) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t@q mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(
          smem_u32(bar)),
      "r"(issue)
      : "memory");
}

// ------------------------------------------------------------------------------------------
// geometry of a key/value slot
// ------------------------------------------------------------------------------------------
// The P tile of a stage (128 rows x 64 keys) takes the place of the stage's K tile, which the
// tensor core has finished reading when the scores arrive; what follows K in the record (V, scale
// blocks) starts behind the larger of the two.
__host__ __device__ constexpr int k_bytes(int d, int cell) { return 32 * d * (cell == kF16 ? 4 : cell == kI8 ? 2 : 1); }
__host__ __device__ constexpr int p_bytes(int cell) { return 4096 * (cell == kF16 ? 4 : cell == kI8 ? 2 : 1); }
__host__ __device__ constexpr int record_bytes(int d, int cell) {
  return cell == kNv ? 64 * d + (d / 64) * 512 + 512 : (cell == kI8 ? 128 * d : 256 * d);
}
__host__ __device__ constexpr int rest_offset(int d, int cell) {
  return k_bytes(d, cell) > p_bytes(cell) ? k_bytes(d, cell) : p_bytes(cell);
}
__host__ __device__ constexpr int slot_bytes(int d, int cell) {
  return (rest_offset(d, cell) + record_bytes(d, cell) - k_bytes(d, cell) + 127) & ~127;
}
// INT8 and FP16: Q is an operand in tensor memory, moved there from its region at the start of the
// phase.  As a shared-memory operand an FP16 stage of D = 128 read 48 KB for QK alone (48 cycles of
// shared-memory bandwidth per instruction of 36) and moved 128 KB = 1,024 cycles in all, which was the
// bound; INT8 gained 2-4 % (16 heads of S = 33,272: 1.59 -> 1.55 ms; Q64, 8 heads of S = 38,247: 1.47 -> 1.41 ms).
// At D = 128 the FP16 Q's 32 KB then serve keys and values, in buffers of their own: four for key tiles, held until
// PV (P replaces them), and two for value tiles, which are not needed before the probabilities are there.
__host__ __device__ constexpr bool split_kv(int d, int cell) { return d == 128 && cell == kF16; }
__host__ __device__ constexpr int stage_bytes(int d, int cell) {  // distance of two slots
  return split_kv(d, cell) ? k_bytes(d, cell) : slot_bytes(d, cell);
}
// The first two key buffers lie in Q's region and are filled last, once Q has moved.
__host__ __device__ constexpr int first_slot(int d, int cell) { return split_kv(d, cell) ? 2 : 0; }
__host__ __device__ constexpr int slot_count(int ring, int d, int cell) {
  const int n = split_kv(d, cell) ? kSplitKeys : ring / slot_bytes(d, cell);
  return n < kRing ? n : kRing;
}
// Score buffer of stage g: D = 128 has a single one, which the softmax warps have read, soon after the
// scores arrived, long before the next stage's are needed.
template <int D>
__device__ __forceinline__ int s_buffer(int g) {
  return D == 128 ? 0 : (g & 1);
}

__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[32]) { tmem_ld32(taddr, r); }
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st(uint32_t taddr, const uint32_t (&r)[32]) { tmem_st32(taddr, r); }
__device__ __forceinline__ void tmem_st(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(
          taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

// O[row][c] *= (colf[c] when given, then) alpha, for all D columns of the thread's row, kCols at a time.  In that
// order: a row whose first stage in a phase comes after its partner's has the two factors at two stages.
template <int D, int kCols>
__device__ __forceinline__ void rescale_o(uint32_t tmem_row, float alpha, const float* colf) {
  const float2 alpha2 = make_float2(alpha, alpha);
#pragma unroll 1
  for (int c0 = 0; c0 < D; c0 += kCols) {
    uint32_t r[kCols];
    tmem_ld(tmem_row + kColO + c0, r);
    tmem_wait_ld();
    if (colf != nullptr) {
#pragma unroll
      for (int j = 0; j < kCols; j += 2) {
        const float2 v = fmul2(make_float2(__uint_as_float(r[j]), __uint_as_float(r[j + 1])),
                               *reinterpret_cast<const float2*>(colf + c0 + j));
        r[j] = __float_as_uint(v.x);
        r[j + 1] = __float_as_uint(v.y);
      }
    }
#pragma unroll
    for (int j = 0; j < kCols; j += 2) {
      const float2 v = fmul2(make_float2(__uint_as_float(r[j]), __uint_as_float(r[j + 1])), alpha2);
      r[j] = __float_as_uint(v.x);
      r[j + 1] = __float_as_uint(v.y);
    }
    tmem_st(tmem_row + kColO + c0, r);
  }
  tmem_wait_st();
}

// ------------------------------------------------------------------------------------------
// softmax side
// ------------------------------------------------------------------------------------------
// Probabilities of the thread's 64 scores, P = 2^(s * scale + bias), rounded to the cell's operand
// format and stored into its row of the K-major P tile 16 bytes at a time (the conversions and
// stores of one piece run under the exponentials of the next); returns their unrounded sum.
template <int CELL, int RAW = kNone>
__device__ __forceinline__ float exp_store(const float (&s)[64], float scale, float bias,
                                           uint8_t* p_row) {
  const float2 scale2 = make_float2(scale, scale);
  const float2 bias2 = make_float2(bias, bias);
  float2 acc0 = make_float2(0.0f, 0.0f), acc1 = make_float2(0.0f, 0.0f);
  constexpr int kPer = CELL == kNv ? 32 : (CELL == kI8 ? 16 : 8);  // keys per 16 bytes
#pragma unroll
  for (int c = 0; c < 64 / kPer; ++c) {
    float e[kPer];
#pragma unroll
    for (int j = 0; j < kPer; j += 4) {
      float2 a0 = make_float2(s[c * kPer + j], s[c * kPer + j + 1]);
      float2 a1 = make_float2(s[c * kPer + j + 2], s[c * kPer + j + 3]);
      a0 = RAW != kNone ? fmul2(fadd2(a0, bias2), scale2) : ffma2(a0, scale2, bias2);
      a1 = RAW != kNone ? fmul2(fadd2(a1, bias2), scale2) : ffma2(a1, scale2, bias2);
      e[j] = ex2(a0.x);
      e[j + 1] = ex2(a0.y);
      e[j + 2] = ex2(a1.x);
      e[j + 3] = ex2(a1.y);
      acc0 = fadd2(acc0, make_float2(e[j], e[j + 1]));
      acc1 = fadd2(acc1, make_float2(e[j + 2], e[j + 3]));
    }
    uint4 v;
    if (RAW == kRawBf16) {
      v = make_uint4(bf16x2(e[0], e[1]), bf16x2(e[2], e[3]), bf16x2(e[4], e[5]), bf16x2(e[6], e[7]));
    } else if (CELL == kF16) {
      v = make_uint4(f16x2(e[0], e[1]), f16x2(e[2], e[3]), f16x2(e[4], e[5]), f16x2(e[6], e[7]));
    } else if (CELL == kI8) {
      v = make_uint4(e4m3x4(e[0], e[1], e[2], e[3]), e4m3x4(e[4 % kPer], e[5 % kPer], e[6 % kPer], e[7 % kPer]),
                     e4m3x4(e[8 % kPer], e[9 % kPer], e[10 % kPer], e[11 % kPer]),
                     e4m3x4(e[12 % kPer], e[13 % kPer], e[14 % kPer], e[15 % kPer]));
    } else {
      v = make_uint4(e2m1x8(e), e2m1x8(e + 8 % kPer), e2m1x8(e + 16 % kPer), e2m1x8(e + 24 % kPer));  // e holds 6 P
    }
    *reinterpret_cast<uint4*>(p_row + c * 128) = v;
  }
  return (acc0.x + acc0.y) + (acc1.x + acc1.y);
}

// The same where the cell is a run-time value: the exponentials take the scores' registers in code that the cells share,
// and only conversion and stores are each cell's own.  That is 64 (128 with three cells) instructions less per copy in
// kernels whose stage code fills the instruction cache, but a piece's conversions no longer run under the next one's
// exponentials.  Separate / shared, us: three cells of D = 64, 7 heads x 11,994 tokens 178 / 166, 8 x 12,240 NVFP4 + INT8 Q64
// 528 / 508.  Not for INT8 + FP16, FP16 having eight stores per stage, and not for three cells of D = 128, which are ahead
// by up to 2.5 % in small calls but lose 1 % in large ones (56 heads x 85,184 tokens 37.4 / 37.8 ms); in halves or with
// two cells at a time the branches cost more than they save (5 x 3,834 three cells 71 / 74).
__host__ __device__ constexpr bool shares(int d, int cells) {
  return cells == kNvI8 || cells == kNvF16 || (d == 64 && cells == kAny);
}
template <int CELLS>
__device__ __forceinline__ float exp_any(float (&s)[64], float scale, float bias, int cell, uint8_t* p_row) {
  const float2 scale2 = make_float2(scale, scale);
  const float2 bias2 = make_float2(bias, bias);
  float2 acc0 = make_float2(0.0f, 0.0f), acc1 = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int j = 0; j < 64; j += 4) {
    const float2 a0 = ffma2(make_float2(s[j], s[j + 1]), scale2, bias2);
    const float2 a1 = ffma2(make_float2(s[j + 2], s[j + 3]), scale2, bias2);
    s[j] = ex2(a0.x);
    s[j + 1] = ex2(a0.y);
    s[j + 2] = ex2(a1.x);
    s[j + 3] = ex2(a1.y);
    acc0 = fadd2(acc0, make_float2(s[j], s[j + 1]));
    acc1 = fadd2(acc1, make_float2(s[j + 2], s[j + 3]));
  }
  if (is<CELLS, kI8>(cell)) {
#pragma unroll
    for (int c = 0; c < 4; ++c)
      *reinterpret_cast<uint4*>(p_row + c * 128) = make_uint4(
          e4m3x4(s[16 * c], s[16 * c + 1], s[16 * c + 2], s[16 * c + 3]),
          e4m3x4(s[16 * c + 4], s[16 * c + 5], s[16 * c + 6], s[16 * c + 7]),
          e4m3x4(s[16 * c + 8], s[16 * c + 9], s[16 * c + 10], s[16 * c + 11]),
          e4m3x4(s[16 * c + 12], s[16 * c + 13], s[16 * c + 14], s[16 * c + 15]));
  } else if (is<CELLS, kNv>(cell)) {
#pragma unroll
    for (int c = 0; c < 2; ++c)
      *reinterpret_cast<uint4*>(p_row + c * 128) = make_uint4(e2m1x8(s + 32 * c), e2m1x8(s + 32 * c + 8),
                                                              e2m1x8(s + 32 * c + 16), e2m1x8(s + 32 * c + 24));
  } else {
#pragma unroll
    for (int c = 0; c < 8; ++c)
      *reinterpret_cast<uint4*>(p_row + c * 128) =
          make_uint4(f16x2(s[8 * c], s[8 * c + 1]), f16x2(s[8 * c + 2], s[8 * c + 3]), f16x2(s[8 * c + 4], s[8 * c + 5]),
                     f16x2(s[8 * c + 6], s[8 * c + 7]));
  }
  return (acc0.x + acc0.y) + (acc1.x + acc1.y);
}

// State of a softmax row.  The two softmax warpgroups alternate stages; the running maximum and
// the denominator travel between them through shared memory.  The denominator is carried two stages
// late, so that a group waits for nothing but the other's maximum: stage g publishes m(g) and d(g - 2),
// and d(g) = d(g - 1) * alpha(g) + sum(g) is formed by the group that ran stage g when it publishes
// stage g + 2 - the order (and rounding) of a strictly sequential walk.
struct SoftmaxWalk {
  uint32_t s_par;     // parity of this group's next scores, where it is kept
  float d;            // denominator before the last two stages of this group's last stage
  float alpha, sum;   // of this group's last stage
};

// One stage.  Padding rows of a 64-row tile, and stages of the other query block of a pair (warp-uniform:
// a warp's rows belong to one block), contribute nothing: P = 0, running maximum and denominator
// untouched.  `kPass`: such a stage has a path of its own, without the scores.  A third of a pair's stages
// are passed over so: Q64 kernels of one cell gain 1-3 % (INT8, 8 heads of S = 38,247: 1.42 -> 1.38 ms); the
// mixed one, whose instruction cache is full, would lose 10 %.
template <int D, int CELLS, bool kPairs, bool kPass, int RAW>
__device__ __forceinline__ void softmax_stage(Shared* b, uint8_t* p_row, uint32_t tmem_row, int row, int g, int cell,
                                              bool live_warp, int my_block, SoftmaxWalk& w) {
  const int at = g & (kRing - 1), before_at = (g - 1) & (kRing - 1);
  uint64_t* m_full = b->m_full[row >> 5];
  const uint32_t lead = (row & 31) == 0;
  const int sb = s_buffer<D>(g);
  constexpr bool kKept = keeps_s_parity(D, CELLS, RAW != kNone);
  wait(&b->wc, &b->s_full[g & 1], kKept ? w.s_par : (g >> 1) & 1, 10);
  if (kKept) w.s_par ^= 1u;
  tc_fence_after_sync();
  const uint32_t tmem_s = tmem_row + (sb ? kColS1 : kColS);
  const auto store_zeros = [&]() {
    const int chunks = p_bytes(cell) / 2048;
#pragma unroll 1
    for (int c = 0; c < chunks; ++c) *reinterpret_cast<uint4*>(p_row + c * 128) = make_uint4(0, 0, 0, 0);
  };
  if (kPass && (!live_warp || __float_as_int(b->meta[at][my_block].y) < 0)) {
    tc_fence_before_sync();
    mbar_arrive_if(&b->s_free[sb], lead);
    wait(&b->wc, &m_full[before_at], ((g - 1) >> 3) & 1, 9);
    const float2 before = b->rec[before_at][row];
    w.d = before.y * w.alpha + w.sum;
    b->rec[at][row] = make_float2(before.x, w.d);
    __syncwarp();
    mbar_arrive_if(&m_full[at], lead);
    w.alpha = 1.0f;
    w.sum = 0.0f;
    if (live_warp) store_zeros();
    fence_proxy_async_smem();
    __syncwarp();
    mbar_arrive_if(&b->p_full[at], lead);
    return;
  }
  float s[64];
  {
    uint32_t r[64];
    tmem_ld32(tmem_s, *reinterpret_cast<uint32_t(*)[32]>(r));
    tmem_ld32(tmem_s + 32, *reinterpret_cast<uint32_t(*)[32]>(r + 32));
    tmem_wait_ld();
#pragma unroll
    for (int j = 0; j < 64; ++j) s[j] = __uint_as_float(r[j]);
  }
  // (the loader wrote the stage's metadata before it started the copy of the stage's key tile)
  const float2 meta = b->meta[at][kPairs ? my_block : 0];
  const float scale = meta.x;
  const int valid = __float_as_int(meta.y);
  tc_fence_before_sync();
  __syncwarp();
  mbar_arrive_if(&b->s_free[sb], lead);
  const bool active = !kPairs || kPass || (live_warp && valid >= 0);
  float mx = -INFINITY;
  if (active) {
    if (is<CELLS, kI8>(cell)) {
#pragma unroll
      for (int j = 0; j < 64; ++j) s[j] = __int2float_rn(__float_as_int(s[j]));  // |score| < 2^22: exact
    }
    if (valid < 64) {
      // ragged blocks usually lose only a few keys: the common case touches the last 8 columns
#pragma unroll
      for (int j = 56; j < 64; ++j) s[j] = j < valid ? s[j] : -INFINITY;
      if (valid < 56) {
#pragma unroll
        for (int j = 0; j < 56; ++j) s[j] = j < valid ? s[j] : -INFINITY;
      }
    }
    float m0 = max3(s[0], s[1], s[2]), m1 = max3(s[3], s[4], s[5]);
    float m2 = max3(s[6], s[7], s[8]), m3 = max3(s[9], s[10], s[11]);
#pragma unroll
    for (int j = 12; j < 60; j += 8) {
      m0 = max3(m0, s[j], s[j + 1]);
      m1 = max3(m1, s[j + 2], s[j + 3]);
      m2 = max3(m2, s[j + 4], s[j + 5]);
      m3 = max3(m3, s[j + 6], s[j + 7]);
    }
    m0 = max3(m0, s[60], s[61]);
    m1 = max3(m1, s[62], s[63]);
    mx = fmaxf(max3(m0, m1, m2), m3);
  }
  // (entry -1 was filled before the roles started, and the phase before a barrier's first counts as over)
  wait(&b->wc, &m_full[before_at], ((g - 1) >> 3) & 1, 9);
  const float2 before = b->rec[before_at][row];
  const float m_new = fmaxf(before.x, RAW != kNone ? mx : mx * scale);
  w.d = before.y * w.alpha + w.sum;
  b->rec[at][row] = make_float2(m_new, w.d);
  __syncwarp();
  mbar_arrive_if(&m_full[at], lead);
  w.alpha = ex2(RAW != kNone ? (before.x - m_new) * scale : before.x - m_new);
  if (kPairs) w.sum = 0.0f;
  if (active) {
    // exponent = s * scale + bias; the NVFP4 cell produces 6 P directly (e2m1 input range),
    // the INT8 cell P * 2^8.807 (e4m3 input range); the sums are scaled back.
    const float bias = (is<CELLS, kI8>(cell) ? kFp8Offset : (is<CELLS, kNv>(cell) ? 2.5849625007f : 0.0f)) - m_new;
    const float sum_scale = is<CELLS, kI8>(cell) ? 0.0022326917f : (is<CELLS, kNv>(cell) ? 0.16666667f : 1.0f);
    float sum;
    if (shares(D, CELLS)) {
      sum = exp_any<CELLS>(s, scale, bias, cell, p_row);
    } else if (is<CELLS, kI8>(cell)) {
      sum = exp_store<kI8>(s, scale, bias, p_row);
    } else if (is<CELLS, kNv>(cell)) {
      sum = exp_store<kNv>(s, scale, bias, p_row);
    } else {
      sum = exp_store<kF16, RAW>(s, scale, bias, p_row);
    }
    w.sum = sum * sum_scale;
  } else if (live_warp) {
    store_zeros();
  }
  fence_proxy_async_smem();
  tc_fence_before_sync();
  __syncwarp();
  mbar_arrive_if(&b->p_full[at], lead);
}

// ------------------------------------------------------------------------------------------
// MMA side
// ------------------------------------------------------------------------------------------
// The operands' descriptors are made once per phase and move with the slot: `step` is the slot's distance from
// the first one in 16-byte units (NVFP4 D = 128 16 heads of S = 32,760 1.50 ms, 1.52 with descriptors made per stage, Q64
// INT8 8 heads of 38,247 1.70 and 1.72; with the early token lookup some 25 of a stage's 2,050 warp instructions: 5.71e8 ->
// 5.64e8 for 8 mixed heads of 33,272).
__device__ __forceinline__ uint64_t moved(uint64_t desc, uint32_t step) {
  // (the address field does not overflow: shared memory ends below 2^18)
  uint32_t lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(desc));
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo + step), "r"(hi));
  return d;
}
template <int D, int CELL, int RAW = kNone>
__device__ __forceinline__ void issue_qk(uint32_t tmem_s, uint32_t tmem, uint64_t q_desc, uint64_t base,
                                         uint32_t step) {  // q_desc: NVFP4 only
  const uint64_t kd = moved(base, step);
  if (RAW != kNone) {
    constexpr uint32_t fmt = RAW == kRawBf16 ? kFmtBF16 : kFmtF16, idesc = instr_desc(fmt, fmt, kAccF32, 128, 64, 0, 0);
#pragma unroll
    for (int k = 0; k < D / 16; ++k)
      mma_f16_ts(tmem_s, tmem + kColQ + k * 8, kd + k / 4 * (64 * 128 / 16) + k % 4 * 2, idesc, k > 0);
  } else if (CELL == kF16) {
    constexpr uint32_t idesc = instr_desc(kFmtF16, kFmtF16, kAccF32, 128, 64, 0, 0);
#pragma unroll
    for (int k = 0; k < D / 16; ++k) mma_f16_ts(tmem_s, tmem + kColQ + k * 8, kd + k * 16, idesc, k > 0);
  } else if (CELL == kI8) {
    constexpr uint32_t idesc = instr_desc(kFmtS8, kFmtS8, kAccS32, 128, 64, 0, 0);
#pragma unroll
    for (int k = 0; k < D / 32; ++k) mma_i8_ts(tmem_s, tmem + kColQ + k * 8, kd + k * 16, idesc, k > 0);
  } else {
    constexpr uint32_t idesc = instr_desc_nvf4(128, 64);
    // the scale blocks follow the codes of V
    const uint64_t sd = smem_desc(0, 128, 128) + ((uint32_t)kd & 0x3fffu) + (rest_offset(D, CELL) + 32 * D) / 16;
#pragma unroll
    for (int k = 0; k < D / 64; ++k) tmem_cp_32x128b_warpx4(tmem + kColSfbK + 4 * k, sd + k * 32);
#pragma unroll
    for (int k = 0; k < D / 64; ++k)
      mma_nvf4_ss(tmem_s, q_desc + k * 16, kd + k * 16, idesc, k > 0, tmem + kColSfaQ + 4 * k,
                  tmem + kColSfbK + 4 * k);
  }
}
// Descriptor of the keys at `addr` (NVFP4: of the query codes, too).
__device__ __forceinline__ uint64_t k_desc(int d, int cell, uint32_t addr) {
  return smem_desc(addr, 128, (uint32_t)d * (cell == kF16 ? 16 : cell == kI8 ? 8 : 4));
}

template <int D, int CELL, int RAW = kNone>
__device__ __forceinline__ void issue_pv(uint32_t tmem, uint64_t pd, uint64_t vd, uint32_t accumulate) {
  if (RAW != kNone) {
    constexpr uint32_t fmt = RAW == kRawBf16 ? kFmtBF16 : kFmtF16, idesc = instr_desc(fmt, fmt, kAccF32, 128, D, 0, 1);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      mma_f16_ss(tmem + kColO, pd + k * 16, vd + k * (2 * 1024 / 16), idesc, k > 0 ? 1u : accumulate);
  } else if (CELL == kF16) {
    constexpr uint32_t idesc = instr_desc(kFmtF16, kFmtF16, kAccF32, 128, D, 0, 1);
    constexpr uint32_t v_lbo = (D / 8) * 128;  // between 8-key groups
#pragma unroll
    for (int k = 0; k < 4; ++k)
      mma_f16_ss(tmem + kColO, pd + k * 16, vd + k * (2 * v_lbo / 16), idesc, k > 0 ? 1u : accumulate);
  } else if (CELL == kI8) {
    constexpr uint32_t idesc = instr_desc(kFmtE4M3, kFmtE4M3, kAccF32, 128, D, 0, 0);
#pragma unroll
    for (int k = 0; k < 2; ++k)
      mma_f8_ss(tmem + kColO, pd + k * 16, vd + k * 16, idesc, k > 0 ? 1u : accumulate);
  } else {
    constexpr uint32_t idesc = instr_desc_nvf4(128, D);
    tmem_cp_32x128b_warpx4(tmem + kColSfbV,
                           smem_desc(0, 128, 128) + ((uint32_t)vd & 0x3fffu) + (32 * D + (D / 64) * 512) / 16);
    mma_nvf4_ss(tmem + kColO, pd, vd, idesc, accumulate, tmem + kColSfaP, tmem + kColSfbV);
  }
}
// Descriptors of the probabilities and the values at `addr`.
__device__ __forceinline__ uint64_t p_desc(int cell, uint32_t addr) {
  return smem_desc(addr, 128, (uint32_t)p_bytes(cell) / 16);
}
__device__ __forceinline__ uint64_t v_desc(int d, int cell, uint32_t addr) {
  return cell == kF16 ? smem_desc(addr, (uint32_t)d * 16, 128) : smem_desc(addr, 128, (uint32_t)p_bytes(cell) / 16);
}

// ------------------------------------------------------------------------------------------
// kernel
// ------------------------------------------------------------------------------------------
// Where a row of the tile goes in `tokens` (element offset of its first channel), -1: a padding row.
template <int D, bool kQ64>
__device__ __forceinline__ int64_t token_offset(const AttnParams& p, int head, int block0, int block1, int row) {
  constexpr int QB = kQ64 ? 64 : 128;
  const bool second = kQ64 && row >= QB;
  const int block = second ? block1 : block0, in = second ? row - QB : row;
  int token = block * QB + in;
  if (p.dense_prefix) {
    if (token >= p.s.prefix_tokens) return -1;
  } else {
    if (in >= p.counts[block]) return -1;
    token = p.s.prefix_tokens + p.indices[token];
  }
  return ((int64_t)token * p.s.heads + head) * D;
}

// The rows of a tile from the parts that the CTAs of the cluster left in their shared memory (softmax threads; a CTA
// takes every parts-th row): O = sum of O_i 2^(m_i - M), the denominator alike.  No row of a tile that misses a part.
template <int D, int RAW>
__device__ __forceinline__ void add_parts(const RawParams& p, const uint8_t* smem, int head, int tile) {
  constexpr int kPieces = D / 8;
  const uint32_t base = smem_u32(smem);
#pragma unroll 1
  for (int i = threadIdx.x; i < 128 * kPieces; i += 256) {
    const int row = (i / kPieces) * p.parts + (int)blockIdx.x, piece = i % kPieces;
    if (row >= 128 || tile * 128 + row >= p.rows) break;
    float2 md[kMostParts];
    float m = kLowest, least = 0.0f;
#pragma unroll
    for (int c = 0; c < kMostParts; ++c) {
      md[c] = c < p.parts ? peer_float2(base + 512 * D + row * 8, c) : make_float2(kLowest, 0.0f);
      m = fmaxf(m, md[c].x);
      least = fminf(least, md[c].y);
    }
    if (least == kNoPart) break;  // a CTA left over a set status word: the rows stay as they are
    float d = 0.0f, o[8] = {};
#pragma unroll
    for (int c = 0; c < kMostParts; ++c) {
      if (c < p.parts) {
        const float f = ex2((md[c].x - m) * sigma(D));
        d += md[c].y * f;
        const float4 a = peer_float4(base + (row * (D / 4) + ((2 * piece) ^ (row & 7))) * 16, c);
        const float4 z = peer_float4(base + (row * (D / 4) + ((2 * piece + 1) ^ (row & 7))) * 16, c);
        o[0] += a.x * f;
        o[1] += a.y * f;
        o[2] += a.z * f;
        o[3] += a.w * f;
        o[4] += z.x * f;
        o[5] += z.y * f;
        o[6] += z.z * f;
        o[7] += z.w * f;
      }
    }
    const float inv = 1.0f / d;  // (no score above -inf: NaN, as 0 / 0)
#pragma unroll
    for (int c = 0; c < 8; ++c) o[c] *= inv;
    uint4 v;
    if (RAW == kRawBf16) {
      v = make_uint4(bf16x2(o[0], o[1]), bf16x2(o[2], o[3]), bf16x2(o[4], o[5]), bf16x2(o[6], o[7]));
    } else {
      v = make_uint4(f16x2(o[0], o[1]), f16x2(o[2], o[3]), f16x2(o[4], o[5]), f16x2(o[6], o[7]));
    }
    *reinterpret_cast<uint4*>(static_cast<uint16_t*>(p.tokens) + (tile * 128 + row) * p.out_token + head * p.out_head +
                              piece * 8) = v;
  }
}

constexpr int kStays = -1;  // in place of a block's factors: O stays in its domain
__host__ __device__ constexpr int factor_sets(int cells, bool q64) { return mixed(cells) && q64 ? 2 : 1; }

// CELLS: the cells that a stage can be of.  A kernel of one cell has that cell's code only and
// its sizes as constants; in mixed kernels the cell is a run-time value and one copy of the
// stage code serves all: the CTAs of an SM are in different phases, and hot code that outgrows the
// instruction cache costs more than the constants give (three whole copies of the softmax stage,
// 100 KB of code: 1.48 us per 64-key stage and SM at D = 64 instead of 1.11).  For the same reason two cells
// have a kernel without the third one's code.  In the kernel for all / their own, us: NVFP4 + INT8 30 heads x 8,415 tokens
// D = 64 Q64 473 / 416, Q128 336 / 320, D = 128 Q64 546 / 513; INT8 + FP16 17 x 7,695 D = 64 184 / 179, 47 x 8,415 D = 128 Q128
// 582 / 566; NVFP4 + FP16 48 x 2,442 D = 64 98 / 89.
template <int D, int CELLS, bool kQ64, int RAW = kNone>
__global__ void __launch_bounds__(kThreads, 2) attention_kernel(const __grid_constant__ Params<RAW> p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  constexpr bool kRaw = RAW != kNone;
  static_assert(!kRaw || (CELLS == kF16 && !kQ64), "dense rows are walked as the FP16 cell's");
  constexpr bool kMixed = mixed(CELLS);
  constexpr int kFirst = !kMixed ? CELLS : has_cell(CELLS, kNv) ? kNv : kI8;
  constexpr int kLast = !kMixed ? CELLS : has_cell(CELLS, kF16) ? kF16 : kI8;
  constexpr int QB = kQ64 ? 64 : 128;
  // Kernels of one cell spill less (and are 1-5 % quicker) if the roles read again from shared memory which tile they
  // work on; those of any mix, and the ones with registers to spare, do not (4-12 % slower).
  constexpr bool kReread = !kMixed && (kQ64 || Regs<D, CELLS, kQ64>::kWide);
  // CTAs start in the order x, y, z: the longest lists of a few heads, the second ones, ..., then the next few heads
  const int head = kRaw ? blockIdx.z : blockIdx.z * gridDim.x + blockIdx.x;
  if (head >= p.s.heads) return;
  const int place = p.first_place + ((int)blockIdx.y < p.turn ? p.turn - 1 - (int)blockIdx.y : (int)blockIdx.y);
  layer::grid_dependency_wait();
  // launch order of the head's query blocks (longest list first) as written by the routing
  // stage; 0 = no order given
  int tile = place;
  const bool table = kQ64 && p.pair_table != nullptr, pairs = table || (kQ64 && p.pair_counts != nullptr);
  const int pair_tiles = (p.s.video_blocks + 1) / 2;
  if (!kRaw && !p.dense_prefix && !table) {
    const int ordered =
        pairs ? p.pair_counts[((int64_t)head * pair_tiles + place) * 4 + 3]
              : p.row_counts[((int64_t)head * p.s.video_blocks + place) * 4 + 3];
    if (ordered > 0) tile = ordered - 1;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // query blocks of this CTA (two for a complete pair) and the first one's index
  // (prefix tiles of 64 rows also go in twos: both walk every stage)
  const bool twos = pairs || (kQ64 && p.dense_prefix);
  int tile_blocks =
      twos && 2 * tile + 1 < (p.dense_prefix ? p.prefix_tiles : p.s.video_blocks) ? 2 : 1;
  int block0 = twos ? 2 * tile : tile, block1 = block0 + 1;

  // ---- this tile's work list ----
  int cnt[3] = {0, p.stages, 0};
  const int32_t* list = nullptr;
  int begin = 0;
  if constexpr (kRaw) {
    begin = (int)((int64_t)p.stages * blockIdx.x / p.parts);
    cnt[kI8] = 0;
    cnt[kF16] = (int)((int64_t)p.stages * (blockIdx.x + 1) / p.parts) - begin;
  } else if (table) {
    const int4* entry = p.pair_table + ((int64_t)head * pair_tiles + tile) * 2;
    const int4 e = entry[0], n = entry[1];
    block0 = e.x;
    block1 = e.y;
    tile_blocks = e.y >= 0 ? 2 : 1;
    list = p.pair_ids + (int64_t)head * p.capacity + e.z;
    cnt[0] = n.x;
    cnt[1] = n.y;
    cnt[2] = n.z;
  } else if (!p.dense_prefix) {
    const int32_t* ra = p.row_counts + ((int64_t)head * p.s.video_blocks + block0) * 4;
    const int32_t* counts = pairs ? p.pair_counts + ((int64_t)head * pair_tiles + tile) * 4 : ra;
    for (int c = 0; c < 3; ++c) cnt[c] = counts[c];
    list = (pairs ? p.pair_ids : p.stage_ids) + (int64_t)head * p.capacity +
           p.row_offset[(int64_t)head * p.s.video_blocks + block0];
  }
  if (cnt[0] + cnt[1] + cnt[2] == 0) {
    // nothing to attend to: +0 rows (packed rows are left alone, the assembly knows)
    if (p.tokens != nullptr)
      for (int i = threadIdx.x; i < QB * tile_blocks * (D / 8); i += kThreads) {
        const int64_t at = token_offset<D, kQ64>(p, head, block0, block1, i / (D / 8));
        if (at >= 0)
          *reinterpret_cast<uint4*>(static_cast<uint16_t*>(p.tokens) + at + i % (D / 8) * 8) = make_uint4(0, 0, 0, 0);
      }
    return;
  }
  // After a give-up anywhere on this device the status word stays set: later CTAs (of this and
  // of later launches, until the host clears the word) return at once instead of each running
  // into its own wait limit.  One thread reads the word for the whole CTA: another CTA may set it at any
  // time, and if only some warps of this one left, the others would go on without tensor memory, without
  // barriers or with a warpgroup short of the warps its setmaxnreg waits for.
  if (__syncthreads_or(threadIdx.x == 0 && *reinterpret_cast<volatile int32_t*>(p.status) != 0)) {
    if constexpr (kRaw) {
      // The other CTAs of the cluster may have seen the word clear.  They meet this one at two barriers (before they add up
      // the parts and before they leave: each role passes exactly these), and find here that this part is missing.
      if (threadIdx.x < 128) reinterpret_cast<float2*>(smem + 512 * D)[threadIdx.x] = make_float2(kLowest, kNoPart);
      cluster_sync();
      cluster_sync();
    }
    return;
  }

  uint8_t* q_smem = smem;
  uint8_t* ring = smem + p.q_region;
  // (two sets of factors for the blocks of a pair, which may come from different phases)
  constexpr int kFactors = factor_sets(CELLS, kQ64);
  float* colf = reinterpret_cast<float*>(ring + (size_t)p.ring_bytes);
  Shared* b = reinterpret_cast<Shared*>(colf + kFactors * D);

  if (warp == 0) {
    if (lane < kRing) {
      mbar_init(&b->kv_full[lane], 1);
      mbar_init(&b->pv_done[lane], 1);
      mbar_init(&b->p_full[lane], 8);
    }
    mbar_init(&b->m_full[0][lane], 1);  // all four quadrants' rings
    if (lane == 0) {
      for (int i = 0; i < kSplitValues; ++i) mbar_init(&b->v_full[i], 1);
      mbar_init(&b->q_moved, 4);
      mbar_init(&b->q_full, 1);
      mbar_init(&b->q_free, 1);
      for (int i = 0; i < 2; ++i) {
        mbar_init(&b->s_full[i], 1);
        mbar_init(&b->s_free[i], 4);
      }
      mbar_init(&b->nv_done, 1);
      mbar_init(&b->all_done, 1);
      mbar_init(&b->qk_done, 1);
      b->wc.abort = 0;
      b->wc.status = p.status;
      b->wc.limit_ns = p.wait_ns;
      b->head = head;
      b->block[0] = block0;
      b->block[1] = block1;
      b->tile_blocks = tile_blocks;
      b->list = list;
      // phase c of a union of neighbours sits where the two blocks' phases before it would end
      const bool apart = pairs && !table;
      const int32_t* ra = apart ? p.row_counts + ((int64_t)head * p.s.video_blocks + block0) * 4 : nullptr;
      int before = begin;
      for (int c = 0; c < 3; ++c) {
        b->cnt[c] = cnt[c];
        b->first_of[c] = before;
        before += apart ? ra[c] + (tile_blocks == 2 ? ra[4 + c] : 0) : cnt[c];
      }
    }
    mbar_init_fence();
  } else if (warp < 5) {
    b->rec[kRing - 1][threadIdx.x - 32] = make_float2(kRaw ? kLowest : -5.0e6f, 0.0f);  // before the first stage
  } else if (kFactors == 2 && warp == 5 && lane < 2) {
    // A block of a pair without a stage of a phase stays in its domain, and one without a phase before it has
    // nothing to move, so that a block's result does not depend on its partner: two steps instead of one, or there
    // and back, round differently.
    bool has[3] = {false, true, false};  // prefix rows
    if (!p.dense_prefix) {
      const int32_t* n =
          p.row_counts + ((int64_t)head * p.s.video_blocks + (lane < tile_blocks && lane ? block1 : block0)) * 4;
#pragma unroll
      for (int c = 0; c < 3; ++c) has[c] = n[c] > 0;
    }
    b->move[lane][0] = has[0] && has[1] ? 0 : kStays;
    b->move[lane][1] = has[2] && (has[0] || has[1]) ? (has[1] ? 0 : D) : kStays;
    b->last[lane] = has[2] ? kF16 : has[1] ? kI8 : kNv;
  }
  // Query rows beyond QB (64-row tiles padded to the 128-row MMA shape) are never
  // initialised: rows are independent, their results stay in TMEM lanes nobody reads.
  if (warp == kPvWarp) {
    tmem_alloc(&b->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = b->tmem_base;

  const float* vscale_kept = p.o.v_e4m3_scale ? p.o.v_e4m3_scale + (int64_t)head * D : nullptr;
  const float nv_dom = p.s.v_global_scale * (1.0f / (6.0f * 448.0f));

  // Register counts move between the warpgroups; all four warps of a warpgroup execute the same
  // setmaxnreg instruction, and each sits at the top of the branch that runs under the new count.
  if (warp >= kLoaderWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegs));
    if (warp == kLoaderWarp) {
      // =============================== loader ===============================
      // The whole warp walks the list with uniform control flow; one lane issues.
      const uint32_t lead = lane == 0;
      const int head_at = kReread ? b->head : head, first_block = kReread ? b->block[0] : block0;
      const int blocks = kReread ? b->tile_blocks : tile_blocks;
      const int32_t* list_at = kReread ? b->list : list;
      const int q_index_fp = head_at * p.s.video_blocks + first_block;  // q_fp16 / q_nvfp4 record
      const int64_t q_index_i8 =
          (int64_t)head_at * p.q_tiles_int8 + (p.dense_prefix ? p.s.video_blocks : 0) + first_block;
      const int step = (kReread ? b->block[1] : block1) - first_block;  // from a pair's first record to its second
      int phase_ord = 0, g = 0, v_fills = 0, moves = 0;
#pragma unroll 1
      for (int cell = kFirst; cell <= kLast; ++cell) {
        const int n = b->cnt[cell];
        if (n == 0) continue;
        if (phase_ord > 0) wait<kMmaRole>(&b->wc, &b->q_free, (phase_ord - 1) & 1, 1);
        const int qbytes = is<CELLS, kNv>(cell) ? (int)rec::q_nvfp4_bytes(QB, D)
                                       : (is<CELLS, kI8>(cell) ? (int)rec::q_int8_bytes(QB, D) : (int)rec::q_fp16_bytes(QB, D));
        const uint8_t* qsrc =
            is<CELLS, kNv>(cell) ? static_cast<const uint8_t*>(p.o.q_nvfp4) + (int64_t)q_index_fp * qbytes
            : is<CELLS, kI8>(cell) ? static_cast<const uint8_t*>(p.o.q_int8) + q_index_i8 * qbytes
                          : static_cast<const uint8_t*>(p.o.q_fp16) + (int64_t)q_index_fp * qbytes;
        mbar_arrive_expect_tx(&b->q_full, qbytes * blocks, lead);
        if constexpr (kRaw) {
#pragma unroll
          for (int c = 0; c < D; c += 64) tensor_g2s(q_smem + c * 256, &p.q, c, head_at, tile * 128, &b->q_full, lead);
        } else if (is<CELLS, kNv>(cell) && kQ64) {
          // codes fill the first half of the 128-row tile; scale blocks follow the full tile.
          // A pair's second record: codes into the second half of the tile, scale blocks behind
          // the first record's (the QK warp folds them into one block before it copies them).
          const int codes = QB * D / 2;
          bulk_g2s(q_smem, qsrc, codes, &b->q_full, lead);
          bulk_g2s(q_smem + 128 * D / 2, qsrc + codes, qbytes - codes, &b->q_full, lead);
          if (blocks == 2) {
            const uint8_t* second = qsrc + (int64_t)step * qbytes;
            bulk_g2s(q_smem + codes, second, codes, &b->q_full, lead);
            bulk_g2s(q_smem + 128 * D / 2 + (qbytes - codes), second + codes, qbytes - codes, &b->q_full, lead);
          }
        } else {
          // two records of 64 rows make a 128-row tile
          bulk_g2s(q_smem, qsrc, qbytes, &b->q_full, lead);
          if (kQ64 && blocks == 2) bulk_g2s(q_smem + qbytes, qsrc + (int64_t)step * qbytes, qbytes, &b->q_full, lead);
        }
        const int kvbytes = record_bytes(D, cell), kbytes = k_bytes(D, cell), rest = rest_offset(D, cell);
        const uint8_t* kvbase =
            (is<CELLS, kNv>(cell) ? static_cast<const uint8_t*>(p.o.kv_nvfp4)
             : is<CELLS, kI8>(cell) ? static_cast<const uint8_t*>(p.o.kv_int8)
                           : static_cast<const uint8_t*>(p.o.kv_fp16)) +
            (int64_t)head_at * p.stages * kvbytes;
        const int first = b->first_of[cell];
        // The ring is cut into equal slots of this phase's size; the slots of the previous phase
        // must all be released before the new geometry is written (PVs complete in stage order).
        const int slot_size = stage_bytes(D, cell);
        const int nslot = slot_count(p.ring_bytes, D, cell);
        if (g > 0) wait<kMmaRole>(&b->wc, &b->pv_done[(g - 1) & (kRing - 1)], ((g - 1) >> 3) & 1, 2);
        float q_scale[2] = {1.0f, 1.0f};
        const float* kscale = nullptr;
        if (is<CELLS, kI8>(cell)) {
          q_scale[0] = p.o.q_int8_scale[q_index_i8];
          if (blocks == 2) q_scale[1] = p.o.q_int8_scale[q_index_i8 + step];
          kscale = p.o.k_int8_scale + (int64_t)head_at * p.stages;
        }
        const float base = is<CELLS, kNv>(cell) ? sigma(D) * p.s.q_global_scale * p.s.k_global_scale : sigma(D);
        // list entries, 32 at a time, one per lane, with their metadata
        int stage_l = 0;
        float2 meta_l[2] = {make_float2(base, 0.0f), make_float2(base, 0.0f)};
        int slot = first_slot(D, cell);
        const bool split = split_kv(D, cell);
        int prev_stage = 0;
        // (split phases: a stage's values follow the next stage's keys)
        const int end = n + (split ? 1 : 0);
#pragma unroll 1
        for (int i = 0; i < end; ++i) {
          if ((i & 31) == 0 && i < n) {
            const int at = i + lane;
            int entry = 0;
            int valid;
            if constexpr (kRaw) {
              entry = first + at;
              stage_l = entry;
              valid = p.tokens_in - stage_l * 64;
            } else {
              if (at < n) entry = list_at != nullptr ? list_at[first + at] : at;
              stage_l = entry & 0x3fffffff;
              valid = p.valid_k[stage_l];
            }
            meta_l[0].y = __int_as_float(!pairs || ((entry >> 30) & 1) ? valid : -1);
            if (kQ64) meta_l[1].y = __int_as_float(entry < 0 || p.dense_prefix ? valid : -1);
            if (is<CELLS, kI8>(cell)) {
              const float ks = kscale[stage_l];
              meta_l[0].x = sigma(D) * (q_scale[0] * ks);
              if (kQ64) meta_l[1].x = sigma(D) * (q_scale[1] * ks);
            }
          }
          const int stage = __shfl_sync(0xffffffffu, stage_l, i & 31);
          const int gi = g + i;
          if (i < n) {
            if (i >= nslot)
              wait<kMmaRole>(&b->wc, &b->pv_done[(gi - nslot) & (kRing - 1)], ((gi - nslot) >> 3) & 1, 2);
            if (split && i == 2) wait<kMmaRole>(&b->wc, &b->q_moved, moves & 1, 2);
            const int at = gi & (kRing - 1);
            if (lane == (i & 31)) {
              b->meta[at][0] = meta_l[0];
              if (kQ64) b->meta[at][1] = meta_l[1];
            }
            __syncwarp();
            const int bytes = split ? kbytes : kvbytes;
            const uint8_t* src = kvbase + (int64_t)stage * kvbytes;
            uint8_t* dst = (split ? smem : ring) + (size_t)slot * slot_size;
            mbar_arrive_expect_tx(&b->kv_full[at], bytes, lead);
            if constexpr (kRaw) {
#pragma unroll
              for (int c = 0; c < D; c += 64)
                tensor_g2s(dst + c * 128, &p.k, c, head_at, stage * 64, &b->kv_full[at], lead);
              if (!split) tensor_g2s(dst + rest, &p.v, 0, head_at, stage * 64, &b->kv_full[at], lead);
            } else if (split || rest == kbytes) {
              bulk_g2s(dst, src, bytes, &b->kv_full[at], lead);
            } else {
              bulk_g2s(dst, src, kbytes, &b->kv_full[at], lead);
              bulk_g2s(dst + rest, src + kbytes, kvbytes - kbytes, &b->kv_full[at], lead);
            }
            slot = slot + 1 == nslot ? 0 : slot + 1;
          }
          if (split && i > 0) {
            const int before = gi - 1 - kSplitValues;  // the stage that had the value buffer
            if (i > kSplitValues) wait<kMmaRole>(&b->wc, &b->pv_done[before & (kRing - 1)], (before >> 3) & 1, 2);
            uint64_t* full = &b->v_full[(i - 1) & 1];
            mbar_arrive_expect_tx(full, kvbytes - kbytes, lead);
            if constexpr (kRaw) {
#pragma unroll
              for (int c = 0; c < D; c += 64)
                tensor_g2s(smem + (kSplitKeys + ((i - 1) & 1)) * slot_size + c * 128, &p.v, c, head_at, prev_stage * 64, full,
                           lead);
            } else {
              bulk_g2s(smem + (kSplitKeys + ((i - 1) & 1)) * slot_size,
                       kvbase + (int64_t)prev_stage * kvbytes + kbytes, kvbytes - kbytes, full, lead);
            }
            ++v_fills;
          }
          prev_stage = stage;
        }
        g += n;
        ++phase_ord;
        moves += !is<CELLS, kNv>(cell);
      }
      if (b->wc.abort) {
        // unwinding: the copies in flight must land before the CTA gives its shared memory back
        for (int k = max(0, g - kRing); k < g; ++k)
          drain_wait(&b->kv_full[k & (kRing - 1)], (k >> 3) & 1, kDrainNs);
        for (int j = max(0, v_fills - kSplitValues); j < v_fills; ++j)
          drain_wait(&b->v_full[j & 1], (j >> 1) & 1, kDrainNs);
        if (phase_ord > 0) drain_wait(&b->q_full, (phase_ord - 1) & 1, kDrainNs);
      }
    } else if (warp == kQkWarp) {
      // =============================== S = Q K^T ===============================
      // Uniform control flow for the whole warp; the tcgen05 instructions are one elected lane's.
      int g = 0, phase_ord = 0;
      int moves = 0;
      uint32_t used = 0, free_par = 0;  // (where the parities are kept)
      const bool leader = elect_one();
      const uint32_t q_addr = smem_u32(q_smem), ring_addr = smem_u32(ring);
#pragma unroll 1
      for (int cell = kFirst; cell <= kLast; ++cell) {
        const int n = b->cnt[cell];
        if (n == 0) continue;
        if (!is<CELLS, kNv>(cell)) {
          wait<kMmaRole>(&b->wc, &b->q_moved, moves & 1, 3);
          ++moves;
        } else {
          wait<kMmaRole>(&b->wc, &b->q_full, phase_ord & 1, 3);
        }
        tc_fence_after_sync();
        const int nslot = slot_count(p.ring_bytes, D, cell);
        const uint32_t stride = stage_bytes(D, cell);
        const uint32_t base_addr = split_kv(D, cell) ? smem_u32(smem) : ring_addr;
        const uint64_t base = kRaw ? swizzled_desc(base_addr, 16) : k_desc(D, cell, base_addr);
        const uint64_t q_desc = k_desc(D, kNv, q_addr);
        if (is<CELLS, kNv>(cell)) {
          if ((kReread ? b->tile_blocks : tile_blocks) == 2) {
            // Scale bytes of rows 0-63 sit in the low eight bytes of every 16-byte chunk, those of
            // rows 64-127 in the high eight.  Both records hold their 64 rows in the low halves:
            // the second record's move up into the first record's empty high halves.
            uint8_t* sfa = q_smem + 128 * D / 2;
            const uint8_t* sfb = sfa + (D / 64) * 512;
            for (int c = lane; c < (D / 64) * 32; c += 32) {
              const uint2 lo = *reinterpret_cast<const uint2*>(sfb + c * 16);
              *reinterpret_cast<uint2*>(sfa + c * 16 + 8) = lo;
            }
            fence_proxy_async_smem();
            __syncwarp();
          }
          const uint32_t qsf = q_addr + 128 * D / 2;
          if (leader) {
#pragma unroll
            for (int k = 0; k < D / 64; ++k)
              tmem_cp_32x128b_warpx4(tmem + kColSfaQ + 4 * k, smem_desc(qsf + 512 * k, 128, 128));
          }
          __syncwarp();
        }
        // a stage's scores are computed as soon as its key tile has landed and its score buffer
        // has been read
        int slot = first_slot(D, cell);
#pragma unroll 1
        for (int i = 0; i < n; ++i, ++g) {
          const int sb = s_buffer<D>(g);
          wait<kMmaRole>(&b->wc, &b->kv_full[g & (kRing - 1)], (g >> 3) & 1, 4);
          if constexpr (keeps_free_parity(D, CELLS, kQ64)) {
            if ((used >> sb) & 1u) {
              wait<kMmaRole>(&b->wc, &b->s_free[sb], (free_par >> sb) & 1u, 5);
              free_par ^= 1u << sb;
            }
            used |= 1u << sb;
          } else {
            // (the buffer's scores before: of the stage before, or, with two buffers, the one before that)
            if (g > (D == 64)) wait<kMmaRole>(&b->wc, &b->s_free[sb], (D == 64 ? (g >> 1) - 1 : g - 1) & 1, 5);
          }
          tc_fence_after_sync();
          if (leader) {
            const uint32_t tmem_s = tmem + (sb ? kColS1 : kColS), step = slot * (stride / 16);
            if (is<CELLS, kI8>(cell)) {
              issue_qk<D, kI8>(tmem_s, tmem, q_desc, base, step);
            } else if (is<CELLS, kNv>(cell)) {
              issue_qk<D, kNv>(tmem_s, tmem, q_desc, base, step);
            } else {
              issue_qk<D, kF16, RAW>(tmem_s, tmem, q_desc, base, step);
            }
            mma_commit(&b->s_full[g & 1]);
            if (i == n - 1) mma_commit(&b->q_free);
          }
          __syncwarp();
          slot = slot + 1 == nslot ? 0 : slot + 1;
        }
        ++phase_ord;
      }
      if (b->wc.abort) {
        if (leader) mma_commit(&b->qk_done);
        __syncwarp();
        drain_wait(&b->qk_done, 0, kDrainNs);
      }
    } else if (warp == kPvWarp) {
      // =============================== O += P V ===============================
      int g = 0;
      const uint32_t ring_addr = smem_u32(ring);
      const bool leader = elect_one();
#pragma unroll 1
      for (int cell = kFirst; cell <= kLast; ++cell) {
        const int n = b->cnt[cell];
        if (n == 0) continue;
        const int nslot = slot_count(p.ring_bytes, D, cell);
        const uint32_t stride = stage_bytes(D, cell);
        const uint32_t base_addr = split_kv(D, cell) ? smem_u32(smem) : ring_addr;
        const uint64_t p_base = p_desc(cell, base_addr);
        const uint32_t v_addr = base_addr + (split_kv(D, cell) ? kSplitKeys * stride : rest_offset(D, cell));
        const uint64_t v_base = kRaw ? swizzled_desc(v_addr, 64 * 128) : v_desc(D, cell, v_addr);
        int slot = first_slot(D, cell);
#pragma unroll 1
        for (int i = 0; i < n; ++i, ++g) {
          // (a tile has at most one phase with value buffers)
          if (split_kv(D, cell)) wait<kMmaRole>(&b->wc, &b->v_full[i & 1], (i >> 1) & 1, 6);
          wait<kMmaRole>(&b->wc, &b->p_full[g & (kRing - 1)], (g >> 3) & 1, 6);
          tc_fence_after_sync();
          if (leader) {
            const uint64_t pd = moved(p_base, slot * (stride / 16));
            const uint64_t vd = moved(v_base, (split_kv(D, cell) ? i & 1 : slot) * (stride / 16));
            if (is<CELLS, kI8>(cell)) {
              issue_pv<D, kI8>(tmem, pd, vd, g > 0);
            } else if (is<CELLS, kNv>(cell)) {
              issue_pv<D, kNv>(tmem, pd, vd, g > 0);
            } else {
              issue_pv<D, kF16, RAW>(tmem, pd, vd, g > 0);
            }
            mma_commit(&b->pv_done[g & (kRing - 1)]);
            if (kMixed && is<CELLS, kNv>(cell) && i == n - 1) mma_commit(&b->nv_done);
          }
          __syncwarp();
          slot = slot + 1 == nslot ? 0 : slot + 1;
        }
      }
      if (leader) mma_commit(&b->all_done);
      __syncwarp();
      // unwinding: the MMAs in flight must be over before tensor memory is given back
      if (b->wc.abort) drain_wait(&b->all_done, 0, kDrainNs);
    }
    if (kRaw) cluster_sync();  // as the softmax warps before they add up the tile's parts
  } else if (warp >= kCorrWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Regs<D, CELLS, kQ64>::kRescale));
    // =============================== O rescale ===============================
    const int row = (warp - kCorrWarp) * 32 + lane;
    uint64_t* m_full = b->m_full[warp - kCorrWarp];
    const uint32_t tmem_row = tmem + ((uint32_t)((warp - kCorrWarp) * 32) << 16);
    const uint32_t lead = lane == 0;
    float m = kRaw ? kLowest : -5.0e6f;
    int g = 0, prev_cell = -1, phase_ord = 0;
#pragma unroll 1
    for (int cell = kFirst; cell <= kLast; ++cell) {
      const int n = b->cnt[cell];
      if (n == 0) continue;
      const bool change = kMixed && prev_cell >= 0;
      if (change) {
        // per-channel factor that moves O from the previous phase's domain into this one's
        asm volatile("bar.sync 5, 128;" ::: "memory");
        const float* vscale = kReread ? p.o.v_e4m3_scale + (int64_t)b->head * D : vscale_kept;
        if (row < D) {
          const float from = is<CELLS, kNv>(prev_cell) ? nv_dom
                                              : (is<CELLS, kI8>(prev_cell) ? vscale[row] * 0.0022326917f : 1.0f);
          const float to = is<CELLS, kI8>(cell) ? vscale[row] * 0.0022326917f : 1.0f;
          colf[row] = to == 0.0f ? 0.0f : from / to;
          if (kFactors == 2) colf[D + row] = nv_dom;  // from NVFP4 into FP16 for a block without the phase between
        }
        asm volatile("bar.sync 5, 128;" ::: "memory");
      }
      const int factors = kFactors == 2 && change ? b->move[row >= QB][cell - kI8] : 0;
      const bool moves = change && (kFactors == 1 || factors != kStays);
      if (!is<CELLS, kNv>(cell)) {
        // Q into tensor memory.  Its columns are free: the INT8 phase's Q has been read when the record
        // that takes its place in shared memory arrives, the NVFP4 phase's scale factors below.
        if (kMixed && b->cnt[kNv] > 0) wait<kRescaleRole>(&b->wc, &b->nv_done, 0, 31);
        wait<kRescaleRole>(&b->wc, &b->q_full, phase_ord & 1, 32);
        const int chunks = is<CELLS, kI8>(cell) ? D / 16 : D / 8;
#pragma unroll 1
        for (int c = 0; c < chunks; c += 2) {
          uint32_t r[8];
          if (kRaw) {
            const uint8_t* from = q_smem + (c >> 3) * (128 * 128) + row * 128;
            *reinterpret_cast<uint4*>(r) = *reinterpret_cast<const uint4*>(from + (((c & 7) ^ (row & 7)) << 4));
            *reinterpret_cast<uint4*>(r + 4) = *reinterpret_cast<const uint4*>(from + ((((c + 1) & 7) ^ (row & 7)) << 4));
          } else {
            *reinterpret_cast<uint4*>(r) = *reinterpret_cast<const uint4*>(q_smem + rec::tile_offset(row, c, chunks));
            *reinterpret_cast<uint4*>(r + 4) =
                *reinterpret_cast<const uint4*>(q_smem + rec::tile_offset(row, c + 1, chunks));
          }
          tmem_st8(tmem_row + kColQ + c * 4, r);
        }
        tmem_wait_st();
        tc_fence_before_sync();
        __syncwarp();
        mbar_arrive_if(&b->q_moved, lead);
      }
      ++phase_ord;
#pragma unroll 1
      for (int i = 0; i < n; ++i, ++g) {
        const int at = g & (kRing - 1);
        wait<kRescaleRole>(&b->wc, &m_full[at], (g >> 3) & 1, 30);
        const float m_new = b->rec[at][row].x;
        const bool first = moves && i == 0;
        if (g > 0 && (first || __any_sync(0xffffffffu, m_new != m))) {
          const float alpha = ex2(kRaw ? (m - m_new) * sigma(D) : m - m_new);
          // O may only be touched once the previous PV is complete
          wait<kRescaleRole>(&b->wc, &b->pv_done[(g - 1) & (kRing - 1)], ((g - 1) >> 3) & 1, 20);
          tc_fence_after_sync();
          rescale_o<D, Regs<D, CELLS, kQ64>::kRescaleColumns>(tmem_row, alpha, first ? colf + factors : nullptr);
          tc_fence_before_sync();
        }
        m = m_new;
        __syncwarp();
        mbar_arrive_if(&b->p_full[at], lead);
      }
      prev_cell = cell;
    }
    if (kRaw) cluster_sync();
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Regs<D, CELLS, kQ64>::kSoftmax));
    // Formed anew where that leaves the loop more registers (pointer_anew): what is derived from the pointer that all roles
    // have is kept from the kernel's start.
    constexpr bool kAnew = pointer_anew(D, CELLS, kQ64) || kRaw;
    uint32_t b_at = p.q_region + p.ring_bytes + kFactors * D * 4;
    if (kAnew) asm volatile("" : "+r"(b_at));
    Shared* const b_kept = b;
    Shared* const b = kAnew ? reinterpret_cast<Shared*>(smem + b_at) : b_kept;
    // =============================== softmax rows ===============================
    const int row = (warp & 3) * 32 + lane;  // query row == TMEM lane
    const int parity = warp >> 2;            // which stages this warpgroup runs
    const uint32_t tmem_row = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    SoftmaxWalk w{0u, 0.0f, 1.0f, 0.0f};
    int g = 0, last_cell = kFirst;
    const int blocks = kReread ? b->tile_blocks : tile_blocks;
    const bool live_warp = !kQ64 || (warp & 3) * 32 < QB * blocks;
    const int my_block = kQ64 && (warp & 3) * 32 >= QB && blocks == 2 ? 1 : 0;  // which block of a pair
    if (kFirst == kNv && b->cnt[kNv] > 0 && parity == 0) {
      tmem_st4(tmem_row + kColSfaP, 0x7e7e7e7eu);  // constant 448 block scale of P
      tmem_wait_st();
    }
#pragma unroll 1
    for (int cell = kFirst; cell <= kLast; ++cell) {
      const int n = b->cnt[cell];
      if (n == 0) continue;
      const int nslot = slot_count(p.ring_bytes, D, cell);
      const int stride = stage_bytes(D, cell);
      uint8_t* p_row = (split_kv(D, cell) ? smem : ring) + rec::tile_offset(row, 0, p_bytes(cell) / 2048);
      const int first = (g & 1) == parity ? 0 : 1;
      int slot = first_slot(D, cell) + first;
#pragma unroll 1
      for (int i = first; i < n; i += 2) {
        softmax_stage<D, CELLS, kQ64, kQ64 && !kMixed, RAW>(b, p_row + slot * stride, tmem_row, row, g + i, cell, live_warp,
                                                        my_block, w);
        slot += 2;
        if (slot >= nslot) slot -= nslot;
      }
      g += n;
      last_cell = cell;
    }
    // ---- epilogue: O_true / d -> fp16, packed row order; each warpgroup writes half the channels ----
    // packed rows: this tile's place; token rows: the row's token, in the caller's type (looked up under the last PV)
    uint16_t* dst = nullptr;
    const int head_at = kReread ? b->head : head;
    const int first_block = kReread ? b->block[0] : block0, second_block = kReread ? b->block[1] : block1;
    if (!kRaw && row < QB * (kReread ? b->tile_blocks : tile_blocks)) {
      if (p.tokens == nullptr) {
        dst = reinterpret_cast<uint16_t*>(p.out) +
              ((int64_t)head_at * p.out_rows + (kQ64 && row >= QB ? second_block * QB + row - QB : first_block * QB + row)) * D;
      } else {
        const int64_t at = token_offset<D, kQ64>(p, head_at, first_block, second_block, row);
        if (at >= 0) dst = static_cast<uint16_t*>(p.tokens) + at;
      }
    }
    const float* vscale = kReread ? p.o.v_e4m3_scale + (int64_t)head_at * D : vscale_kept;
    wait(&b->wc, &b->all_done, 0, 7);
    // d(G-1) from d(G-3) and the last two stages' (alpha, sum), which the two groups hold; every
    // other use of rec is over
    const bool last_mine = ((g - 1) & 1) == parity;
    // (a part's maxima are needed, too: its last stage's entries stay)
    const int free0 = kRaw ? g & (kRing - 1) : 0, free1 = kRaw ? (g + 1) & (kRing - 1) : 1;
    if (!last_mine) b->rec[free0][row] = make_float2(w.alpha, w.sum);
    asm volatile("bar.sync 6, 256;" ::: "memory");
    if (last_mine) {
      const float2 other = b->rec[free0][row];
      b->rec[free1][row] = make_float2((w.d * other.x + other.y) * w.alpha + w.sum, 0.0f);
    }
    asm volatile("bar.sync 6, 256;" ::: "memory");
    if constexpr (kRaw) {
      // This CTA's part of the tile, before the division: rows of fp32 (16-byte pieces swizzled: a warp's
      // rows are 4 * D bytes apart), maxima and denominators behind them.
      tc_fence_after_sync();
#pragma unroll 1
      for (int c0 = parity * (D / 2); c0 < (parity + 1) * (D / 2); c0 += 32) {
        uint32_t r[32];
        tmem_ld32(tmem_row + kColO + c0, r);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 32; j += 4)
          reinterpret_cast<uint4*>(smem)[row * (D / 4) + (((c0 + j) / 4) ^ (row & 7))] =
              make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
      }
      if (parity == 0)
        reinterpret_cast<float2*>(smem + 512 * D)[row] =
            make_float2(b->rec[(g - 1) & (kRing - 1)][row].x, b->rec[free1][row].x);
      cluster_sync();
      add_parts<D, RAW>(p, smem, head_at, tile);
    } else if (live_warp) {
      tc_fence_after_sync();
      if (kFactors == 2) last_cell = b->last[my_block];
      const float d = b->rec[1][row].x;
      const float inv = d > 0.0f ? 1.0f / d : 0.0f;
      const bool bf16 = p.tokens != nullptr && p.tokens_bf16;
#pragma unroll 1
      for (int c0 = parity * (D / 2); c0 < (parity + 1) * (D / 2); c0 += 32) {
        uint32_t r[32];
        tmem_ld32(tmem_row + kColO + c0, r);
        tmem_wait_ld();
        if (dst != nullptr) {
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            float f[8];
            if constexpr (kFactors == 2) {
              // (the channels' factors are loaded together: one by one under a condition that is not known to be the
              // warp's, each is waited for, 3 us of a small call: 7 heads x 2,293 tokens, D = 128 65.3, now 62.1)
              float factor[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) factor[i] = is<CELLS, kNv>(last_cell) ? nv_dom : 1.0f;
              if (is<CELLS, kI8>(last_cell)) {
#pragma unroll
                for (int i = 0; i < 8; ++i) factor[i] = vscale[c0 + j + i] * 0.0022326917f;
              }
#pragma unroll
              for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(r[j + i]) * factor[i] * inv;
            } else {
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                f[i] = __uint_as_float(r[j + i]);
                if (is<CELLS, kNv>(last_cell)) f[i] *= nv_dom;
                if (is<CELLS, kI8>(last_cell)) f[i] *= vscale[c0 + j + i] * 0.0022326917f;
                f[i] *= inv;
              }
            }
            uint4 v = make_uint4(f16x2(f[0], f[1]), f16x2(f[2], f[3]), f16x2(f[4], f[5]), f16x2(f[6], f[7]));
            if (bf16)
              v = make_uint4(bf16x2_of_f16x2(v.x), bf16x2_of_f16x2(v.y), bf16x2_of_f16x2(v.z), bf16x2_of_f16x2(v.w));
            // a block of a pair may have an empty list of its own: +0 rows
            if (d == 0.0f) v = make_uint4(0, 0, 0, 0);
            *reinterpret_cast<uint4*>(dst + c0 + j) = v;
          }
        }
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == kPvWarp) tmem_dealloc(tmem, kTmemCols);
  if (kRaw) cluster_sync();  // the others have read this CTA's part
}

// Heads whose query tiles start in turns, longest lists first: as many as keep keys and values of up to 48 MB in use (they
// stay in L2).  With heads one after the other a call of a few waves of CTAs ends with the last head's lists, whichever they
// are; lists of different lengths gain up to 13 %, equal ones nothing.  One after the other / in turns, us: NVFP4 D = 64,
// Q64, 9 heads x 14,161 tokens 201.5 / 177.6, Q128, 8 x 9,360 106.6 / 97.1; INT8 + NVFP4 D = 128, 11 x 9,464 450 / 407; INT8
// Q128, 33 x 2,790 95.9 / 91.8.  24 MB gain less (11 x 9,464 424), past L2 it turns (10 MB per head, 56 x 38,247 tokens INT8,
// with 2, 4, 6, 16 and 56 heads at a time 9.66, 9.82, 9.92, 10.32 and 10.69 ms).  Calls of less than a CTA per SM lose: 70 / 71.
// Calls of one to four CTAs per SM: the lists of the first 148 CTAs start shortest first, so that the SM of the shortest gets
// the longest of the others (4 x 6,664 tokens NVFP4 D = 64, 208 CTAs, 60.4 / 54.9, without the turn 55.3; 8 x 4,485 INT8,
// 360 CTAs, 91.0 and 94.9 without; 1 x 43,680, 342 CTAs, 424 and 445; past four CTAs nothing).
constexpr int kSms = 148;
constexpr int64_t kHeadsBytes = 48 << 20;
// FP16 alone at D = 128, whose stages are the largest (one or two heads of 33,272 tokens at a time), gains the least: Q128, lists
// of different lengths, 20 heads x 7,800 tokens (4 waves) 244 / 223, 16 x 20,280 (9) 913 / 883, 24 x 20,280 (13) 1,351 / 1,308,
// 45 x 14,040 (17) 1,268 / 1,268, 20 x 33,272 (18) 2,599 / 2,595; with pairs 24 x 20,280 1,420 / 1,394, 20 x 33,272 2,882 / 2,785.
// Equal lists, which past ten waves are limited by power, lose up to 1.3 % there (45 x 14,040 1,377 / 1,392, 20 x 33,272 2,740 /
// 2,776, 12 x 20,280 729 / 721).
// In how many groups the heads of a launch start: one after the other, the heads of a group in turns.
int head_groups(const AttnParams& p, int64_t ctas) {
  if (p.dense_prefix || ctas <= kSms) return p.s.heads;
  const int64_t bytes = (p.s.has_nvfp4 ? rec::kv_nvfp4_bytes(p.s.head_dim) : 0) +
                        (p.s.has_int8 ? rec::kv_int8_bytes(p.s.head_dim) : 0) +
                        (p.s.has_fp16 ? rec::kv_fp16_bytes(p.s.head_dim) : 0);
  const int most = (int)max((int64_t)1, min((int64_t)p.s.heads, kHeadsBytes / (bytes * p.stages)));
  return (p.s.heads + most - 1) / most;
}

template <int D, int CELLS, bool kQ64>
int launch_kernel(AttnParams& p, int tiles, size_t smem, cudaStream_t st) {
  auto kernel = attention_kernel<D, CELLS, kQ64>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
      cudaSuccess)
    return ANEMOI_SM100_ELAUNCH;
  const int64_t ctas = (int64_t)tiles * p.s.heads;
  const int groups = head_groups(p, ctas);
  p.turn = !p.dense_prefix && groups == 1 && ctas > kSms && ctas <= 4 * kSms ? kSms / p.s.heads : 0;
  // (the tiles of a head are the grid's y: a prefix of millions of rows takes several launches)
  for (p.first_place = 0; p.first_place < tiles; p.first_place += 65535) {
    const dim3 grid((p.s.heads + groups - 1) / groups, min(65535, tiles - p.first_place), groups);
    if (layer::launch(kernel, grid, dim3(kThreads), smem, st, p) != cudaSuccess) return ANEMOI_SM100_ELAUNCH;
  }
  return ANEMOI_SM100_OK;
}

template <int D, bool kQ64>
int launch(AttnParams& p, int tiles, cudaStream_t st) {
  int q_region = 0, slot = 0;
  const bool use[3] = {p.s.has_nvfp4 && !p.dense_prefix, p.s.has_int8 != 0, p.s.has_fp16 && !p.dense_prefix};
  for (int cell = 0; cell < 3; ++cell) {
    if (!use[cell]) continue;
    // a pair of Q64 blocks brings a second set of scale blocks
    q_region = max(q_region, cell == kNv ? 128 * D / 2 + (D / 64) * 512 * (p.pair_counts || p.pair_table ? 2 : 1)
                                         : (cell == kI8 ? 128 * D : 256 * D));
    slot = max(slot, slot_bytes(D, cell));
  }
  // Prefix tiles run beside video tiles: in the same kernel, so that an SM's CTAs share their code in the
  // instruction cache.
  constexpr int kKernel[8] = {kAny, kNv, kI8, kNvI8, kF16, kNvF16, kI8F16, kAny};
  const int one = kKernel[(p.s.has_nvfp4 != 0) + 2 * (p.s.has_int8 != 0) + 4 * (p.s.has_fp16 != 0)];
  q_region = (q_region + 127) & ~127;
  const int fixed = q_region + factor_sets(one, kQ64) * D * 4 + (int)sizeof(Shared);
  // two CTAs per SM: measured limit is 115,528 bytes of dynamic shared memory per CTA
  const int budget = 115528;
  int ring = ((budget - fixed) / 128) * 128;
  ring = max(ring, 2 * slot);
  ring = min(ring, kRing * slot);
  p.ring_bytes = ring;
  p.q_region = q_region;
  const size_t smem = (size_t)fixed + (size_t)ring;
  switch (one) {
    case kNv: return launch_kernel<D, kNv, kQ64>(p, tiles, smem, st);
    case kI8: return launch_kernel<D, kI8, kQ64>(p, tiles, smem, st);
    case kF16: return launch_kernel<D, kF16, kQ64>(p, tiles, smem, st);
    case kNvI8: return launch_kernel<D, kNvI8, kQ64>(p, tiles, smem, st);
    case kI8F16: return launch_kernel<D, kI8F16, kQ64>(p, tiles, smem, st);
    case kNvF16: return launch_kernel<D, kNvF16, kQ64>(p, tiles, smem, st);
    default: return launch_kernel<D, kAny, kQ64>(p, tiles, smem, st);
  }
}

int launch_for(AttnParams& p, int tiles, cudaStream_t st) {
  if (p.s.query_block == 64)
    return p.s.head_dim == 64 ? launch<64, true>(p, tiles, st) : launch<128, true>(p, tiles, st);
  return p.s.head_dim == 64 ? launch<64, false>(p, tiles, st) : launch<128, false>(p, tiles, st);
}

// ---- dense rows ----
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                 const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encode_tiled() {
  static const EncodeTiled fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult found;
    return cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &found) == cudaSuccess &&
                   found == cudaDriverEntryPointSuccess
               ? reinterpret_cast<EncodeTiled>(f)
               : nullptr;
  }();
  return fn;
}

bool encode(CUtensorMap* map, const void* base, bool bf16, int d, int heads, int tokens, int64_t token_stride,
            int64_t head_stride, int box_tokens) {
  const cuuint64_t dims[3] = {(cuuint64_t)d, (cuuint64_t)heads, (cuuint64_t)tokens};
  const cuuint64_t strides[2] = {(cuuint64_t)head_stride * 2, (cuuint64_t)token_stride * 2};
  const cuuint32_t box[3] = {64, 1, (cuuint32_t)box_tokens}, step[3] = {1, 1, 1};
  return encode_tiled()(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3,
                        const_cast<void*>(base), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Parts of a tile, by the lengths of sequence and prefix alone (a head's rows are then the same whichever heads are with it).
// A part costs some 8 us beside its stages (half a microsecond each, twice that with two CTAs on the SM), so short sequences
// have few.  Alone, one / two / four / eight parts, us: 16 heads x 2,500 tokens, 400 rows 36 / 24 / 26 / 38, 30 x 9,000, 200
// rows 108 / 62 / 53 / 73, 53 x 13,093, 37 rows 153 / 84 / 73 / 83, 7 x 33,272, 512 rows 357 / 186 / 101 / 85.  In a call what
// many heads cost weighs more, and they are behind torch's attention first: more than one tile has at most two parts below
// 256 stages, more than three only one below 96.  FP16 cells of D = 128, us, torch's attention / up to four parts / so:
// 44 heads x 2,592 tokens, 392 rows 143 / 159 / 145, 56 x 2,080, 1,000 rows 171 / 192 / 169, 24 x 3,080, 1,000 rows 124 / 135 /
// 121, 14 x 9,856, 256 rows 353 / 369 / 337, and where few heads want more, 6 x 3,032, 392 rows 119 / 43 / 51.
int dense_parts(int stages, int tiles) {
  if (tiles > 3) return stages < 96 ? 1 : 2;
  const int most = stages < 32 ? 1 : stages < 96 ? 2 : stages < 256 ? 4 : kMostParts;
  return tiles > 1 ? min(most, stages < 256 ? 2 : 4) : most;
}

template <int D, int RAW>
int launch_dense(RawParams& p, cudaStream_t st) {
  auto kernel = attention_kernel<D, kF16, false, RAW>;
  constexpr int kQ = 256 * D, kFixed = kQ + D * 4 + (int)sizeof(Shared);
  constexpr int kRingBytes = (115528 - kFixed) / 128 * 128;
  static_assert(kQ + kRingBytes >= 512 * D + 1024, "a CTA's part takes the place of Q and the ring");
  p.q_region = kQ;
  p.ring_bytes = kRingBytes;
  const size_t smem = kFixed + kRingBytes;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return ANEMOI_SM100_ELAUNCH;
  const int tiles = (p.rows + 127) / 128;
  p.parts = dense_parts(p.stages, tiles);
  for (p.first_place = 0; p.first_place < tiles; p.first_place += 65535) {
    const dim3 grid(p.parts, min(65535, tiles - p.first_place), p.s.heads);
    if (layer::launch_cluster(kernel, grid, dim3(p.parts), dim3(kThreads), smem, st, p) != cudaSuccess)
      return ANEMOI_SM100_ELAUNCH;
  }
  return ANEMOI_SM100_OK;
}

int check_ops(const anemoi_sm100_shape& s, const anemoi_sm100_operands& o, bool dense_prefix) {
  if (s.has_int8 && (!o.q_int8 || !o.kv_int8 || !o.q_int8_scale || !o.k_int8_scale || !o.v_e4m3_scale))
    return ANEMOI_SM100_EINVAL;
  if (dense_prefix) return s.has_int8 ? ANEMOI_SM100_OK : ANEMOI_SM100_EINVAL;
  if (s.has_fp16 && (!o.q_fp16 || !o.kv_fp16)) return ANEMOI_SM100_EINVAL;
  if (s.has_nvfp4 && (!o.q_nvfp4 || !o.kv_nvfp4)) return ANEMOI_SM100_EINVAL;
  return ANEMOI_SM100_OK;
}

uint64_t g_wait_limit_ns = 2000000000ull;

// A one-CTA kernel whose single wait can never be satisfied: nothing arrives on the barrier
// and no copy or MMA is in flight.  It exercises the give-up path of the bounded waits.
__global__ void wait_selftest_kernel(uint64_t limit_ns, int32_t* status) {
  __shared__ uint64_t bar;
  __shared__ WaitContext wc;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    wc.abort = 0;
    wc.status = status;
    wc.limit_ns = limit_ns;
    mbar_init_fence();
  }
  __syncthreads();
  if (threadIdx.x == 0) wait(&wc, &bar, 0, 99);
  __syncthreads();
  // every other thread's wait must now return at once
  if (threadIdx.x != 0) wait(&wc, &bar, 0, 98);
}

}  // namespace

extern "C" int anemoi_sm100_set_wait_limit_ns(uint64_t limit_ns) {
  if (limit_ns == 0) return ANEMOI_SM100_EINVAL;
  g_wait_limit_ns = limit_ns;
  return ANEMOI_SM100_OK;
}

extern "C" int anemoi_sm100_wait_selftest(uint64_t limit_ns, int32_t* status, void* stream) {
  if (limit_ns == 0 || limit_ns > 100000000ull || status == nullptr) return ANEMOI_SM100_EINVAL;
  wait_selftest_kernel<<<1, 64, 0, static_cast<cudaStream_t>(stream)>>>(limit_ns, status);
  return cudaGetLastError() == cudaSuccess ? ANEMOI_SM100_OK : ANEMOI_SM100_ELAUNCH;
}

namespace {
void set_rows(AttnParams& p, const TokenRows* rows) {
  if (rows == nullptr) return;
  p.tokens = rows->out;
  p.tokens_bf16 = p.s.input_is_bf16;
  p.indices = rows->indices;
  p.counts = rows->counts;
}

int video_attention(const anemoi_sm100_shape* shape, const anemoi_sm100_operands* ops,
                    const int32_t* row_offset, const int32_t* row_counts, const int32_t* stage_ids,
                    const int32_t* pair_counts, const int32_t* pair_ids, int64_t list_capacity,
                    const int32_t* valid_k, void* out_packed, const TokenRows* rows, int32_t* status,
                    void* stream, const int32_t* pair_table = nullptr) {
  if (rec::validate_shape(shape) != ANEMOI_SM100_OK || !ops || !row_offset || !row_counts ||
      !valid_k || (!out_packed && !rows) || !status || list_capacity <= 0)
    return ANEMOI_SM100_EINVAL;
  if (check_ops(*shape, *ops, false) != ANEMOI_SM100_OK) return ANEMOI_SM100_EINVAL;
  AttnParams p{};
  p.s = *shape;
  p.o = *ops;
  p.row_offset = row_offset;
  p.row_counts = row_counts;
  p.stage_ids = stage_ids;
  p.pair_counts = pair_counts;
  p.pair_ids = pair_ids;
  p.pair_table = reinterpret_cast<const int4*>(pair_table);
  p.capacity = list_capacity;
  p.valid_k = valid_k;
  p.out = static_cast<__half*>(out_packed);
  p.status = status;
  p.wait_ns = g_wait_limit_ns;
  p.dense_prefix = 0;
  p.stages = rec::stages(*shape);
  p.q_tiles_int8 = shape->video_blocks + rec::prefix_query_tiles(*shape);
  p.out_rows = shape->video_blocks * shape->query_block;
  set_rows(p, rows);
  const int tiles = pair_counts || pair_table ? (shape->video_blocks + 1) / 2 : shape->video_blocks;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return launch_for(p, tiles, st);
}
}  // namespace

extern "C" int anemoi_sm100_attention(const anemoi_sm100_shape* shape,
                                      const anemoi_sm100_operands* ops, const int32_t* row_offset,
                                      const int32_t* row_counts, const int32_t* stage_ids,
                                      int64_t list_capacity, const int32_t* valid_k,
                                      void* out_packed, int32_t* status, void* stream) {
  if (!stage_ids) return ANEMOI_SM100_EINVAL;
  return video_attention(shape, ops, row_offset, row_counts, stage_ids, nullptr, nullptr,
                         list_capacity, valid_k, out_packed, nullptr, status, stream);
}

extern "C" int anemoi_sm100_head_groups(const anemoi_sm100_shape* shape, int pairs) {
  if (rec::validate_shape(shape) != ANEMOI_SM100_OK) return 0;
  AttnParams p{};
  p.s = *shape;
  p.stages = rec::stages(*shape);
  const int R = shape->video_blocks, tiles = pairs && shape->query_block == 64 ? (R + 1) / 2 : R;
  return head_groups(p, (int64_t)tiles * shape->heads);
}

extern "C" int anemoi_sm100_attention_pairs(const anemoi_sm100_shape* shape,
                                            const anemoi_sm100_operands* ops,
                                            const int32_t* row_offset, const int32_t* row_counts,
                                            const int32_t* pair_counts, const int32_t* pair_ids,
                                            int64_t list_capacity, const int32_t* valid_k,
                                            void* out_packed, int32_t* status, void* stream) {
  if (!pair_counts || !pair_ids || !shape || shape->query_block != 64) return ANEMOI_SM100_EINVAL;
  return video_attention(shape, ops, row_offset, row_counts, nullptr, pair_counts, pair_ids,
                         list_capacity, valid_k, out_packed, nullptr, status, stream);
}

extern "C" int anemoi_sm100_attention_matched(const anemoi_sm100_shape* shape, const anemoi_sm100_operands* ops,
                                              const int32_t* row_offset, const int32_t* row_counts,
                                              const int32_t* pair_table, const int32_t* pair_ids, int64_t list_capacity,
                                              const int32_t* valid_k, void* out_packed, int32_t* status, void* stream) {
  if (!pair_table || reinterpret_cast<uintptr_t>(pair_table) % 16 || !pair_ids || !shape || shape->query_block != 64)
    return ANEMOI_SM100_EINVAL;
  return video_attention(shape, ops, row_offset, row_counts, nullptr, nullptr, pair_ids, list_capacity, valid_k, out_packed,
                         nullptr, status, stream, pair_table);
}

namespace {
int prefix_attention(const anemoi_sm100_shape* shape, const anemoi_sm100_operands* ops, const int32_t* valid_k,
                     void* out_prefix, const TokenRows* rows, int32_t* status, void* stream) {
  if (rec::validate_shape(shape) != ANEMOI_SM100_OK || !ops || !valid_k || (!out_prefix && !rows) || !status)
    return ANEMOI_SM100_EINVAL;
  if (!shape->has_prefix_query_int8 || shape->prefix_tokens == 0) return ANEMOI_SM100_EINVAL;
  if (check_ops(*shape, *ops, true) != ANEMOI_SM100_OK) return ANEMOI_SM100_EINVAL;
  AttnParams p{};
  p.s = *shape;
  p.o = *ops;
  p.valid_k = valid_k;
  p.out = static_cast<__half*>(out_prefix);
  p.status = status;
  p.wait_ns = g_wait_limit_ns;
  p.dense_prefix = 1;
  p.stages = rec::stages(*shape);
  const int blocks = rec::prefix_query_tiles(*shape);
  const int tiles = shape->query_block == 64 ? (blocks + 1) / 2 : blocks;
  p.prefix_tiles = blocks;
  p.q_tiles_int8 = shape->video_blocks + blocks;
  p.out_rows = blocks * shape->query_block;
  set_rows(p, rows);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return launch_for(p, tiles, st);
}
}  // namespace

extern "C" int anemoi_sm100_dense_parts(int tokens, int rows) {
  return rows > 0 && tokens >= rows ? dense_parts((tokens + 63) / 64, (rows + 127) / 128) : ANEMOI_SM100_EINVAL;
}

extern "C" int anemoi_sm100_dense_rows(int heads, int head_dim, int tokens, int rows, int is_bf16, const void* q,
                                       const void* k, const void* v, const int64_t* strides, void* out, int64_t out_token,
                                       int64_t out_head, int32_t* status, void* stream) {
  if (heads <= 0 || heads > 65535 || (head_dim != 64 && head_dim != 128) || rows <= 0 || tokens < rows || !q || !k || !v ||
      !out || !status)
    return ANEMOI_SM100_EINVAL;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
       reinterpret_cast<uintptr_t>(out)) % 16 || out_token % 8 || out_head % 8)
    return ANEMOI_SM100_EINVAL;
  int64_t stride[6];
  for (int i = 0; i < 6; ++i) {
    const int64_t packed = i & 1 ? (int64_t)head_dim : (int64_t)heads * head_dim;
    stride[i] = strides == nullptr || (heads == 1 && i & 1) ? packed : strides[i];
    // (what a tensor map takes)
    if (stride[i] <= 0 || stride[i] % 8 || stride[i] >= (1ll << 39)) return ANEMOI_SM100_EINVAL;
  }
  if (encode_tiled() == nullptr) return ANEMOI_SM100_ELAUNCH;
  RawParams p{};
  if (!encode(&p.q, q, is_bf16, head_dim, heads, tokens, stride[0], stride[1], 128) ||
      !encode(&p.k, k, is_bf16, head_dim, heads, tokens, stride[2], stride[3], 64) ||
      !encode(&p.v, v, is_bf16, head_dim, heads, tokens, stride[4], stride[5], 64))
    return ANEMOI_SM100_EINVAL;
  p.s.heads = heads;
  p.s.head_dim = head_dim;
  p.s.video_blocks = 1;
  p.rows = rows;
  p.tokens_in = tokens;
  p.stages = (tokens + 63) / 64;
  p.tokens = out;
  p.out_token = out_token;
  p.out_head = out_head;
  p.status = status;
  p.wait_ns = g_wait_limit_ns;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (head_dim == 64) return is_bf16 ? launch_dense<64, kRawBf16>(p, st) : launch_dense<64, kRawF16>(p, st);
  return is_bf16 ? launch_dense<128, kRawBf16>(p, st) : launch_dense<128, kRawF16>(p, st);
}

extern "C" int anemoi_sm100_prefix_attention(const anemoi_sm100_shape* shape,
                                             const anemoi_sm100_operands* ops,
                                             const int32_t* valid_k, void* out_prefix,
                                             int32_t* status, void* stream) {
  return prefix_attention(shape, ops, valid_k, out_prefix, nullptr, status, stream);
}

namespace layer {

int video_rows(const anemoi_sm100_shape& s, const anemoi_sm100_operands& ops, const int32_t* row_offset,
               const int32_t* row_counts, const int32_t* stage_ids, const int32_t* pair_counts,
               const int32_t* pair_ids, int64_t capacity, const int32_t* valid_k, const TokenRows& rows,
               int32_t* status, cudaStream_t st, const int32_t* pair_table) {
  return video_attention(&s, &ops, row_offset, row_counts, stage_ids, pair_counts, pair_ids, capacity, valid_k,
                         nullptr, &rows, status, st, pair_table);
}

uint64_t wait_limit_ns() { return g_wait_limit_ns; }

int prefix_rows(const anemoi_sm100_shape& s, const anemoi_sm100_operands& ops, const int32_t* valid_k,
                const TokenRows& rows, int32_t* status, cudaStream_t st) {
  return prefix_attention(&s, &ops, valid_k, nullptr, &rows, status, st);
}

}  // namespace layer
