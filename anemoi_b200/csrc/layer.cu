// One anemoi_attention call in one entry point: operands, draft map, routing, video attention and
// prefix attention, with the results written straight to their tokens.
//
// A small call is bound by its launches, not by its kernels: with one Python wrapper, allocation and
// marshaling per stage the 1,024-token call takes 210 us, here 19.5 (host work and kernels are about as
// long, call behind call).  The host work is one function: one workspace cut up by offsets, three to twelve kernels
// (up to eight where routing is one, which it is for most shapes, forming the draft map of short calls, too; the output
// needs no assembly pass), programmatic dependent launches between them.
//
// Order of the launches.  The prefix rows' tiles walk every stage of the head: few CTAs, each as
// long as the whole video launch of a small call, so they start on the side stream as soon as the
// operands are there and run beside draft and routing.  When there is one for every SM they start after
// routing, in front of the video tiles: a CTA holds half of an SM for up to milliseconds, and the routing
// kernel needs a whole one's shared memory.  Where they leave routing few SMs the two orders are close; early /
// late, D = 128, a 1,000-token prefix (eight tiles per head): 18 heads (144 tiles) with 7,800 video tokens 400 /
// 419 us, 32,760 tokens 3.09 / 3.11 ms, 84,672 tokens 15.11 / 14.99 ms; 12 heads of the latter 10.05 / 10.01; past
// the line, 24 heads (192 tiles), 526 / 550 us and 20.02 / 19.94 ms.  With few tiles early is the quicker one (8
// heads, 16 tiles, 7,800 tokens: 183 / 221 us).
#include <cuda_runtime.h>

#include "layer.cuh"
#include "records.cuh"

namespace {

constexpr int64_t kAlign = 256;
constexpr int kMatchMaxBlocks = 4096;
constexpr int kPrefixFillsGpu = 148;  // prefix CTAs from which they start after routing: one per SM

int64_t up(int64_t n) { return (n + kAlign - 1) / kAlign * kAlign; }

struct Workspace {
  anemoi_sm100_operands ops;
  uint8_t* prob;
  int32_t *row_offset, *row_counts, *stage_ids, *pair_counts, *pair_ids;
  int32_t* pair_table;  // pairs chosen by what their lists share; null: neighbours
  layer::PairBits pair_bits;
  uint8_t* scratch;
  int64_t scratch_bytes, bytes;
};

// Whether the Q64 pairs are chosen by what their lists share (match.cu) rather than by index: where that many
// stages, the blocks' lists summed, are walked that the choice, some 10 us between routing and attention, pays even for
// inputs in which no blocks attend alike.  Index / chosen, us, 80 % dropped and 200 tokens of prefix, such inputs and ones with
// two loud channels:  INT8, D = 128, 4 heads x 225 blocks (44,100 stages) 187 / 196, 211 / 195; 8 x 225 (88,200) 304 / 304,
// 324 / 286; 8 x 525 (457,800) 1,181 / 1,171, 1,218 / 1,005.  NVFP4, D = 64, 5 x 247 (61,010) 186 / 190, 191 / 171;
// 8 x 225 236 / 235, 242 / 212.  Several cells, whose lists share less (a column in the same cell), D = 64:  8 x 225 362 /
// 369, 370 / 340; 16 x 225 (176,400) 644 / 647, 663 / 587; 8 x 525 1,351 / 1,348, 1,376 / 1,175.
constexpr int64_t kMatchStages = 80000, kMatchStagesMixed = 160000;
bool matches(const anemoi_sm100_layer_plan& p) {
  const int R = p.shape.video_blocks;
  const int64_t stages = p.shape.heads * (p.n16 + p.n8 + p.n4 + (int64_t)R * rec::prefix_stages(p.shape));
  const int cells = (p.n16 > 0) + (p.n8 > 0) + (p.n4 > 0);
  return R > 32 && R <= kMatchMaxBlocks && rec::stages(p.shape) < (1 << 30) &&
         stages >= (cells > 1 ? kMatchStagesMixed : kMatchStages);
}

layer::PairBits pair_bits(const anemoi_sm100_layer_plan& p, uint32_t* words) {
  const int64_t budget[3] = {p.n4, p.n8, p.n16};
  layer::PairBits bits = {words, 0, {}};
  for (int c = 0; c < 3; ++c) bits.slot[c] = budget[c] > 0 ? bits.phases++ : -1;
  return bits;
}
int64_t pair_bits_bytes(const anemoi_sm100_layer_plan& p) {
  const int64_t H = p.shape.heads, R = p.shape.video_blocks;
  return H * pair_bits(p, nullptr).phases * R * layer::pair_bit_words(R) * 4;
}

// Routing and the chosen pairs' lists.
int route_matched(const anemoi_sm100_layer_plan& p, const void* probability, void* scratch, int32_t* row_offset,
                  int32_t* row_counts, const layer::PairBits& bits, int32_t* table, int32_t* pair_ids, cudaStream_t st) {
  const anemoi_sm100_shape& s = p.shape;
  const int phase = s.prefix_tokens > 0 || p.prefix_phase < 0 || p.prefix_phase > 2 ? p.prefix_phase : -1;
  const int code = layer::route_bits(s, probability, p.n16, p.n8, p.n4, phase, scratch, row_offset, row_counts, bits,
                                     p.list_capacity, st);
  return code != ANEMOI_SM100_OK ? code
                                 : layer::match_pairs(s, bits, phase, row_offset, row_counts, table, pair_ids,
                                                      p.list_capacity, p.status, st);
}

// Cuts `base` (null: only the size is wanted) into the call's buffers.
Workspace cut(const anemoi_sm100_layer_plan& p, uint8_t* base) {
  const anemoi_sm100_shape& s = p.shape;
  const int64_t H = s.heads, R = s.video_blocks;
  Workspace w = {};
  int64_t at = 0;
  auto take = [&](int64_t n) -> uint8_t* {
    uint8_t* ptr = n > 0 && base != nullptr ? base + at : nullptr;
    at += up(n);
    return ptr;
  };
  auto operand = [&](int which) { return take(anemoi_sm100_operand_bytes(&s, which)); };
  w.ops.v_amax = reinterpret_cast<float*>(operand(ANEMOI_SM100_BUF_V_AMAX));
  w.ops.q_fp16 = operand(ANEMOI_SM100_BUF_Q_FP16);
  w.ops.kv_fp16 = operand(ANEMOI_SM100_BUF_KV_FP16);
  w.ops.q_int8 = operand(ANEMOI_SM100_BUF_Q_INT8);
  w.ops.kv_int8 = operand(ANEMOI_SM100_BUF_KV_INT8);
  w.ops.q_nvfp4 = operand(ANEMOI_SM100_BUF_Q_NVFP4);
  w.ops.kv_nvfp4 = operand(ANEMOI_SM100_BUF_KV_NVFP4);
  w.ops.q_int8_scale = reinterpret_cast<float*>(operand(ANEMOI_SM100_BUF_Q_INT8_SCALE));
  w.ops.k_int8_scale = reinterpret_cast<float*>(operand(ANEMOI_SM100_BUF_K_INT8_SCALE));
  w.ops.v_e4m3_scale = reinterpret_cast<float*>(operand(ANEMOI_SM100_BUF_V_E4M3_SCALE));
  w.ops.q_pool = operand(ANEMOI_SM100_BUF_POOL);
  w.ops.k_pool = operand(ANEMOI_SM100_BUF_POOL);
  if (s.has_maxpool) {
    w.ops.q_max_pool = operand(ANEMOI_SM100_BUF_POOL);
    w.ops.k_max_pool = operand(ANEMOI_SM100_BUF_POOL);
  }
  const bool pairs = p.pair_q64 && s.query_block == 64, matched = pairs && matches(p);
  w.prob = take(H * R * R * 2);
  w.row_offset = reinterpret_cast<int32_t*>(take(H * R * 4));
  w.row_counts = reinterpret_cast<int32_t*>(take(H * R * 16));
  const bool fused = pairs && layer::routes_pairs(s);
  const int64_t list = H * p.list_capacity * 4;
  // (routed in one kernel, the pairs need neither the blocks' own lists nor scratch)
  if (!fused && !matched) w.stage_ids = reinterpret_cast<int32_t*>(take(list));
  if (matched) {
    w.pair_bits = pair_bits(p, reinterpret_cast<uint32_t*>(take(pair_bits_bytes(p))));
    w.pair_table = reinterpret_cast<int32_t*>(take(H * ((R + 1) / 2) * 32));
  } else if (pairs) {
    w.pair_counts = reinterpret_cast<int32_t*>(take(H * ((R + 1) / 2) * 16));
  }
  if (pairs) {
    w.pair_ids = reinterpret_cast<int32_t*>(take(list));
  }
  w.scratch_bytes = fused ? 0 : anemoi_sm100_route_scratch_bytes(&s);
  w.scratch = take(w.scratch_bytes);
  w.bytes = at;
  return w;
}

bool valid(const anemoi_sm100_layer_plan* p) {
  return p != nullptr && rec::validate_shape(&p->shape) == ANEMOI_SM100_OK && p->indices && p->counts &&
         p->valid_k && p->status && p->shape.has_maxpool != 2 && p->list_capacity > 0;
}

}  // namespace

extern "C" int anemoi_sm100_stream_create(void** stream) {
  return stream == nullptr ? ANEMOI_SM100_EINVAL
         : cudaStreamCreateWithFlags(reinterpret_cast<cudaStream_t*>(stream), cudaStreamNonBlocking) == cudaSuccess
             ? ANEMOI_SM100_OK
             : ANEMOI_SM100_ELAUNCH;
}

extern "C" int anemoi_sm100_routes_in_one_kernel(const anemoi_sm100_shape* shape) {
  return rec::validate_shape(shape) == ANEMOI_SM100_OK && layer::routes_pairs(*shape);
}

extern "C" int anemoi_sm100_drafts_in_routing(const anemoi_sm100_shape* shape) {
  return rec::validate_shape(shape) == ANEMOI_SM100_OK && layer::drafts_in_routing(*shape);
}

extern "C" int anemoi_sm100_matches_pairs(const anemoi_sm100_layer_plan* plan) {
  return valid(plan) && plan->pair_q64 && plan->shape.query_block == 64 && matches(*plan);
}

extern "C" int64_t anemoi_sm100_pair_bits_bytes(const anemoi_sm100_layer_plan* plan) {
  return anemoi_sm100_matches_pairs(plan) ? pair_bits_bytes(*plan) : ANEMOI_SM100_EINVAL;
}

extern "C" int anemoi_sm100_route_matched(const anemoi_sm100_layer_plan* plan, const void* probability, void* scratch,
                                          int64_t scratch_bytes, int32_t* row_offset, int32_t* row_counts, void* bits,
                                          int32_t* pair_table, int32_t* pair_ids, void* stream) {
  if (!anemoi_sm100_matches_pairs(plan) || !probability || !row_offset || !row_counts || !bits || !pair_table || !pair_ids)
    return ANEMOI_SM100_EINVAL;
  // (read 16 bytes at a time)
  if ((reinterpret_cast<uintptr_t>(row_counts) | reinterpret_cast<uintptr_t>(bits) |
       reinterpret_cast<uintptr_t>(pair_table)) % 16)
    return ANEMOI_SM100_EINVAL;
  if (!scratch || scratch_bytes < anemoi_sm100_route_scratch_bytes(&plan->shape)) return ANEMOI_SM100_EINVAL;
  return route_matched(*plan, probability, scratch, row_offset, row_counts,
                       pair_bits(*plan, static_cast<uint32_t*>(bits)), pair_table, pair_ids,
                       static_cast<cudaStream_t>(stream));
}

extern "C" int64_t anemoi_sm100_layer_workspace_bytes(const anemoi_sm100_layer_plan* plan) {
  return valid(plan) ? cut(*plan, nullptr).bytes : ANEMOI_SM100_EINVAL;
}

extern "C" int anemoi_sm100_layer(const anemoi_sm100_layer_plan* plan, const void* q, const void* k, const void* v,
                                  const int64_t* strides, const float* nvfp4_scales, const void* prefix_out,
                                  int64_t prefix_rows, int prefix_is_caller_dtype, void* out, void* workspace,
                                  int64_t workspace_bytes, void* stream, void* side_stream) {
  if (!valid(plan) || !q || !k || !v || !out || !workspace) return ANEMOI_SM100_EINVAL;
  anemoi_sm100_layer_plan p = *plan;
  anemoi_sm100_shape& s = p.shape;
  if (nvfp4_scales != nullptr) {
    s.q_global_scale = nvfp4_scales[0];
    s.k_global_scale = nvfp4_scales[1];
    s.v_global_scale = nvfp4_scales[2];
    if (rec::validate_shape(&s) != ANEMOI_SM100_OK) return ANEMOI_SM100_EINVAL;
  }
  const bool native_prefix = s.has_prefix_query_int8 && s.prefix_tokens > 0;
  const bool dense_prefix = s.prefix_tokens > 0 && !native_prefix && prefix_out == nullptr &&
                            prefix_is_caller_dtype == ANEMOI_SM100_PREFIX_DENSE;
  if (s.prefix_tokens > 0 && !native_prefix && !dense_prefix && prefix_out == nullptr) return ANEMOI_SM100_EINVAL;
  if (s.prefix_tokens > 0 && side_stream == nullptr) return ANEMOI_SM100_EINVAL;
  const Workspace w = cut(p, static_cast<uint8_t*>(workspace));
  if (workspace_bytes < w.bytes) return ANEMOI_SM100_EINVAL;
  cudaStream_t st = static_cast<cudaStream_t>(stream), side = static_cast<cudaStream_t>(side_stream);
  const layer::TokenRows rows{out, p.indices, p.counts};

  // fork and join of the side stream: an event each, destroyed when its use is over
  cudaEvent_t fork = nullptr, join = nullptr;
  auto done = [&](int c) {
    if (c != ANEMOI_SM100_OK && fork != nullptr && join == nullptr &&
        cudaEventCreateWithFlags(&join, cudaEventDisableTiming) == cudaSuccess &&
        cudaEventRecord(join, side) == cudaSuccess)
      cudaStreamWaitEvent(st, join, 0);  // the workspace is not free before the side stream is done with it
    if (fork) cudaEventDestroy(fork);
    if (join) cudaEventDestroy(join);
    return c;
  };
  auto to_side = [&]() {
    return cudaEventCreateWithFlags(&fork, cudaEventDisableTiming) == cudaSuccess &&
           cudaEventRecord(fork, st) == cudaSuccess && cudaStreamWaitEvent(side, fork, 0) == cudaSuccess;
  };
  auto prefix = [&]() -> int {
    return to_side() ? layer::prefix_rows(s, w.ops, p.valid_k, rows, p.status, side) : ANEMOI_SM100_ELAUNCH;
  };
  // (dense rows need the caller's tensors only)
  if (dense_prefix && !to_side()) return done(ANEMOI_SM100_ELAUNCH);
  int code = anemoi_sm100_prepare(&s, q, k, v, strides, p.indices, p.counts, &w.ops, stream);
  if (code == ANEMOI_SM100_OK && dense_prefix)
    code = anemoi_sm100_dense_rows(s.heads, s.head_dim, s.seq_tokens, s.prefix_tokens, s.input_is_bf16, q, k, v, strides, out,
                                   (int64_t)s.heads * s.head_dim, s.head_dim, p.status, side_stream);
  if (code != ANEMOI_SM100_OK) return done(code);
  const int prefix_ctas = (rec::prefix_query_tiles(s) * s.query_block + 127) / 128 * s.heads;
  const bool late = native_prefix && prefix_ctas >= kPrefixFillsGpu;
  if (native_prefix && !late && (code = prefix()) != ANEMOI_SM100_OK) return done(code);

  const int32_t* pair_counts = w.pair_counts;
  if (layer::drafts_in_routing(s)) {
    code = layer::draft_and_route(s, w.ops, p.maxpool_weight, w.prob, p.n16, p.n8, p.n4, p.prefix_phase, w.row_offset,
                                  w.row_counts, w.stage_ids, w.pair_counts, w.pair_ids, p.list_capacity, st);
  } else {
    code = anemoi_sm100_draft_probability(&s, w.ops.q_pool, w.ops.k_pool, w.ops.q_max_pool, w.ops.k_max_pool,
                                          p.maxpool_weight, w.prob, stream);
    if (code != ANEMOI_SM100_OK) return done(code);
    if (w.pair_table != nullptr) {
      code = route_matched(p, w.prob, w.scratch, w.row_offset, w.row_counts, w.pair_bits, w.pair_table, w.pair_ids, st);
    } else if (pair_counts != nullptr && layer::routes_pairs(s)) {
      code = anemoi_sm100_route_pairs(&s, w.prob, p.n16, p.n8, p.n4, p.prefix_phase, w.row_offset, w.row_counts,
                                      w.pair_counts, w.pair_ids, p.list_capacity, stream);
    } else {
      code = anemoi_sm100_route(&s, w.prob, p.n16, p.n8, p.n4, p.prefix_phase, w.scratch, w.scratch_bytes,
                                w.row_offset, w.row_counts, w.stage_ids, p.list_capacity, stream);
      if (code == ANEMOI_SM100_OK && pair_counts != nullptr)
        code = anemoi_sm100_pair_lists(&s, w.row_offset, w.row_counts, w.stage_ids, p.list_capacity, w.pair_counts,
                                       w.pair_ids, stream);
    }
  }
  if (code != ANEMOI_SM100_OK) return done(code);
  if (late && (code = prefix()) != ANEMOI_SM100_OK) return done(code);
  code = layer::video_rows(s, w.ops, w.row_offset, w.row_counts, w.stage_ids, pair_counts, w.pair_ids,
                           p.list_capacity, p.valid_k, rows, p.status, st, w.pair_table);
  if (code != ANEMOI_SM100_OK) return done(code);
  if (s.prefix_tokens > 0) {
    if (cudaEventCreateWithFlags(&join, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventRecord(join, side) != cudaSuccess || cudaStreamWaitEvent(st, join, 0) != cudaSuccess)
      return done(ANEMOI_SM100_ELAUNCH);
    if (!native_prefix && !dense_prefix)
      code = layer::assemble_prefix(s, prefix_out, prefix_rows, prefix_is_caller_dtype, out, st);
  }
  return done(code);
}
