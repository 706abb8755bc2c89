// Which two Q64 query blocks share a CTA of the attention kernel, and the lists of those pairs.
//
// Two blocks of a head fill the 128 rows of the MMA shape and walk the union of their lists, so a CTA's time
// goes with the union: a stage that only one block needs takes about as long as one that both need.
// Neighbours by index (2t and 2t + 1) share little where blocks that attend alike lie apart.
//
// One kernel behind the routing, which leaves a bit per (block, phase, column).  A CTA takes up to 128 blocks of
// a head and
//   counts the columns that every two of them share, phase by phase: the product of a 0/1 matrix
//   [blocks x columns] with its transpose, on the tensor core (exact);
//   chooses the pairs: the block with the longest list first, with the free block it shares most columns with;
//   writes the pairs' lists.
// A choice among 128 is nearly as good as one among all of a head's blocks, which takes several launches and a
// chain of steps as long as the head: on smooth fields with two loud channels (56 heads x 592 blocks, 80 % dropped)
// unions of neighbours are 0.838 of the lists' sum, of these pairs 0.577, of pairs out of all blocks 0.557 (0.5 is
// the least possible); without loud channels (three cells, 247 blocks) 0.933, 0.899 and 0.891.
//
// Bound by latency: of some 10 us for 225 blocks of 4 heads 5.5 are the choice (one warp, 64 steps of 180 cycles,
// a reduction and what hangs on it), 3 the lists, whose integer operations are the rest.  The 592-block call above,
// INT8, D = 128: 11.58 -> 9.36 ms; 225 blocks of 16 heads, FP16: 0.732 -> 0.602 ms.
#include <algorithm>

#include "bounded_wait.cuh"
#include "layer.cuh"
#include "records.cuh"
#include "sm100_primitives.cuh"

namespace {

using namespace sm100;

constexpr int kGroup = 128;                 // blocks of a CTA
constexpr int kParts = 8;                   // threads per block of the group
constexpr int kThreads = kParts * kGroup;
constexpr int kWarps = kThreads / 32;
constexpr int kRing = 4;                    // pieces of 128 columns in shared memory at a time
constexpr int kPieceBytes = kGroup * 128;   // a byte per column
constexpr int kShareRow = kGroup + 4;       // words per row of the table of shares (16-byte rows, shifted by a bank group)

struct MatchShared {
  uint64_t done;  // MMAs that read the ring
  WaitContext wc;
  uint32_t tmem_base;
  alignas(16) int key[kGroup];  // longer blocks, of those earlier ones, have larger keys
  int below[kGroup];            // how many keys are smaller
  int block[kGroup];      // by place in the order: the block, and its stages
  int stages[kGroup];
  uint2 pairs[kGroup / 2];  // first block's place, its best entry (0: a block alone)
};

__host__ __device__ inline int groups(int R) { return (R + kGroup - 1) / kGroup; }
// Blocks of every group but the last: even, so that no group but the last leaves a block alone.
__host__ __device__ inline int group_blocks(int R) { return ((R + groups(R) - 1) / groups(R) + 1) & ~1; }

// Four bits -> four bytes 0 or 1, the lowest bit in the lowest byte.
__device__ __forceinline__ uint32_t bytes_of(uint32_t nibble) { return (nibble * 0x00204081u) & 0x01010101u; }

__global__ void __launch_bounds__(kThreads) match_kernel(const uint32_t* bits, int R, int words, int phases, int3 slot,
                                                         const int32_t* row_offset, const int32_t* row_counts,
                                                         int prefix_stages, int prefix_phase, int64_t capacity,
                                                         int4* table, int32_t* pair_ids, int32_t* status,
                                                         uint64_t wait_ns) {
  extern __shared__ __align__(128) uint8_t smem[];
  MatchShared& sh = *reinterpret_cast<MatchShared*>(smem + max(kRing * kPieceBytes, kGroup * kShareRow * 4));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, head = blockIdx.y, group = blockIdx.x;
  const int per = group_blocks(R), first = group * per, count = min(per, R - first);
  if (threadIdx.x == 0) {
    mbar_init(&sh.done, 1);
    sh.wc.abort = 0;
    sh.wc.status = status;
    sh.wc.limit_ns = wait_ns;
    mbar_init_fence();
  }
  if (warp == 0) {
    tmem_alloc(&sh.tmem_base, kGroup);
    tmem_relinquish();
  }
  layer::grid_dependency_wait();
  layer::grid_dependency_trigger();

  // ---- the group's blocks by length, the longest at the last place; a thread has an eighth of a block's piece ----
  const int block = threadIdx.x & (kGroup - 1), part = threadIdx.x / kGroup;
  const bool real = block < count;
  const int row_pieces = words / 4, pieces = phases * row_pieces;
  // (phases lie [phase][row][words]: the next piece, and the end of the row that it is in)
  const uint16_t* src = reinterpret_cast<const uint16_t*>(bits + ((int64_t)head * phases * R + first + block) * words) + part;
  const uint16_t* row_end = src + 2 * words;
  int unread = pieces;
  const auto piece = [&]() -> uint32_t {
    if (!real || unread-- <= 0) return 0;
    const uint32_t v = __ldg(src);
    src += 8;
    if (src == row_end) {
      src += (int64_t)(R - 1) * 2 * words;
      row_end = src + 2 * words;
    }
    return v;
  };
  uint32_t next[kRing];
#pragma unroll
  for (int u = 0; u < kRing; ++u) next[u] = piece();
  int length = -1;
  if (real) {
    const int4 c = *reinterpret_cast<const int4*>(row_counts + ((int64_t)head * R + first + block) * 4);
    length = c.x + c.y + c.z;
  }
  const int key = length * kGroup + kGroup - 1 - block;  // (lengths below 2^24)
  if (part == 0) {
    sh.key[block] = key;
    sh.below[block] = 0;
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = sh.tmem_base, base = smem_u32(smem);
  int smaller = 0;
#pragma unroll
  for (int j = 0; j < kGroup / kParts; j += 4) {
    const int4 k = *reinterpret_cast<const int4*>(&sh.key[part * (kGroup / kParts) + j]);
    smaller += (k.x < key) + (k.y < key) + (k.z < key) + (k.w < key);
  }
  atomicAdd(&sh.below[block], smaller);
  __syncthreads();
  const int place = sh.below[block];
  if (part == 0) {
    sh.block[place] = first + block;
    sh.stages[place] = length;
  }

  // ---- shares: 128 columns at a time become bytes, and operand of the tensor core for both sides ----
  constexpr uint32_t idesc = instr_desc(kFmtS8, kFmtS8, kAccS32, kGroup, kGroup, 0, 0);
  // (a ring at a time: the fence and the barrier between writing and reading it cost more than the writing)
  for (int k0 = 0; k0 < pieces; k0 += kRing) {
    if (k0 > 0) wait(&sh.wc, &sh.done, (k0 / kRing - 1) & 1, 41);
#pragma unroll
    for (int at = 0; at < kRing; ++at) {
      const uint32_t now = next[at];
      next[at] = piece();
      *reinterpret_cast<uint4*>(smem + at * kPieceBytes + rec::tile_offset(place, part, 8)) =
          make_uint4(bytes_of(now & 15), bytes_of((now >> 4) & 15), bytes_of((now >> 8) & 15), bytes_of(now >> 12));
    }
    fence_proxy_async_smem();
    __syncthreads();
    if (threadIdx.x == 0) {
      tc_fence_after_sync();
      for (int at = 0; at < min(kRing, pieces - k0); ++at) {
        const uint64_t d = smem_desc(base + at * kPieceBytes, 128, 8 * 128);
#pragma unroll
        for (int s = 0; s < 4; ++s) mma_i8_ss(tmem, d + s * 16, d + s * 16, idesc, (k0 | at | s) != 0);
      }
      mma_commit(&sh.done);
    }
    __syncwarp();
  }
  const uint32_t last = ((pieces + kRing - 1) / kRing - 1) & 1;
  wait(&sh.wc, &sh.done, last, 42);
  // unwinding: the MMAs in flight must be over before tensor memory is given back
  if (sh.wc.abort) drain_wait(&sh.done, last, 100000000);
  tc_fence_after_sync();
  // Entry: one above the share, then the column (7 bits): the largest is the block with the largest share, of those the
  // longest.  Only left of the diagonal: the blocks to the right, which are longer, have their partners by then.
  uint32_t* share = reinterpret_cast<uint32_t*>(smem);
  {
    const int r = (warp & 3) * 32 + lane, c0 = (warp >> 2) * (kGroup / kParts);
    uint32_t v[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(tmem + ((uint32_t)((warp & 3) * 32) << 16) + c0)
        : "memory");
    tmem_wait_ld();
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = c0 + j < r ? v[j] * kGroup + (uint32_t)(kGroup + c0 + j) : 0;
#pragma unroll
    for (int j = 0; j < 16; j += 4)
      *reinterpret_cast<uint4*>(share + r * kShareRow + c0 + j) = make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]);
  }
  tc_fence_before_sync();
  __syncthreads();

  // ---- pairs, longest first: one warp, four columns per lane ----
  const int pairs = (count + 1) / 2;
  if (warp == 0) {
    // A lane's columns 4 lane .. + 3 (~0: free), and, in lane w, the free ones of places 32 w .. + 31
    uint32_t open[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) open[c] = 4 * lane + c >= kGroup - count ? 0xffffffffu : 0;
    const int none = kGroup - count - 32 * lane;  // places of this word that no block has
    uint32_t mine = none <= 0 ? 0xffffffffu : none < 32 ? 0xffffffffu << none : 0;
    const auto row = [&](int r) { return *reinterpret_cast<const uint4*>(share + r * kShareRow + 4 * lane); };
    uint2* out = sh.pairs;
#pragma unroll 1
    for (int w = kGroup / 32 - 1; w >= 0; --w) {
      uint32_t left = __shfl_sync(0xffffffffu, mine, w);
      int a = -1;
      uint4 v = make_uint4(0, 0, 0, 0);
      while (a >= 0 || left) {
        if (a < 0) {
          const int n = 31 - __clz(left);
          a = w * 32 + n;
          v = row(a);
          left &= ~(1u << n);
        }
        // (the next block's row is read under the reduction, before it is known that this block does not take it)
        const int n = 31 - __clz(left), next = w * 32 + n;
        const uint4 ahead = row(max(next, 0));
        const uint32_t best = __reduce_max_sync(
            0xffffffffu, max(max(v.x & open[0], v.y & open[1]), max(v.z & open[2], v.w & open[3])));
        if (lane == 0) *out = make_uint2(a, best);
        ++out;
        const int b = best & (kGroup - 1);
        const uint32_t others = ~(1u << (b & 31));
        if (lane == b >> 5) mine &= others;
        if (w == b >> 5) left &= others;
        a = -1;
        if (n >= 0 && next != b) {
          a = next;
          left &= ~(1u << n);
        }
        v = ahead;
#pragma unroll
        for (int c = 0; c < 4; ++c) open[c] = b == 4 * lane + c ? 0 : open[c];
      }
    }
  }
  __syncthreads();

  // ---- lists: one warp per pair, a lane per word of a phase; per phase the columns of either block, ascending, with
  // a bit per block, the prefix stages in front of the phase that carries them.  The group's lists follow one another
  // from where those of its blocks would start.  Launch order: the first pairs of all groups, then the second ones, ...
  const unsigned lower = (1u << lane) - 1u;
  const int all = groups(R), in_last = (R - (all - 1) * per + 1) / 2;
  const int64_t start = row_offset[(int64_t)head * R + first];
  const bool gave_up = sh.wc.abort != 0;  // (the shares are not valid, nor is the call's result: empty lists)
  int sum[2], size[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int t = h * 32 + lane;
    const uint2 two = t < pairs ? sh.pairs[t] : make_uint2(0, 0);
    size[h] = t < pairs ? sh.stages[two.x] : 0;
    if (two.y)
      size[h] += sh.stages[two.y & (kGroup - 1)] - (int)(two.y / kGroup - 1) - (prefix_phase >= 0 ? prefix_stages : 0);
    sum[h] = size[h];
  }
#pragma unroll
  for (int off = 1; off < 32; off <<= 1)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int v = __shfl_up_sync(0xffffffffu, sum[h], off);
      if (lane >= off) sum[h] += v;
    }
  sum[1] += __shfl_sync(0xffffffffu, sum[0], 31);
  const int used = (R + 31) / 32, items = phases * used;
  const uint32_t* own = bits + (int64_t)head * phases * R * words;
  // this lane's word among the first 32: phase (by place among those with a budget, and by number) and where it is
  const auto phase_of = [&](int at) { return slot.z == at ? 2 : slot.y == at ? 1 : 0; };
  const int near_at = lane / used, near_word = lane % used, near_phase = phase_of(near_at);
  const auto blocks_of = [&](int t, int& a, int& b) {
    a = sh.block[sh.pairs[t].x];
    b = sh.pairs[t].y ? sh.block[sh.pairs[t].y & (kGroup - 1)] : -1;
  };
  const auto near = [&](int block_) {
    return lane < items && block_ >= 0 ? __ldg(own + ((int64_t)near_at * R + block_) * words + near_word) : 0u;
  };
  int a = 0, b = -1;
  uint32_t wa = 0, wb = 0;
  const int first_pair = warp * gridDim.z + blockIdx.z, step = gridDim.z * kWarps;
  if (first_pair < pairs) {
    blocks_of(first_pair, a, b);
    wa = near(a);
    wb = near(b);
  }
  for (int t = first_pair; t < pairs; t += step) {
    int next_a = 0, next_b = -1;
    uint32_t next_wa = 0, next_wb = 0;
    if (t + step < pairs) {
      blocks_of(t + step, next_a, next_b);
      next_wa = near(next_a);
      next_wb = near(next_b);
    }
    const int upto = __shfl_sync(0xffffffffu, t < 32 ? sum[0] : sum[1], t & 31);
    const int stages = __shfl_sync(0xffffffffu, t < 32 ? size[0] : size[1], t & 31);
    const int64_t offset = start + upto - stages;
    const bool fits = !gave_up && offset + stages <= capacity;  // (the latter always with exact budgets)
    int32_t* list = pair_ids + (int64_t)head * capacity + offset;
    int n[3] = {prefix_phase == 0 ? prefix_stages : 0, prefix_phase == 1 ? prefix_stages : 0,
                prefix_phase == 2 ? prefix_stages : 0};
    int before = 0;  // columns in the words of earlier rounds
    for (int q0 = 0; q0 < items; q0 += 32) {
      int at = near_at, w = near_word, c = near_phase;
      if (q0 > 0) {
        const int q = q0 + lane;
        at = q / used;
        w = q - at * used;
        c = phase_of(at);
        wa = q < items ? __ldg(own + ((int64_t)at * R + a) * words + w) : 0;
        wb = q < items && b >= 0 ? __ldg(own + ((int64_t)at * R + b) * words + w) : 0;
      }
      const int many = __popc(wa | wb);
      int incl = many;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += v;
      }
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if ((k == 0 ? slot.x : k == 1 ? slot.y : slot.z) >= 0) n[k] += __reduce_add_sync(0xffffffffu, c == k ? many : 0);
      // every word in turn, a lane per column
      const int from = before + incl - many + (prefix_phase >= 0 && c >= prefix_phase ? prefix_stages : 0);
      const int column = prefix_stages + w * 32;
      const int ends = min(32, items - q0);
#pragma unroll 4
      for (int q = 0; q < ends; ++q) {
        const uint32_t ma = __shfl_sync(0xffffffffu, wa, q), mb = __shfl_sync(0xffffffffu, wb, q);
        const int to = __shfl_sync(0xffffffffu, from, q), col = __shfl_sync(0xffffffffu, column, q);
        const uint32_t flags = (__funnelshift_l(ma, ma, 30 - lane) & 1u << 30) | (__funnelshift_l(mb, mb, 31 - lane) & 1u << 31);
        if (flags && fits) list[to + __popc((ma | mb) & lower)] = (int)(flags | (uint32_t)(col + lane));
      }
      before += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (prefix_phase >= 0 && fits) {
      int32_t* to = list + (prefix_phase > 0 ? n[0] : 0) + (prefix_phase > 1 ? n[1] : 0);
      for (int k = lane; k < prefix_stages; k += 32) to[k] = k | (b >= 0 ? (int)0xc0000000u : 1 << 30);
    }
    if (lane == 0) {
      const int s = t < in_last ? t * all + group : in_last * all + (t - in_last) * (all - 1) + group;
      int4* entry = table + ((int64_t)head * ((R + 1) / 2) + s) * 2;
      entry[0] = make_int4(a, b, (int)offset, stages);
      entry[1] = fits ? make_int4(n[0], n[1], n[2], 0) : make_int4(0, 0, 0, 0);
    }
    a = next_a;
    b = next_b;
    wa = next_wa;
    wb = next_wb;
  }
  if (warp == 0) tmem_dealloc(tmem, kGroup);
}

}  // namespace

namespace layer {

int match_pairs(const anemoi_sm100_shape& s, const PairBits& bits, int prefix_phase, const int32_t* row_offset,
                const int32_t* row_counts, int32_t* table, int32_t* pair_ids, int64_t capacity, int32_t* status,
                cudaStream_t st) {
  const int R = s.video_blocks;
  const size_t smem = std::max(kRing * kPieceBytes, kGroup * kShareRow * 4) + sizeof(MatchShared);
  if (cudaFuncSetAttribute(match_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return ANEMOI_SM100_ELAUNCH;
  // The lists of few groups are written by several CTAs each, which all make the choice.
  const int parts = groups(R) * s.heads > 74 ? 1 : groups(R) * s.heads > 37 ? 2 : 4;
  return launch(match_kernel, dim3(groups(R), s.heads, parts), dim3(kThreads), smem, st, bits.words, R, pair_bit_words(R),
                bits.phases, make_int3(bits.slot[0], bits.slot[1], bits.slot[2]), row_offset, row_counts,
                rec::prefix_stages(s), prefix_phase, capacity, reinterpret_cast<int4*>(table), pair_ids, status,
                wait_limit_ns()) == cudaSuccess
             ? ANEMOI_SM100_OK
             : ANEMOI_SM100_ELAUNCH;
}

}  // namespace layer
