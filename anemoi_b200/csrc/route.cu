// Routing: global per-head top-k over the [R][R] fp16 probability map with
// precision assigned by rank, emitted as compact ragged lists of 64-key stages
// per query block.
//
// Reference behaviour (csrc/attention/cuda/sm120/h3_route_precision.cu:111-158,
// 222-369 and anemoi/layers/attention/mpa/routing.py:158-235): pairs are ranked
// by descending probability, ties by ascending flat index row*R+col (the
// reference sorts all pairs with a stable radix sort on the 15-bit magnitude);
// ranks < n16 run in FP16, the next n8 in INT8, the next n4 in NVFP4.  Per row
// the list holds the NVFP4 columns, then INT8, then FP16, each ascending; every
// logical block expands to QB/64 consecutive stages and the prefix stages are
// placed at the front of the phase that carries them.
//
// Here the sort is replaced by selection.  A 32768-bin histogram of the keys of
// a head gives, for each of the three rank boundaries, the key that straddles it
// and how many items of that key fall above it (the quota).  One pass per row then
// counts the keys above and equal to each straddling key; a per-head scan over the
// rows turns the equal-counts into each row's position inside the straddling bins,
// from which the row's stages per phase, its list offset (an exclusive scan: the
// layout is the same at every call) and the launch order follow without touching
// the map again; a last pass per row writes the lists.  The per-row passes use one
// warp per row: ranks inside a row come from ballots, no block-wide barrier.
#include <climits>
#include <cooperative_groups.h>
#include <cuda_fp16.h>

#include "canonical.cuh"
#include "layer.cuh"
#include "records.cuh"

namespace {

constexpr int kBins = 32768;
constexpr int kHistThreads = 512;
constexpr int kRowWarps = 8;  // rows per CTA in the per-row passes, one warp each
constexpr int kStat = 6;      // ints per row: keys above boundary 0,1,2; keys equal to its key 0,1,2

struct RouteScratch {
  int* hist;  // [H][kBins]
  int* thr;   // [H][8]: key0, quota0, key1, quota1, key2, quota2, -, -
  int* stat;  // [H][R][kStat]; the equal-counts become exclusive prefixes over the rows
};

__host__ __device__ inline int64_t scratch_ints(int H, int R) {
  return (int64_t)H * (kBins + 8 + kStat * (int64_t)R);
}

// A CTA counts the keys of one half of the key range (blockIdx.z) in its chunk of a head: 64 KB of
// shared-memory bins, so that it fits on an SM beside one CTA of the prefix rows' attention launch,
// which runs on a side stream at the same time (with all 128 KB of bins in one CTA the histogram
// waited for those long CTAs to retire).  The map is L2-resident; reading it twice costs little.
constexpr int kHalfBins = kBins / 2;
__global__ void __launch_bounds__(kHistThreads) hist_kernel(const unsigned short* prob,
                                                            int64_t items, int chunks,
                                                            int* hist) {
  extern __shared__ int local[];
  for (int i = threadIdx.x; i < kHalfBins; i += kHistThreads) local[i] = 0;
  __syncthreads();
  const int head = blockIdx.y, half = blockIdx.z;
  const int64_t per = (items + chunks - 1) / chunks;
  const int64_t lo = (int64_t)blockIdx.x * per, hi = min(items, lo + per);
  const unsigned short* src = prob + (int64_t)head * items;
  for (int64_t i = lo + threadIdx.x; i < hi; i += kHistThreads) {
    const int key = __ldg(src + i) & 0x7fff;
    if ((key >> 14) == half) atomicAdd(&local[key & (kHalfBins - 1)], 1);
  }
  __syncthreads();
  int* out = hist + (int64_t)head * kBins + half * kHalfBins;
  for (int i = threadIdx.x; i < kHalfBins; i += kHistThreads)
    if (local[i]) atomicAdd(out + i, local[i]);
}

// Exclusive prefix of `v` over the threads of a 1024-thread CTA; `total` gets the sum.
// `warp_sum` is shared scratch of 32 entries; the call ends with the scratch free again.
__device__ __forceinline__ long long block_exclusive(long long v, long long* warp_sum,
                                                     long long& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  long long incl = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const long long n = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += n;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  long long base = 0, all = 0;
#pragma unroll
  for (int w = 0; w < 32; ++w) {
    const long long t = warp_sum[w];
    base += w < warp ? t : 0;
    all += t;
  }
  __syncthreads();
  total = all;
  return base + incl - v;
}

// One CTA per head: finds, for each boundary B, the key whose bin contains rank B (keys
// ranked from the largest down) and B's offset inside that bin.  Two levels: sums of 32-bin
// blocks (coalesced reads, one warp reduction each), a scan over the 1024 blocks, then one
// warp per boundary resolves the bin inside the block that straddles it.
// `sub` (optional): a second histogram that is subtracted bin by bin (the anchored variant ranks
// the items that are not anchors).  The results go to thr[head * thr_stride + thr_first ..].
__global__ void __launch_bounds__(1024) threshold_kernel(const int* hist, const int* sub, int* thr,
                                                         int thr_stride, int thr_first, int64_t b0,
                                                         int64_t b1, int64_t b2) {
  __shared__ long long warp_sum[32];
  __shared__ int block_sum[1024];
  __shared__ int hit_block[3];
  __shared__ long long hit_off[3];
  const int head = blockIdx.x;
  const int* h = hist + (int64_t)head * kBins;
  const int* hs = sub ? sub + (int64_t)head * kBins : nullptr;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int mine = 0;
#pragma unroll 4
  for (int i = 0; i < 32; ++i) {
    const int bin = (warp * 32 + i) * 32 + lane;
    const int sum = __reduce_add_sync(0xffffffffu, h[bin] - (hs ? hs[bin] : 0));
    if (lane == i) mine = sum;
  }
  block_sum[threadIdx.x] = mine;
  if (threadIdx.x < 3) hit_block[threadIdx.x] = -1;
  __syncthreads();
  // thread t owns block 1023 - t: blocks in descending key order
  const int blk = 1023 - threadIdx.x;
  const long long total = block_sum[blk];
  long long all;
  const long long above = block_exclusive(total, warp_sum, all);
  const long long bound[3] = {b0, b1, b2};
#pragma unroll
  for (int b = 0; b < 3; ++b)
    if (total > 0 && above <= bound[b] && bound[b] < above + total) {
      hit_block[b] = blk;
      hit_off[b] = bound[b] - above;
    }
  __syncthreads();
  if (warp < 3) {
    int key = -1, quota = 0;  // boundary at or past the last item: every key lies above it
    const int hb = hit_block[warp];
    if (hb >= 0) {
      const int bin = hb * 32 + 31 - lane;  // descending inside the block
      const int n = h[bin] - (hs ? hs[bin] : 0);
      int incl = n;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int m = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += m;
      }
      const long long off = hit_off[warp];
      const bool here = n > 0 && incl - n <= off && off < incl;
      const unsigned who = __ballot_sync(0xffffffffu, here);
      const int src = __ffs(who) - 1;
      key = __shfl_sync(0xffffffffu, bin, src);
      quota = __shfl_sync(0xffffffffu, (int)(off - (incl - n)), src);
    }
    if (lane == 0) {
      thr[head * thr_stride + thr_first + 2 * warp] = key;
      thr[head * thr_stride + thr_first + 2 * warp + 1] = quota;
    }
  }
}

// One warp per row: keys above each straddling key, keys equal to it.
__global__ void __launch_bounds__(kRowWarps * 32) rowstat_kernel(const unsigned short* prob, int R,
                                                                 const int* thr, int* stat) {
  const int row = blockIdx.x * kRowWarps + (threadIdx.x >> 5), head = blockIdx.y;
  if (row >= R) return;
  const int lane = threadIdx.x & 31;
  const int k0 = thr[head * 8], k1 = thr[head * 8 + 2], k2 = thr[head * 8 + 4];
  const unsigned short* src = prob + ((int64_t)head * R + row) * R;
  int g0 = 0, g1 = 0, g2 = 0, e0 = 0, e1 = 0, e2 = 0;
  for (int j = lane; j < R; j += 32) {
    const int key = __ldg(src + j) & 0x7fff;
    g0 += key > k0;
    g1 += key > k1;
    g2 += key > k2;
    e0 += key == k0;
    e1 += key == k1;
    e2 += key == k2;
  }
  g0 = __reduce_add_sync(0xffffffffu, g0);
  g1 = __reduce_add_sync(0xffffffffu, g1);
  g2 = __reduce_add_sync(0xffffffffu, g2);
  e0 = __reduce_add_sync(0xffffffffu, e0);
  e1 = __reduce_add_sync(0xffffffffu, e1);
  e2 = __reduce_add_sync(0xffffffffu, e2);
  if (lane < kStat) {
    const int v = lane == 0 ? g0 : lane == 1 ? g1 : lane == 2 ? g2 : lane == 3 ? e0 : lane == 4 ? e1 : e2;
    stat[((int64_t)head * R + row) * kStat + lane] = v;
  }
}

// One CTA per head, rows in chunks of 1024: position of every row inside the straddling bins
// (exclusive scan of the equal-counts), hence its stages per phase, and its list offset
// (exclusive scan of the totals).  Then the launch order of the head's query blocks for the
// attention kernel: longest list first (ties by block index), written as block + 1 into the
// fourth entry of row_counts, slot = position; the last CTAs of a launch are then the short
// ones, which shortens the tail during which SMs run out of work.  Blocks are ranked by
// counting (R^2 / threads comparisons per thread); very large block counts keep the identity
// order (the fourth entries stay 0).
constexpr int kOrderMaxBlocks = 4096;
__global__ void __launch_bounds__(1024) headscan_kernel(int R, const int* thr, int* stat, int factor,
                                                        int prefix_stages, int prefix_phase, bool ordered,
                                                        int32_t* row_offset, int32_t* row_counts) {
  __shared__ long long warp_sum[32];
  __shared__ int total_s[kOrderMaxBlocks];
  const int head = blockIdx.x;
  int quota[3];
#pragma unroll
  for (int b = 0; b < 3; ++b) quota[b] = thr[head * 8 + 2 * b + 1];
  const int p = prefix_phase >= 0 ? prefix_stages : 0;
  long long carry[4] = {0, 0, 0, 0};  // equal-counts of earlier rows (3), stages of earlier rows
  for (int r0 = 0; r0 < R; r0 += 1024) {
    const int row = r0 + threadIdx.x;
    const bool in = row < R;
    int* st = stat + ((int64_t)head * R + row) * kStat;
    int below[3];
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const int eq = in ? st[3 + b] : 0;
      long long all;
      const long long pre = carry[b] + block_exclusive(eq, warp_sum, all);
      carry[b] += all;
      // items of the straddling key in this row that still fall above the boundary
      const long long room = (long long)quota[b] - pre;
      const int take = (int)max(0ll, min((long long)eq, room));
      below[b] = in ? st[b] + take : 0;
      if (in) st[3 + b] = (int)pre;
    }
    int n[3];
    n[0] = (below[2] - below[1]) * factor + (prefix_phase == 0 ? p : 0);  // NVFP4
    n[1] = (below[1] - below[0]) * factor + (prefix_phase == 1 ? p : 0);  // INT8
    n[2] = below[0] * factor + (prefix_phase == 2 ? p : 0);               // FP16
    const int total = in ? n[0] + n[1] + n[2] : 0;
    long long all;
    const long long off = carry[3] + block_exclusive(total, warp_sum, all);
    carry[3] += all;
    if (in) {
      row_offset[(int64_t)head * R + row] = (int32_t)off;
      int32_t* rc = row_counts + ((int64_t)head * R + row) * 4;
      rc[0] = n[0];
      rc[1] = n[1];
      rc[2] = n[2];
      rc[3] = 0;
      if (row < kOrderMaxBlocks) total_s[row] = total;
    }
  }
  if (!ordered || R > kOrderMaxBlocks) return;
  __syncthreads();
  int32_t* rc = row_counts + (int64_t)head * R * 4;
  for (int i = threadIdx.x; i < R; i += 1024) {
    const int mine = total_s[i];
    int rank = 0;
    for (int j = 0; j < R; ++j) rank += (total_s[j] > mine) || (total_s[j] == mine && j < i);
    rc[rank * 4 + 3] = i + 1;
  }
}

// One warp per row writes the row's list: NVFP4 columns, INT8 columns, FP16 columns, each
// ascending, every logical block expanded to `factor` stages, prefix stages at the front of
// the phase that carries them.
__global__ void __launch_bounds__(kRowWarps * 32) emit_kernel(
    const unsigned short* prob, int R, const int* thr, const int* stat, int factor,
    int prefix_stages, int prefix_phase, int64_t capacity, const int32_t* row_offset,
    const int32_t* row_counts, int32_t* stage_ids) {
  const int row = blockIdx.x * kRowWarps + (threadIdx.x >> 5), head = blockIdx.y;
  if (row >= R) return;
  const int lane = threadIdx.x & 31;
  const unsigned lower = (1u << lane) - 1u;
  int key_b[3], quota_b[3], run[3];
  const int* st = stat + ((int64_t)head * R + row) * kStat;
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    key_b[b] = thr[head * 8 + 2 * b];
    quota_b[b] = thr[head * 8 + 2 * b + 1];
    run[b] = st[3 + b];  // items of the straddling key in earlier rows
  }
  const int32_t* rc = row_counts + ((int64_t)head * R + row) * 4;
  const int n0 = rc[0], n1 = rc[1], n2 = rc[2];
  const int total = n0 + n1 + n2;
  if (total == 0) return;
  const int64_t base = row_offset[(int64_t)head * R + row];
  if (base + total > capacity) return;  // cannot happen with exact budgets
  int32_t* list = stage_ids + (int64_t)head * capacity + base;
  const int p = prefix_phase >= 0 ? prefix_stages : 0;
  // where the video stages of each phase start
  int at[3] = {prefix_phase == 0 ? p : 0, n0 + (prefix_phase == 1 ? p : 0),
               n0 + n1 + (prefix_phase == 2 ? p : 0)};
  if (prefix_phase >= 0) {
    const int seg = prefix_phase == 0 ? 0 : (prefix_phase == 1 ? n0 : n0 + n1);
    for (int s = lane; s < p; s += 32) list[seg + s] = s;
  }
  const unsigned short* src = prob + ((int64_t)head * R + row) * R;
  for (int j0 = 0; j0 < R; j0 += 32) {
    const int j = j0 + lane;
    const bool in = j < R;
    const int key = in ? (__ldg(src + j) & 0x7fff) : -2;
    // rank < boundary b  <=>  key above the straddling key, or inside its bin before the quota
    bool below[3];
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const bool tie = in && key == key_b[b];
      const unsigned ties = __ballot_sync(0xffffffffu, tie);
      below[b] = key > key_b[b] || (tie && run[b] + __popc(ties & lower) < quota_b[b]);
      run[b] += __popc(ties);
    }
    const int c = !in ? 0 : (below[0] ? 3 : (below[1] ? 2 : (below[2] ? 1 : 0)));
#pragma unroll
    for (int k = 1; k <= 3; ++k) {
      const unsigned members = __ballot_sync(0xffffffffu, c == k);
      if (c == k) {
        int32_t* dst = list + at[k - 1] + __popc(members & lower) * factor;
        for (int e = 0; e < factor; ++e) dst[e] = prefix_stages + j * factor + e;
      }
      at[k - 1] += __popc(members) * factor;
    }
  }
}

// ---- routing with anchors (an experimental variant of the reference,
// anemoi/layers/attention/mpa/routing.py:190-203, sm120/h3_route_precision.cu:160-220) -------------
// Anchor pairs (a fixed [R][R] mask shared by the heads: the same-frame neighbours of a block) that
// the ranking dropped are forced into the lowest active precision, and as many of the
// lowest-ranked pairs of that precision that are not anchors are dropped instead.  Restated as
// selection: every anchor is kept (at the precision of its rank, or the lowest one), and of
// the other pairs exactly the retained - anchor_count best ranked are kept, at the precision
// of their rank among all pairs.  So a fourth boundary is taken in the ranking of the pairs
// that are not anchors (their histogram is the full one minus the anchors').  A pair's
// precision then depends on the anchor mask, and the per-row counts are taken by a pass of
// their own before the offsets are scanned.
constexpr int kAnchorStat = 4;  // ints per row: items equal to straddling key 0,1,2; non-anchors equal to key 3

__global__ void __launch_bounds__(256) anchor_hist_kernel(const unsigned short* prob, int64_t items,
                                                          const int32_t* anchor_ids, int count,
                                                          int* hist_anchor) {
  const int i = blockIdx.x * 256 + threadIdx.x, head = blockIdx.y;
  if (i >= count) return;
  const int key = __ldg(prob + (int64_t)head * items + anchor_ids[i]) & 0x7fff;
  atomicAdd(hist_anchor + (int64_t)head * kBins + key, 1);
}

struct AnchorRow {
  int key_b[4], quota_b[4], run[4];
};

__device__ __forceinline__ AnchorRow anchor_row(const int* thr, const int* stat, int head, int R,
                                                int row) {
  AnchorRow a;
  const int* st = stat + ((int64_t)head * R + row) * kAnchorStat;
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    a.key_b[b] = thr[head * 16 + (b < 3 ? 2 * b : 8)];
    a.quota_b[b] = thr[head * 16 + (b < 3 ? 2 * b + 1 : 9)];
    a.run[b] = st[b];
  }
  return a;
}

// Precision code of the lane's column (0 = dropped); advances the row's tie counters.
__device__ __forceinline__ int anchor_code(AnchorRow& a, int key, bool in, bool anchor, unsigned lower,
                                           int lowest_code) {
  bool below[3];
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    const bool tie = in && key == a.key_b[b];
    const unsigned ties = __ballot_sync(0xffffffffu, tie);
    below[b] = key > a.key_b[b] || (tie && a.run[b] + __popc(ties & lower) < a.quota_b[b]);
    a.run[b] += __popc(ties);
  }
  const bool tie = in && !anchor && key == a.key_b[3];
  const unsigned ties = __ballot_sync(0xffffffffu, tie);
  const bool kept = key > a.key_b[3] || (tie && a.run[3] + __popc(ties & lower) < a.quota_b[3]);
  a.run[3] += __popc(ties);
  const int ranked = below[0] ? 3 : (below[1] ? 2 : (below[2] ? 1 : 0));
  if (!in) return 0;
  if (anchor) return ranked ? ranked : lowest_code;
  return kept ? ranked : 0;
}

// One warp per row: items equal to each straddling key (the fourth among the non-anchors only).
__global__ void __launch_bounds__(kRowWarps * 32) anchor_rowstat_kernel(const unsigned short* prob,
                                                                        const uint8_t* anchors, int R,
                                                                        const int* thr, int* stat) {
  const int row = blockIdx.x * kRowWarps + (threadIdx.x >> 5), head = blockIdx.y;
  if (row >= R) return;
  const int lane = threadIdx.x & 31;
  const int k0 = thr[head * 16], k1 = thr[head * 16 + 2], k2 = thr[head * 16 + 4],
            k3 = thr[head * 16 + 8];
  const unsigned short* src = prob + ((int64_t)head * R + row) * R;
  const uint8_t* an = anchors + (int64_t)row * R;
  int e0 = 0, e1 = 0, e2 = 0, e3 = 0;
  for (int j = lane; j < R; j += 32) {
    const int key = __ldg(src + j) & 0x7fff;
    e0 += key == k0;
    e1 += key == k1;
    e2 += key == k2;
    e3 += key == k3 && !an[j];
  }
  e0 = __reduce_add_sync(0xffffffffu, e0);
  e1 = __reduce_add_sync(0xffffffffu, e1);
  e2 = __reduce_add_sync(0xffffffffu, e2);
  e3 = __reduce_add_sync(0xffffffffu, e3);
  if (lane < 4)
    stat[((int64_t)head * R + row) * kAnchorStat + lane] = lane == 0 ? e0 : lane == 1 ? e1 : lane == 2 ? e2 : e3;
}

// One CTA per head: the equal-counts become exclusive prefixes over the rows.
__global__ void __launch_bounds__(1024) anchor_tiescan_kernel(int R, int* stat) {
  __shared__ long long warp_sum[32];
  const int head = blockIdx.x;
  long long carry[4] = {0, 0, 0, 0};
  for (int r0 = 0; r0 < R; r0 += 1024) {
    const int row = r0 + threadIdx.x;
    const bool in = row < R;
    int* st = stat + ((int64_t)head * R + row) * kAnchorStat;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int eq = in ? st[b] : 0;
      long long all;
      const long long pre = carry[b] + block_exclusive(eq, warp_sum, all);
      carry[b] += all;
      if (in) st[b] = (int)pre;
    }
  }
}

// One warp per row: pairs per precision (entries 0..2 of the row's counts, in logical blocks).
__global__ void __launch_bounds__(kRowWarps * 32) anchor_count_kernel(const unsigned short* prob,
                                                                      const uint8_t* anchors, int R,
                                                                      const int* thr, const int* stat,
                                                                      int lowest_code, int32_t* row_counts) {
  const int row = blockIdx.x * kRowWarps + (threadIdx.x >> 5), head = blockIdx.y;
  if (row >= R) return;
  const int lane = threadIdx.x & 31;
  const unsigned lower = (1u << lane) - 1u;
  AnchorRow a = anchor_row(thr, stat, head, R, row);
  const unsigned short* src = prob + ((int64_t)head * R + row) * R;
  const uint8_t* an = anchors + (int64_t)row * R;
  int n[3] = {0, 0, 0};
  for (int j0 = 0; j0 < R; j0 += 32) {
    const int j = j0 + lane;
    const bool in = j < R;
    const int key = in ? (__ldg(src + j) & 0x7fff) : -2;
    const int c = anchor_code(a, key, in, in && an[j] != 0, lower, lowest_code);
#pragma unroll
    for (int k = 1; k <= 3; ++k) n[k - 1] += __popc(__ballot_sync(0xffffffffu, c == k));
  }
  if (lane < 3) row_counts[((int64_t)head * R + row) * 4 + lane] = n[lane];
}

// One CTA per head: stages per phase from the pair counts, list offsets in row order, launch order.
__global__ void __launch_bounds__(1024) anchor_offsets_kernel(int R, int factor, int prefix_stages,
                                                              int prefix_phase, int32_t* row_offset,
                                                              int32_t* row_counts) {
  __shared__ long long warp_sum[32];
  __shared__ int total_s[kOrderMaxBlocks];
  const int head = blockIdx.x;
  const int p = prefix_phase >= 0 ? prefix_stages : 0;
  long long carry = 0;
  for (int r0 = 0; r0 < R; r0 += 1024) {
    const int row = r0 + threadIdx.x;
    const bool in = row < R;
    int32_t* rc = row_counts + ((int64_t)head * R + row) * 4;
    int n[3] = {0, 0, 0};
    if (in)
      for (int c = 0; c < 3; ++c) n[c] = rc[c] * factor + (prefix_phase == c ? p : 0);
    const int total = n[0] + n[1] + n[2];
    long long all;
    const long long off = carry + block_exclusive(total, warp_sum, all);
    carry += all;
    if (in) {
      row_offset[(int64_t)head * R + row] = (int32_t)off;
      rc[0] = n[0];
      rc[1] = n[1];
      rc[2] = n[2];
      rc[3] = 0;
      if (row < kOrderMaxBlocks) total_s[row] = total;
    }
  }
  if (R > kOrderMaxBlocks) return;
  __syncthreads();
  int32_t* rc = row_counts + (int64_t)head * R * 4;
  for (int i = threadIdx.x; i < R; i += 1024) {
    const int mine = total_s[i];
    int rank = 0;
    for (int j = 0; j < R; ++j) rank += (total_s[j] > mine) || (total_s[j] == mine && j < i);
    rc[rank * 4 + 3] = i + 1;
  }
}

// One warp per row writes the row's list (as emit_kernel, with the anchored codes).
__global__ void __launch_bounds__(kRowWarps * 32) anchor_emit_kernel(
    const unsigned short* prob, const uint8_t* anchors, int R, const int* thr, const int* stat,
    int lowest_code, int factor, int prefix_stages, int prefix_phase, int64_t capacity,
    const int32_t* row_offset, const int32_t* row_counts, int32_t* stage_ids) {
  const int row = blockIdx.x * kRowWarps + (threadIdx.x >> 5), head = blockIdx.y;
  if (row >= R) return;
  const int lane = threadIdx.x & 31;
  const unsigned lower = (1u << lane) - 1u;
  AnchorRow a = anchor_row(thr, stat, head, R, row);
  const int32_t* rc = row_counts + ((int64_t)head * R + row) * 4;
  const int n0 = rc[0], n1 = rc[1], n2 = rc[2];
  const int total = n0 + n1 + n2;
  if (total == 0) return;
  const int64_t base = row_offset[(int64_t)head * R + row];
  if (base + total > capacity) return;
  int32_t* list = stage_ids + (int64_t)head * capacity + base;
  const int p = prefix_phase >= 0 ? prefix_stages : 0;
  int at[3] = {prefix_phase == 0 ? p : 0, n0 + (prefix_phase == 1 ? p : 0),
               n0 + n1 + (prefix_phase == 2 ? p : 0)};
  if (prefix_phase >= 0) {
    const int seg = prefix_phase == 0 ? 0 : (prefix_phase == 1 ? n0 : n0 + n1);
    for (int s = lane; s < p; s += 32) list[seg + s] = s;
  }
  const unsigned short* src = prob + ((int64_t)head * R + row) * R;
  const uint8_t* an = anchors + (int64_t)row * R;
  for (int j0 = 0; j0 < R; j0 += 32) {
    const int j = j0 + lane;
    const bool in = j < R;
    const int key = in ? (__ldg(src + j) & 0x7fff) : -2;
    const int c = anchor_code(a, key, in, in && an[j] != 0, lower, lowest_code);
#pragma unroll
    for (int k = 1; k <= 3; ++k) {
      const unsigned members = __ballot_sync(0xffffffffu, c == k);
      if (c == k) {
        int32_t* dst = list + at[k - 1] + __popc(members & lower) * factor;
        for (int e = 0; e < factor; ++e) dst[e] = prefix_stages + j * factor + e;
      }
      at[k - 1] += __popc(members) * factor;
    }
  }
}

// ---- the whole routing of a head in one kernel ------------------------------------------------
// One cluster of 1-8 CTAs per head, each with a contiguous range of the head's rows: histogram
// (32,768 bins in shared memory), boundaries, per-row counts, scans over the rows, lists, launch
// order; with kPairs the union lists of the Q64 query-block pairs instead of the rows' own lists.
// The CTAs of a cluster add up histograms and row totals through distributed shared memory.  The
// map is read three times from L2; what bounds the kernel is the shared-memory atomics of the
// histogram and, for short maps, its dozen barriers.  Those are why the scans of the three boundaries share
// theirs, the CTAs of a cluster exchange their sums once, a cluster of one uses the CTA's barrier, block sums
// go by exchanges of halves and only warps that have rows scan.  Alone, in several launches (five, seven with
// pairs) / in this one, us: 56 x 273 75 / 46, 56 x 672 235 / 190; with pairs 56 x 592 277 / 122.
constexpr int kFusedThreads = 1024;
constexpr int kFusedWarps = kFusedThreads / 32;

struct FusedShared {
  int block_sum[1024];   // items per 32 bins, this CTA's rows
  int4 warp_sum[kFusedWarps];
  int part[4];           // this CTA's sums over its rows, read by the CTAs behind it
  int hit_block[3], hit_off[3];
  int key[3], quota[3];
};

__host__ __device__ inline size_t fused_smem() { return (size_t)kBins * 4 + sizeof(FusedShared); }

// CTAs per head: as many as keep every head on an SM of its own at once, down to 64 rows each (two per
// warp).  Clusters do not cross GPCs, so 15 of eight fit
// at a time and 33 of four.  672 blocks, us: 15 heads in clusters of eight 59, of four 105; 16 heads 115, 105; 33 heads
// in clusters of four 105, of two 188; 37 heads 208, 188; 66 heads in clusters of two 191, of one 359.
inline int fused_ctas(int H, int R) {
  int c = 1;
  while (c < 8 && R > 64 * c && H * c * 2 <= (c == 4 ? 120 : c == 2 ? 132 : 148)) c *= 2;
  return c;
}
inline int fused_rows(int R, int ctas) { return ((R + ctas - 1) / ctas + 1) & ~1; }
// The rows' counts take the histogram's place, which bounds the rows of a CTA.  Otherwise one kernel where at
// least half the SMs have a CTA (of clusters of four, 60), or a CTA has no more than 65,536 pairs: few heads with
// long maps leave most SMs without work, and launches over all rows are quicker.  Lists, us in several kernels / in
// one: 2 heads x 500 blocks 52 / 37, 7 x 672 75 / 58, 16 x 592 90 / 84, 66 x 672 277 / 191; refused 2 x 1,501 163 / 228,
// 4 x 1,000 104 / 108, 36 x 672 160 / 188; on the wrong side of the line 34 x 400 86 / 79 and 37 x 672 166 / 188.  The line is
// that of the lists; pair lists, which cost two kernels more, would gain beyond it (2 x 1,501 225 / 174, 36 x 672
// 246 / 150).
inline bool fused_fits(int H, int R) {
  const int ctas = fused_ctas(H, R);
  if (R > 4096 || 9 * fused_rows(R, ctas) + R > kBins) return false;
  return H * ctas >= (ctas == 4 ? 60 : 74) || (int64_t)R * R / ctas <= 65536;
}

// Exclusive prefixes of the N values over the CTA's threads (two barriers for all of them); `total`
// gets the sums.  Warps that are not `live` have zeros, take part in the barriers only and get nothing.
template <int N>
__device__ __forceinline__ void fused_exclusive(int (&v)[N], int4* warp_sum, int (&total)[N], bool live = true) {
  static_assert(N <= 4, "one int4 per warp");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (!live) {
    if (lane == 0) warp_sum[warp] = make_int4(0, 0, 0, 0);
    __syncthreads();
    __syncthreads();
    return;
  }
  int incl[N];
#pragma unroll
  for (int k = 0; k < N; ++k) incl[k] = v[k];
#pragma unroll
  for (int off = 1; off < 32; off <<= 1)
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const int n = __shfl_up_sync(0xffffffffu, incl[k], off);
      if (lane >= off) incl[k] += n;
    }
  if (lane == 31)
#pragma unroll
    for (int k = 0; k < N; ++k) reinterpret_cast<int*>(&warp_sum[warp])[k] = incl[k];
  __syncthreads();
  int w[N], winc[N];
#pragma unroll
  for (int k = 0; k < N; ++k) winc[k] = w[k] = reinterpret_cast<int*>(&warp_sum[lane])[k];
#pragma unroll
  for (int off = 1; off < 32; off <<= 1)
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const int n = __shfl_up_sync(0xffffffffu, winc[k], off);
      if (lane >= off) winc[k] += n;
    }
#pragma unroll
  for (int k = 0; k < N; ++k) {
    total[k] = __shfl_sync(0xffffffffu, winc[k], 31);
    v[k] = __shfl_sync(0xffffffffu, winc[k] - w[k], warp) + incl[k] - v[k];
  }
  __syncthreads();
}

constexpr int kAhead = 8;  // 32-column pieces of a row whose keys are loaded before the first is looked at

// The keys of columns [j0, j0 + 32 * kAhead) of a row, -2 past its end.
__device__ __forceinline__ void fused_keys(const unsigned short* src, int j0, int R, int (&key)[kAhead]) {
#pragma unroll
  for (int u = 0; u < kAhead; ++u) {
    const int j = j0 + u * 32 + (threadIdx.x & 31);
    key[u] = j < R ? (__ldg(src + j) & 0x7fff) : -2;
  }
}

// Precision code (3 FP16, 2 INT8, 1 NVFP4, 0 dropped) of the lane's column; advances the row's
// counters of straddling keys met so far.  Straddling keys are rare: one vote skips their ranks.
__device__ __forceinline__ int fused_code(int key, const int (&key_b)[3], const int (&quota_b)[3], int (&run)[3],
                                          unsigned lower) {
  int c = (key > key_b[0]) + (key > key_b[1]) + (key > key_b[2]);
  if (__any_sync(0xffffffffu, key == key_b[0] || key == key_b[1] || key == key_b[2])) {
    c = 0;
#pragma unroll
    for (int b = 2; b >= 0; --b) {
      const unsigned ties = __ballot_sync(0xffffffffu, key == key_b[b]);
      const bool below = key > key_b[b] || (key == key_b[b] && run[b] + __popc(ties & lower) < quota_b[b]);
      run[b] += __popc(ties);
      c = below ? 3 - b : c;
    }
  }
  return c;
}

// ---- the draft map in the routing kernel: up to 32 blocks per head ---------------------------------
// The arithmetic of draft.cu with a column per lane.  Up to there a head's map is 1-2 us of work, and a launch of its own costs
// 2.5 us on the host and as much on the device (INT8 without a prefix, in two launches / in one, D = 64, 1 head x 8 blocks
// 22.3 / 20.4, 24 x 24, two maps 43.3 / 40.5, D = 128, 8 x 16, two maps 34.6 / 28.9).
constexpr int kDraftBlocks = 32;
struct DraftPools {
  const __half* q[2];  // mean, max
  const __half* k[2];
  int maps;      // 1 or 2
  float weight;  // of the max pools' map
  unsigned short* map;
};

// The map's entries of kRows neighbouring rows per warp, a column per lane.
template <int D, int kRows, int kThreads>
__device__ __forceinline__ void draft_rows(const DraftPools& d, int head, int R, uint32_t* smem, float (&out)[kRows]) {
  uint32_t* kc = smem;                                                         // [maps][D / 2][32], two channels a word
  float* qs = reinterpret_cast<float*>(smem + d.maps * D / 2 * kDraftBlocks);  // [maps][32][D]
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    if (m >= d.maps) break;
    for (int idx = threadIdx.x; idx < kDraftBlocks * (D / 8); idx += kThreads) {
      const int col = idx % kDraftBlocks, c8 = idx / kDraftBlocks;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (col < R) v = __ldg(reinterpret_cast<const uint4*>(d.k[m] + ((int64_t)head * R + col) * D) + c8);
      uint32_t* dst = kc + (m * (D / 2) + c8 * 4) * kDraftBlocks + col;
      dst[0] = v.x;
      dst[kDraftBlocks] = v.y;
      dst[2 * kDraftBlocks] = v.z;
      dst[3 * kDraftBlocks] = v.w;
    }
    for (int idx = threadIdx.x; idx < R * (D / 2); idx += kThreads)
      reinterpret_cast<float2*>(qs + m * kDraftBlocks * D)[idx] =
          __half22float2(__ldg(reinterpret_cast<const __half2*>(d.q[m] + (int64_t)head * R * D) + idx));
  }
  __syncthreads();
  const int r0 = (threadIdx.x >> 5) * kRows, lane = threadIdx.x & 31;
  const bool in = lane < R;
#pragma unroll
  for (int r = 0; r < kRows; ++r) out[r] = 0.0f;
  if (r0 >= R) return;
  float p[2][kRows];
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    if (m >= d.maps) break;
    // (rows past the map are read from rows of it)
    const float4* q[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) q[r] = reinterpret_cast<const float4*>(qs + (m * kDraftBlocks + min(r0 + r, R - 1)) * D);
    const uint32_t* k = kc + m * (D / 2) * kDraftBlocks + lane;
    float acc[kRows] = {};
#pragma unroll 8
    for (int c4 = 0; c4 < D / 4; ++c4) {
      const uint32_t w0 = k[2 * c4 * kDraftBlocks], w1 = k[(2 * c4 + 1) * kDraftBlocks];
      const float2 k0 = __half22float2(*reinterpret_cast<const __half2*>(&w0));
      const float2 k1 = __half22float2(*reinterpret_cast<const __half2*>(&w1));
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
        const float4 qv = q[r][c4];
        acc[r] = __fmaf_rn(qv.y, k0.y, __fmaf_rn(qv.x, k0.x, acc[r]));
        acc[r] = __fmaf_rn(qv.w, k1.y, __fmaf_rn(qv.z, k1.x, acc[r]));
      }
    }
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const float logit =
          __half2float(__float2half_rn(__fmul_rn(acc[r], D == 64 ? 0.125f : __int_as_float(0x3db504f3))));
      float mx = in ? fmaxf(-INFINITY, logit) : -INFINITY;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
      const float e = canonical::exp_canonical(__fsub_rn(logit, mx));
      float sum = in ? e : 0.0f;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, off));
      p[m][r] = __fmul_rn(e, __fdiv_rn(1.0f, sum));
    }
  }
#pragma unroll
  for (int r = 0; r < kRows; ++r)
    out[r] = d.maps == 1 ? p[0][r]
                         : __fadd_rn(__fmul_rn(__fsub_rn(1.0f, d.weight), p[0][r]), __fmul_rn(d.weight, p[1][r]));
}

// What the kernel leaves: the rows' lists, the union lists of neighbouring Q64 blocks, or a bit per (row, phase,
// column) for the choice of the pairs (match.cu).
enum Leaves : int { kLists = 0, kNeighbours = 1, kBits = 2 };

// A row's bits, 32 columns (a word) at a time: lane w keeps word w of each phase until 32 are there.
struct RowBits {
  uint32_t* out[3];  // by precision code - 1; null: no budget
  uint32_t keep[3];
  __device__ __forceinline__ void put(int k, int word, uint32_t members) {
    if ((word & 31) == (int)(threadIdx.x & 31)) keep[k] = members;
  }
  // After word `word` (the row's last of `words` in use, or the last of a group of 32); rows are `stride` words.
  __device__ __forceinline__ void flush(int word, int words, int stride) {
    if ((word & 31) != 31 && word != words - 1) return;
    const int lane = threadIdx.x & 31, at = (word & ~31) + lane;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (out[k] != nullptr && at < stride) out[k][at] = keep[k];
      keep[k] = 0;
    }
  }
};
__device__ __forceinline__ RowBits row_bits(const layer::PairBits& bits, int head, int R, int row, int stride) {
  RowBits b = {};
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (bits.slot[k] >= 0) b.out[k] = bits.words + (((int64_t)head * bits.phases + bits.slot[k]) * R + row) * stride;
  return b;
}

template <int kLeaves>
__global__ void __launch_bounds__(kFusedThreads, 1) route_fused_kernel(
    const unsigned short* prob, int R, int rows_per, int b0, int b1, int b2, int factor, int prefix_stages,
    int prefix_phase, int64_t capacity, int32_t* row_offset, int32_t* row_counts, int32_t* stage_ids,
    int32_t* pair_counts, int32_t* pair_ids, const layer::PairBits bits) {
  constexpr bool kPairs = kLeaves == kNeighbours;
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) int hist[];
  FusedShared& sh = *reinterpret_cast<FusedShared*>(hist + kBins);
  cg::cluster_group cluster = cg::this_cluster();
  const int ctas = cluster.num_blocks(), me = cluster.block_rank();
  auto sync_all = [&]() {
    if (ctas > 1) {
      cluster.sync();
    } else {
      __syncthreads();
    }
  };
  const int head = blockIdx.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lower = (1u << lane) - 1u;
  const int r0 = min(R, me * rows_per), r1 = min(R, r0 + rows_per), mine = r1 - r0;
  const unsigned short* map = prob + (int64_t)head * R * R;

  // ---- histogram of this CTA's rows ----
  for (int i = threadIdx.x; i < kBins / 4; i += kFusedThreads) reinterpret_cast<int4*>(hist)[i] = make_int4(0, 0, 0, 0);
  __syncthreads();
  layer::grid_dependency_wait();
  layer::grid_dependency_trigger();
  {
    const unsigned short* src = map + (int64_t)r0 * R;
    const int items = mine * R;
    const int head_items = min(items, (int)((16 - (reinterpret_cast<uintptr_t>(src) & 15)) & 15) / 2);
    const int vecs = (items - head_items) / 8;
    const uint4* v = reinterpret_cast<const uint4*>(src + head_items);
    if ((int)threadIdx.x < head_items) atomicAdd(&hist[__ldg(src + threadIdx.x) & 0x7fff], 1);
    const int tail = head_items + vecs * 8;
    if (tail + (int)threadIdx.x < items && threadIdx.x < 8) 
      atomicAdd(&hist[__ldg(src + tail + threadIdx.x) & 0x7fff], 1);
#pragma unroll 2
    for (int i = threadIdx.x; i < vecs; i += kFusedThreads) {
      const uint4 q = __ldg(v + i);
      const unsigned w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        atomicAdd(&hist[w[k] & 0x7fff], 1);
        atomicAdd(&hist[(w[k] >> 16) & 0x7fff], 1);
      }
    }
  }
  __syncthreads();
  // ---- the key that straddles each boundary (keys ranked from the largest down) ----
  {
    // eight lanes hold four bins each of a block, of eight blocks; every exchange halves the blocks a
    // lane still sums, so that each ends with one
    int sum[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int4 bins = *reinterpret_cast<const int4*>(hist + warp * 1024 + k * 128 + lane * 4);
      sum[k] = (bins.x + bins.y) + (bins.z + bins.w);
    }
#pragma unroll
    for (int half = 4; half > 0; half >>= 1) {
      const bool upper = lane & half;
#pragma unroll
      for (int k = 0; k < half; ++k) {
        const int got = __shfl_xor_sync(0xffffffffu, upper ? sum[k] : sum[k + half], half);
        sum[k] = (upper ? sum[k + half] : sum[k]) + got;
      }
    }
    sh.block_sum[warp * 32 + 4 * (lane & 7) + (lane >> 3)] = sum[0];
  }
  if (threadIdx.x < 3) sh.hit_block[threadIdx.x] = -1;
  if (threadIdx.x < 4) sh.part[threadIdx.x] = 0;
  sync_all();
  {
    const int blk = 1023 - threadIdx.x;  // blocks in descending key order
    int total = 0;
    for (int c = 0; c < ctas; ++c) total += cluster.map_shared_rank(sh.block_sum, c)[blk];
    int before[1] = {total}, all[1];
    fused_exclusive(before, sh.warp_sum, all);
    const int above = before[0];
    const int bound[3] = {b0, b1, b2};
#pragma unroll
    for (int b = 0; b < 3; ++b)
      if (total > 0 && above <= bound[b] && bound[b] < above + total) {
        sh.hit_block[b] = blk;
        sh.hit_off[b] = bound[b] - above;
      }
  }
  __syncthreads();
  if (warp < 3) {
    int key = -1, quota = 0;  // boundary at or past the last item: every key lies above it
    const int hb = sh.hit_block[warp];
    if (hb >= 0) {
      const int bin = hb * 32 + 31 - lane;  // descending inside the block
      int n = 0;
      for (int c = 0; c < ctas; ++c) n += cluster.map_shared_rank(hist, c)[bin];
      int incl = n;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int m = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += m;
      }
      const int off = sh.hit_off[warp];
      const int src = __ffs(__ballot_sync(0xffffffffu, n > 0 && incl - n <= off && off < incl)) - 1;
      key = __shfl_sync(0xffffffffu, bin, src);
      quota = __shfl_sync(0xffffffffu, off - (incl - n), src);
    }
    if (lane == 0) {
      sh.key[warp] = key;
      sh.quota[warp] = quota;
    }
  }
  sync_all();  // the histograms are read; their space holds the rows' counts from here on
  const int key_b[3] = {sh.key[0], sh.key[1], sh.key[2]};
  const int quota_b[3] = {sh.quota[0], sh.quota[1], sh.quota[2]};
  int* stat = hist;                    // [mine][6]: keys above boundary 0-2, equal to its key 0-2
  int* totals = stat + 6 * rows_per;   // [mine] stages of a row
  int* offset = totals + rows_per;     // [mine] where its list starts
  int* unions = offset + rows_per;     // [pairs of mine] stages of a pair's union
  int* every = unions + rows_per;      // [R] the totals (unions) of the whole head

  // ---- per row: keys above and equal to each straddling key ----
  for (int i = warp; i < mine; i += kFusedWarps) {
    const unsigned short* src = map + (int64_t)(r0 + i) * R;
    int n[3] = {0, 0, 0};  // keys above | equal << 16 (a row has 4,096 at most)
    for (int j0 = 0; j0 < R; j0 += 32 * kAhead) {
      int key[kAhead];
      fused_keys(src, j0, R, key);
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        if (j0 + u * 32 >= R) break;
#pragma unroll
        for (int b = 0; b < 3; ++b) n[b] += key[u] > key_b[b] ? 1 : (key[u] == key_b[b] ? 1 << 16 : 0);
      }
    }
    int v = 0;
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const int both = __reduce_add_sync(0xffffffffu, n[b]);
      v = lane == b ? both & 0xffff : (lane == 3 + b ? both >> 16 : v);
    }
    if (lane < 6) stat[i * 6 + lane] = v;
    // the CTA's sums: keys equal to each boundary's key, keys above the last boundary
    if (ctas > 1 && lane >= 2 && lane < 6) atomicAdd(&sh.part[lane - 2], v);
  }
  sync_all();
  // ---- scans over the rows: position inside the straddling bins, stages per phase, list offset ----
  const int p = prefix_phase >= 0 ? prefix_stages : 0;
  int carry[4] = {0, 0, 0, 0};  // of the rows before: keys equal to each boundary's key, stages
  for (int c = 0; c < me; ++c) {
    const int* part = cluster.map_shared_rank(sh.part, c);
    const int rows = min(R, (c + 1) * rows_per) - min(R, c * rows_per);
    carry[3] += (part[0] + max(0, min(part[3], quota_b[2] - carry[2]))) * factor + rows * p;
#pragma unroll
    for (int b = 0; b < 3; ++b) carry[b] += part[1 + b];
  }
  for (int i0 = 0; i0 < mine; i0 += kFusedThreads) {
    const int i = i0 + threadIdx.x;
    const bool in = i < mine;
    int pre[3], all[3] = {0, 0, 0}, below[3];
#pragma unroll
    for (int b = 0; b < 3; ++b) pre[b] = in ? stat[i * 6 + 3 + b] : 0;
    const bool live = i0 + warp * 32 < mine;
    fused_exclusive(pre, sh.warp_sum, all, live);
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      pre[b] += carry[b];
      carry[b] += all[b];
      // items of the straddling key in this row that still fall above the boundary
      below[b] = in ? stat[i * 6 + b] + max(0, min(stat[i * 6 + 3 + b], quota_b[b] - pre[b])) : 0;
    }
    const int n0 = (below[2] - below[1]) * factor + (prefix_phase == 0 ? p : 0);  // NVFP4
    const int n1 = (below[1] - below[0]) * factor + (prefix_phase == 1 ? p : 0);  // INT8
    const int n2 = below[0] * factor + (prefix_phase == 2 ? p : 0);               // FP16
    int off[1] = {in ? n0 + n1 + n2 : 0}, sum[1] = {0};
    fused_exclusive(off, sh.warp_sum, sum, live);
    off[0] += carry[3];
    carry[3] += sum[0];
    if (in) {
#pragma unroll
      for (int b = 0; b < 3; ++b) stat[i * 6 + 3 + b] = pre[b];
      stat[i * 6] = n0;
      stat[i * 6 + 1] = n1;
      stat[i * 6 + 2] = n2;
      totals[i] = n0 + n1 + n2;
      offset[i] = off[0];
      row_offset[(int64_t)head * R + r0 + i] = off[0];
      // (with pairs there is no launch order of single blocks; the other kernel fills it in.  One by one: a caller's
      // arrays are on four bytes)
      int32_t* rc = row_counts + ((int64_t)head * R + r0 + i) * 4;
      rc[0] = n0;
      rc[1] = n1;
      rc[2] = n2;
      rc[3] = 0;
    }
  }
  __syncthreads();
  // ---- lists ----
  const bool active[3] = {b2 > b1, b1 > b0, b0 > 0};  // phases with a budget
  if constexpr (kLeaves == kBits) {
    const int words = (R + 31) / 32, stride = layer::pair_bit_words(R);
    for (int i = warp; i < mine; i += kFusedWarps) {
      RowBits row = row_bits(bits, head, R, r0 + i, stride);
      int run[3] = {stat[i * 6 + 3], stat[i * 6 + 4], stat[i * 6 + 5]};
      const unsigned short* src = map + (int64_t)(r0 + i) * R;
      for (int j0 = 0; j0 < R; j0 += 32 * kAhead) {
        int key[kAhead];
        fused_keys(src, j0, R, key);
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          if (j0 + u * 32 >= R) break;
          const int c = fused_code(key[u], key_b, quota_b, run, lower);
#pragma unroll
          for (int k = 1; k <= 3; ++k)
            if (active[k - 1]) row.put(k - 1, j0 / 32 + u, __ballot_sync(0xffffffffu, c == k));
          row.flush(j0 / 32 + u, words, stride);
        }
      }
    }
    if (ctas > 1) cluster.sync();  // no CTA leaves while another may still read its sums
    return;
  } else if constexpr (!kPairs) {
    for (int i = warp; i < mine; i += kFusedWarps) {
      const int n0 = stat[i * 6], n1 = stat[i * 6 + 1], total = totals[i];
      const int64_t base = offset[i];
      if (total == 0 || base + total > capacity) continue;  // (the latter cannot happen with exact budgets)
      int32_t* list = stage_ids + (int64_t)head * capacity + base;
      // where the video stages of each phase start
      int at[3] = {prefix_phase == 0 ? p : 0, n0 + (prefix_phase == 1 ? p : 0),
                   n0 + n1 + (prefix_phase == 2 ? p : 0)};
      if (prefix_phase >= 0) {
        const int seg = prefix_phase == 0 ? 0 : (prefix_phase == 1 ? n0 : n0 + n1);
        for (int s = lane; s < p; s += 32) list[seg + s] = s;
      }
      int run[3] = {stat[i * 6 + 3], stat[i * 6 + 4], stat[i * 6 + 5]};
      const unsigned short* src = map + (int64_t)(r0 + i) * R;
      for (int j0 = 0; j0 < R; j0 += 32 * kAhead) {
        int key[kAhead];
        fused_keys(src, j0, R, key);
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          if (j0 + u * 32 >= R) break;
          const int stage = prefix_stages + (j0 + u * 32 + lane) * factor;
          const int c = fused_code(key[u], key_b, quota_b, run, lower);
#pragma unroll
          for (int k = 1; k <= 3; ++k) {
            if (!active[k - 1]) continue;
            const unsigned members = __ballot_sync(0xffffffffu, c == k);
            if (c == k) {
              int32_t* dst = list + at[k - 1] + __popc(members & lower) * factor;
              dst[0] = stage;
              if (factor == 2) dst[1] = stage + 1;
            }
            at[k - 1] += __popc(members) * factor;
          }
        }
      }
    }
  } else {
    // One warp per pair (blocks 2t and 2t+1; rows_per is even): a stage of either block's list
    // enters the union of its phase once, with a bit per block.  The union of phase c starts where
    // the two blocks' phases before it would end, so no offsets are scanned.
    const int pairs_all = (R + 1) / 2;
    for (int i = 2 * warp; i < mine; i += 2 * kFusedWarps) {
      const bool has_b = i + 1 < mine;
      const int a = i, bb = has_b ? i + 1 : i;
      const int n0 = stat[a * 6] + (has_b ? stat[bb * 6] : 0), n1 = stat[a * 6 + 1] + (has_b ? stat[bb * 6 + 1] : 0);
      const int total = totals[a] + (has_b ? totals[bb] : 0);
      const int64_t base = offset[a];
      const bool fits = base + total <= capacity;
      int32_t* list = pair_ids + (int64_t)head * capacity + base;
      const int start[3] = {0, n0, n0 + n1};
      int at[3] = {start[0], start[1], start[2]};
      const int both = has_b ? (int)0xc0000000u : 1 << 30;
      if (prefix_phase >= 0 && fits) {
        for (int s = lane; s < p; s += 32) list[start[prefix_phase] + s] = s | both;
        at[prefix_phase] += p;
      }
      int run_a[3] = {stat[a * 6 + 3], stat[a * 6 + 4], stat[a * 6 + 5]};
      int run_b[3] = {stat[bb * 6 + 3], stat[bb * 6 + 4], stat[bb * 6 + 5]};
      const unsigned short* src_a = map + (int64_t)(r0 + a) * R;
      const unsigned short* src_b = map + (int64_t)(r0 + bb) * R;
      for (int j0 = 0; j0 < R; j0 += 32 * kAhead) {
        int ka[kAhead], kb[kAhead];
        fused_keys(src_a, j0, R, ka);
        fused_keys(src_b, j0, has_b ? R : 0, kb);
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          if (j0 + u * 32 >= R) break;
          const int stage = prefix_stages + j0 + u * 32 + lane;
          const int ca = fused_code(ka[u], key_b, quota_b, run_a, lower);
          const int cb = fused_code(kb[u], key_b, quota_b, run_b, lower);
#pragma unroll
          for (int k = 1; k <= 3; ++k) {
            if (!active[k - 1]) continue;
            const bool in = ca == k || cb == k;
            const unsigned members = __ballot_sync(0xffffffffu, in);
            if (in && fits)
              list[at[k - 1] + __popc(members & lower)] =
                  stage | (ca == k ? 1 << 30 : 0) | (cb == k ? (int)(1u << 31) : 0);
            at[k - 1] += __popc(members);
          }
        }
      }
      const int u[3] = {at[0] - start[0], at[1] - start[1], at[2] - start[2]};
      if (lane < 3) pair_counts[((int64_t)head * pairs_all + (r0 + i) / 2) * 4 + lane] = lane == 0 ? u[0] : lane == 1 ? u[1] : u[2];
      if (lane == 0) unions[i / 2] = u[0] + u[1] + u[2];
    }
  }
  // ---- launch order: longest list first, ties by block index, as block + 1 in the fourth entry of
  // the position's counts ----
  const int unit = kPairs ? 2 : 1;
  const int count = (R + unit - 1) / unit, per = rows_per / unit, first = r0 / unit;
  const int own = (mine + unit - 1) / unit;
  sync_all();
  for (int j = threadIdx.x; j < count; j += kFusedThreads)
    every[j] = cluster.map_shared_rank(kPairs ? unions : totals, j / per)[j % per];
  __syncthreads();
  int32_t* order = (kPairs ? pair_counts + (int64_t)head * count * 4 : row_counts + (int64_t)head * count * 4) + 3;
  // (eight lanes per position: a thread each was 273 steps for 273 blocks)
  for (int i0 = 0; i0 < own; i0 += kFusedThreads / 8) {
    const int i = i0 + threadIdx.x / 8, me_i = first + min(i, own - 1), len = every[me_i];
    int rank = 0;
#pragma unroll 4
    for (int j = threadIdx.x & 7; j < count; j += 8) rank += every[j] > len || (every[j] == len && j < me_i);
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, off);
    if (i < own && (threadIdx.x & 7) == 0) order[rank * 4] = me_i + 1;
  }
  if (ctas > 1) cluster.sync();  // no CTA leaves while another may still read its totals
}

template <int kLeaves>
int launch_fused(const anemoi_sm100_shape& s, const void* probability, int64_t n16, int64_t n8, int64_t n4,
                 int prefix_phase, int32_t* row_offset, int32_t* row_counts, int32_t* stage_ids, int64_t capacity,
                 int32_t* pair_counts, int32_t* pair_ids, cudaStream_t st, const layer::PairBits& bits = {}) {
  const int H = s.heads, R = s.video_blocks, ctas = fused_ctas(H, R);
  auto kernel = route_fused_kernel<kLeaves>;
  // Function attributes belong to a device: the opt-in is made at every call (a cheap host-side
  // driver call), so a process that routes on several GPUs, or from several host threads,
  // never launches the kernel without the opt-in for its dynamic shared memory.
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fused_smem()) != cudaSuccess)
    return ANEMOI_SM100_ELAUNCH;
  return layer::launch_cluster(kernel, dim3(ctas, H), dim3(ctas), dim3(kFusedThreads), fused_smem(), st,
                               static_cast<const unsigned short*>(probability), R, fused_rows(R, ctas), (int)n16,
                               (int)(n16 + n8), (int)(n16 + n8 + n4), s.query_block / 64, rec::prefix_stages(s),
                               prefix_phase, capacity, row_offset, row_counts, stage_ids, pair_counts, pair_ids,
                               bits) == cudaSuccess
             ? ANEMOI_SM100_OK
             : ANEMOI_SM100_ELAUNCH;
}

// ---- short maps: up to 64 blocks per head -------------------------------------------------------
// One CTA per head with the map's keys in registers: a lane has columns lane and lane + 32, a warp kCols * 2
// neighbouring rows.  The kernel is a chain of latencies (and int operations run at half rate), so the
// histogram is of 1,024 bins of 32 keys, resolved by a second one of the bins that hold the boundaries, rows
// are counted by ballots, and every warp scans all rows for itself instead of waiting for one that does.  A CTA
// leaves room for one of the prefix rows beside it, which the kernel above does not.
// Whole calls, with the kernel above / with this one, us: 4 heads x 16 blocks INT8 D = 64 (with the map) 23.9 / 19.5,
// 24 x 18 NVFP4 33.6 / 30.6, 2 x 12 and 288 tokens of prefix 37.0 / 32.9, 21 x 17 pairs 51.3 / 47.2, 1 x 42 three cells
// 47.2 / 42.6, 11 x 44 FP16 35.4 / 31.5; 50 x 64 INT8 366 / 365.
constexpr int kShortThreads = 512;
constexpr int kShortWarps = kShortThreads / 32;
constexpr int kShortBlocks = 64;

struct ShortShared {
  alignas(16) int bins[1024];
  int fine[3][32];
  int warp_sum[kShortWarps];
  int hit[3], off[3];
  int equal[3][kShortBlocks], above[3][kShortBlocks];
  int unions[kShortBlocks / 2];
};
__host__ __device__ constexpr int draft_words(int D, int maps) {  // both pools of the map: halves, and floats
  return maps * (D / 2 * kDraftBlocks + kDraftBlocks * D);
}

template <int kCols, bool kPairs, int kDraft>
__global__ void __launch_bounds__(kShortThreads) route_short_kernel(
    const DraftPools draft, const unsigned short* prob, int R, int b0, int b1, int b2, int factor, int prefix_stages,
    int prefix_phase, int64_t capacity, int32_t* row_offset, int32_t* row_counts, int32_t* stage_ids,
    int32_t* pair_counts, int32_t* pair_ids) {
  static_assert(kDraft == 0 || kCols == 1, "the map is formed up to 32 blocks");
  constexpr int kRows = 2 * kCols;  // of a warp
  extern __shared__ __align__(16) uint32_t pools[];
  __shared__ ShortShared sh;
  const int head = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row0 = warp * kRows;
  const unsigned lower = (1u << lane) - 1u;
  for (int i = threadIdx.x; i < 1024; i += kShortThreads) sh.bins[i] = 0;
  if (threadIdx.x < 96) sh.fine[threadIdx.x / 32][lane] = 0;
  if (threadIdx.x < 3) sh.hit[threadIdx.x] = -1;
  layer::grid_dependency_wait();
  layer::grid_dependency_trigger();

  // ---- keys, -2 past the map ----
  int key[kRows][kCols];
  if constexpr (kDraft != 0) {
    float p[kRows];
    draft_rows<kDraft, kRows, kShortThreads>(draft, head, R, pools, p);
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const bool in = row0 + r < R && lane < R;
      const unsigned short entry = __half_as_ushort(__float2half_rn(p[r]));
      if (in) draft.map[((int64_t)head * R + row0 + r) * R + lane] = entry;
      key[r][0] = in ? entry & 0x7fff : -2;
    }
  } else {
#pragma unroll
    for (int r = 0; r < kRows; ++r)
#pragma unroll
      for (int c = 0; c < kCols; ++c) {
        const int j = c * 32 + lane;
        key[r][c] = row0 + r < R && j < R ? __ldg(prob + ((int64_t)head * R + row0 + r) * R + j) & 0x7fff : -2;
      }
    __syncthreads();  // the bins are empty
  }
  // ---- bins of 32 keys that hold the boundaries, then the keys ----
#pragma unroll
  for (int r = 0; r < kRows; ++r)
#pragma unroll
    for (int c = 0; c < kCols; ++c)
      if (key[r][c] >= 0) atomicAdd(&sh.bins[key[r][c] >> 5], 1);
  __syncthreads();
  {
    // thread t has bins 1023 - 2t and 1022 - 2t: keys in descending order
    const int2 two = *reinterpret_cast<const int2*>(&sh.bins[1022 - 2 * threadIdx.x]);
    int incl = two.x + two.y;
    const int mine = incl;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += v;
    }
    if (lane == 31) sh.warp_sum[warp] = incl;
    __syncthreads();
    const int before = __reduce_add_sync(0xffffffffu, lane < warp ? sh.warp_sum[lane & (kShortWarps - 1)] : 0);
    const int start[2] = {before + incl - mine, before + incl - mine + two.y}, count[2] = {two.y, two.x};
    const int bound[3] = {b0, b1, b2};
#pragma unroll
    for (int b = 0; b < 3; ++b)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (start[h] <= bound[b] && bound[b] < start[h] + count[h]) {
          sh.hit[b] = 1023 - 2 * (int)threadIdx.x - h;
          sh.off[b] = bound[b] - start[h];
        }
  }
  __syncthreads();
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    const int bin = sh.hit[b];
#pragma unroll
    for (int r = 0; r < kRows; ++r)
#pragma unroll
      for (int c = 0; c < kCols; ++c)
        if (key[r][c] >= 0 && key[r][c] >> 5 == bin) atomicAdd(&sh.fine[b][key[r][c] & 31], 1);
  }
  __syncthreads();
  int key_b[3], quota_b[3];
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    const int n = sh.fine[b][31 - lane], off = sh.off[b], bin = sh.hit[b];  // descending
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    const int src = __ffs(__ballot_sync(0xffffffffu, n > 0 && incl - n <= off && off < incl)) - 1;
    // (a boundary at or past the last item: every key lies above it)
    key_b[b] = bin < 0 ? -1 : bin * 32 + 31 - src;
    quota_b[b] = bin < 0 ? 0 : off - __shfl_sync(0xffffffffu, incl - n, src & 31);
  }
  // ---- per row: keys above and equal to each straddling key ----
#pragma unroll
  for (int r = 0; r < kRows; ++r)
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      int above = 0, equal = 0;
#pragma unroll
      for (int c = 0; c < kCols; ++c) {
        above += __popc(__ballot_sync(0xffffffffu, key[r][c] > key_b[b]));
        equal += __popc(__ballot_sync(0xffffffffu, key[r][c] == key_b[b]));
      }
      if (lane == 0) {
        sh.above[b][row0 + r] = above;
        sh.equal[b][row0 + r] = equal;
      }
    }
  __syncthreads();
  // ---- scans over the rows, a lane per row of 32: position inside the straddling bins, stages, list offsets ----
  const int p = prefix_phase >= 0 ? prefix_stages : 0;
  int pre[kCols][3], n[kCols][3], total[kCols], offset[kCols];
  int carry[4] = {0, 0, 0, 0};
#pragma unroll
  for (int h = 0; h < kCols; ++h) {
    const int row = h * 32 + lane;
    int below[3];
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const int equal = row < R ? sh.equal[b][row] : 0;
      int incl = equal;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      pre[h][b] = carry[b] + incl - equal;
      carry[b] += __shfl_sync(0xffffffffu, incl, 31);
      // items of the straddling key in this row that still fall above the boundary
      below[b] = row < R ? sh.above[b][row] + max(0, min(equal, quota_b[b] - pre[h][b])) : 0;
    }
    n[h][0] = (below[2] - below[1]) * factor + (prefix_phase == 0 ? p : 0);  // NVFP4
    n[h][1] = (below[1] - below[0]) * factor + (prefix_phase == 1 ? p : 0);  // INT8
    n[h][2] = below[0] * factor + (prefix_phase == 2 ? p : 0);               // FP16
    total[h] = row < R ? n[h][0] + n[h][1] + n[h][2] : -1;
    int incl = max(total[h], 0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    offset[h] = carry[3] + incl - max(total[h], 0);
    carry[3] += __shfl_sync(0xffffffffu, incl, 31);
    if (warp == h && row < R) {
      row_offset[(int64_t)head * R + row] = offset[h];
      int32_t* rc = row_counts + ((int64_t)head * R + row) * 4;
#pragma unroll
      for (int b = 0; b < 3; ++b) rc[b] = n[h][b];
      if (kPairs) rc[3] = 0;
    }
  }
  // A row's own numbers (row0 is even: the rows of a warp lie in one half)
  const int half = kCols == 2 && row0 >= 32 ? 1 : 0;
  const auto of_row = [&](const int (&v)[kCols], int row) {
    return __shfl_sync(0xffffffffu, kCols == 2 && half ? v[kCols - 1] : v[0], row & 31);
  };
  int mine[kRows][3], run[kRows][3], len[kRows], at0[kRows];
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      int v[kCols], w[kCols];
#pragma unroll
      for (int h = 0; h < kCols; ++h) {
        v[h] = n[h][b];
        w[h] = pre[h][b];
      }
      mine[r][b] = of_row(v, row0 + r);
      run[r][b] = of_row(w, row0 + r);
    }
    len[r] = of_row(total, row0 + r);
    at0[r] = of_row(offset, row0 + r);
  }
  if constexpr (!kPairs) {
    // ---- launch order: longest list first, ties by block index, as block + 1 in the fourth entry of the
    // position's counts ----
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      int rank = 0;
#pragma unroll
      for (int h = 0; h < kCols; ++h)
        rank += __popc(__ballot_sync(0xffffffffu, total[h] > len[r] || (total[h] == len[r] && h * 32 + lane < row0 + r)));
      if (lane == 0 && row0 + r < R) row_counts[((int64_t)head * R + rank) * 4 + 3] = row0 + r + 1;
    }
  }
  const bool active[3] = {b2 > b1, b1 > b0, b0 > 0};  // phases with a budget
  // ---- lists ----
  if constexpr (!kPairs) {
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      if (len[r] <= 0 || (int64_t)at0[r] + len[r] > capacity) continue;  // (the latter cannot happen with exact budgets)
      int32_t* list = stage_ids + (int64_t)head * capacity + at0[r];
      const int n0 = mine[r][0], n1 = mine[r][1];
      int at[3] = {prefix_phase == 0 ? p : 0, n0 + (prefix_phase == 1 ? p : 0), n0 + n1 + (prefix_phase == 2 ? p : 0)};
      if (prefix_phase >= 0) {
        const int seg = prefix_phase == 0 ? 0 : (prefix_phase == 1 ? n0 : n0 + n1);
        for (int k = lane; k < p; k += 32) list[seg + k] = k;
      }
#pragma unroll
      for (int c = 0; c < kCols; ++c) {
        const int stage = prefix_stages + (c * 32 + lane) * factor;
        const int code = fused_code(key[r][c], key_b, quota_b, run[r], lower);
#pragma unroll
        for (int k = 1; k <= 3; ++k) {
          if (!active[k - 1]) continue;
          const unsigned members = __ballot_sync(0xffffffffu, code == k);
          if (code == k) {
            int32_t* dst = list + at[k - 1] + __popc(members & lower) * factor;
            dst[0] = stage;
            if (factor == 2) dst[1] = stage + 1;
          }
          at[k - 1] += __popc(members) * factor;
        }
      }
    }
  } else {
    // One pair after the other (blocks 2t and 2t + 1): as in the kernel above
    const int pairs_all = (R + 1) / 2;
#pragma unroll
    for (int r = 0; r < kRows; r += 2) {
      const int a = row0 + r;
      if (a >= R) continue;
      const bool has_b = a + 1 < R;
      const int n0 = mine[r][0] + (has_b ? mine[r + 1][0] : 0), n1 = mine[r][1] + (has_b ? mine[r + 1][1] : 0);
      const bool fits = (int64_t)at0[r] + len[r] + (has_b ? len[r + 1] : 0) <= capacity;
      int32_t* list = pair_ids + (int64_t)head * capacity + at0[r];
      const int start[3] = {0, n0, n0 + n1};
      int at[3] = {start[0], start[1], start[2]};
      const int both = has_b ? (int)0xc0000000u : 1 << 30;
      if (prefix_phase >= 0) {
        if (fits)
          for (int k = lane; k < p; k += 32) list[start[prefix_phase] + k] = k | both;
        at[0] += prefix_phase == 0 ? p : 0;
        at[1] += prefix_phase == 1 ? p : 0;
        at[2] += prefix_phase == 2 ? p : 0;
      }
#pragma unroll
      for (int c = 0; c < kCols; ++c) {
        const int stage = prefix_stages + c * 32 + lane;
        const int ca = fused_code(key[r][c], key_b, quota_b, run[r], lower);
        const int cb = fused_code(key[r + 1][c], key_b, quota_b, run[r + 1], lower);
#pragma unroll
        for (int k = 1; k <= 3; ++k) {
          if (!active[k - 1]) continue;
          const bool in = ca == k || cb == k;
          const unsigned members = __ballot_sync(0xffffffffu, in);
          if (in && fits)
            list[at[k - 1] + __popc(members & lower)] = stage | (ca == k ? 1 << 30 : 0) | (cb == k ? (int)(1u << 31) : 0);
          at[k - 1] += __popc(members);
        }
      }
      if (lane == 0) {
        int32_t* pc = pair_counts + ((int64_t)head * pairs_all + a / 2) * 4;
#pragma unroll
        for (int b = 0; b < 3; ++b) pc[b] = at[b] - start[b];
        sh.unions[a / 2] = at[0] + at[1] + at[2] - start[1] - start[2];
      }
    }
    __syncthreads();
    const int mine_union = lane < pairs_all ? sh.unions[lane] : -1;
#pragma unroll
    for (int r = 0; r < kRows; r += 2) {
      const int t = (row0 + r) / 2, length = t < pairs_all ? sh.unions[t] : 0;
      const int rank = __popc(__ballot_sync(0xffffffffu, mine_union > length || (mine_union == length && lane < t)));
      if (lane == 0 && t < pairs_all) pair_counts[((int64_t)head * pairs_all + rank) * 4 + 3] = t + 1;
    }
  }
}

template <bool kPairs, int kDraft>
int launch_short(const anemoi_sm100_shape& s, const DraftPools& draft, const void* probability, int64_t n16, int64_t n8,
                 int64_t n4, int prefix_phase, int32_t* row_offset, int32_t* row_counts, int32_t* stage_ids,
                 int64_t capacity, int32_t* pair_counts, int32_t* pair_ids, cudaStream_t st) {
  const int R = s.video_blocks;
  const size_t smem = (size_t)draft_words(kDraft, kDraft ? draft.maps : 0) * 4;
  auto kernel = route_short_kernel<1, kPairs, kDraft>;
  if constexpr (kDraft == 0)
    if (R > 32) kernel = route_short_kernel<2, kPairs, 0>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return ANEMOI_SM100_ELAUNCH;
  return layer::launch(kernel, dim3(s.heads), dim3(kShortThreads), smem, st, draft,
                       static_cast<const unsigned short*>(probability), R, (int)n16, (int)(n16 + n8),
                       (int)(n16 + n8 + n4), s.query_block / 64, rec::prefix_stages(s), prefix_phase, capacity,
                       row_offset, row_counts, stage_ids, pair_counts, pair_ids) == cudaSuccess
             ? ANEMOI_SM100_OK
             : ANEMOI_SM100_ELAUNCH;
}

// One warp per row writes the row's bits instead, for the choice of the Q64 pairs (match.cu).
__global__ void __launch_bounds__(kRowWarps * 32) emit_bits_kernel(const unsigned short* prob, int R, const int* thr,
                                                                   const int* stat, const layer::PairBits bits) {
  const int row = blockIdx.x * kRowWarps + (threadIdx.x >> 5), head = blockIdx.y;
  if (row >= R) return;
  const int lane = threadIdx.x & 31;
  const unsigned lower = (1u << lane) - 1u;
  int key_b[3], quota_b[3], run[3];
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    key_b[b] = thr[head * 8 + 2 * b];
    quota_b[b] = thr[head * 8 + 2 * b + 1];
    run[b] = stat[((int64_t)head * R + row) * kStat + 3 + b];
  }
  const int words = (R + 31) / 32, stride = layer::pair_bit_words(R);
  RowBits out = row_bits(bits, head, R, row, stride);
  const unsigned short* src = prob + ((int64_t)head * R + row) * R;
  for (int w = 0; w < words; ++w) {
    const int j = w * 32 + lane;
    const int c = fused_code(j < R ? (__ldg(src + j) & 0x7fff) : -2, key_b, quota_b, run, lower);
#pragma unroll
    for (int k = 1; k <= 3; ++k) out.put(k - 1, w, __ballot_sync(0xffffffffu, c == k));
    out.flush(w, words, stride);
  }
}

// Q64 query blocks 2t and 2t+1 of a head run as one CTA of the attention kernel (rows 0-63 and
// 64-127 of the 128-row MMA shape).  That CTA walks, phase by phase, the union of the two
// blocks' lists; bits 30 and 31 of an entry say which of the two blocks the stage belongs to.
// One warp per pair, one lane per phase (a two-pointer merge of two ascending lists).  The union
// of phase c is written where the two blocks' phases before c would end, inside the space the two
// lists occupy in the stage list (a buffer of the same capacity), so no offsets are scanned.
// The pairs of a head are then ranked longest first, like the blocks.
__global__ void __launch_bounds__(kRowWarps * 32) pair_kernel(int R, int64_t capacity,
                                                              const int32_t* row_offset,
                                                              const int32_t* row_counts,
                                                              const int32_t* stage_ids,
                                                              int32_t* pair_counts,
                                                              int32_t* pair_ids) {
  const int pairs = (R + 1) / 2;
  const int pair = blockIdx.x * kRowWarps + (threadIdx.x >> 5), head = blockIdx.y;
  if (pair >= pairs) return;
  const int lane = threadIdx.x & 31;
  const int a = 2 * pair;
  const bool has_b = a + 1 < R;
  const int32_t* ca = row_counts + ((int64_t)head * R + a) * 4;
  const int64_t base = row_offset[(int64_t)head * R + a];
  const int32_t* la = stage_ids + (int64_t)head * capacity + base;
  const int32_t* lb = la + (ca[0] + ca[1] + ca[2]);  // lists follow one another in row order
  int32_t* out = pair_ids + (int64_t)head * capacity + base;
  int n = 0;
  if (lane < 3) {
    int sa = 0, sb = 0, so = 0;  // starts of this lane's phase in A, in B and in the union
    for (int c = 0; c < lane; ++c) {
      sa += ca[c];
      sb += has_b ? ca[4 + c] : 0;
    }
    so = sa + sb;
    const int na = ca[lane], nb = has_b ? ca[4 + lane] : 0;
    int i = 0, j = 0;
    while (i < na || j < nb) {
      const int x = i < na ? la[sa + i] : INT_MAX;
      const int y = j < nb ? lb[sb + j] : INT_MAX;
      const int v = min(x, y);
      out[so + n++] = v | (x == v ? 1 << 30 : 0) | (y == v ? (int)(1u << 31) : 0);
      i += x == v;
      j += y == v;
    }
  }
  if (lane < 4) pair_counts[((int64_t)head * pairs + pair) * 4 + lane] = lane < 3 ? n : 0;
}

// Launch order of a head's pairs: longest union first (ties by pair index), as for the blocks.
__global__ void __launch_bounds__(1024) pair_order_kernel(int pairs, int32_t* pair_counts) {
  __shared__ int total_s[kOrderMaxBlocks];
  const int head = blockIdx.x;
  int32_t* pc = pair_counts + (int64_t)head * pairs * 4;
  for (int i = threadIdx.x; i < pairs; i += 1024) total_s[i] = pc[i * 4] + pc[i * 4 + 1] + pc[i * 4 + 2];
  __syncthreads();
  for (int i = threadIdx.x; i < pairs; i += 1024) {
    const int mine = total_s[i];
    int rank = 0;
    for (int j = 0; j < pairs; ++j) rank += (total_s[j] > mine) || (total_s[j] == mine && j < i);
    pc[rank * 4 + 3] = i + 1;
  }
}

// The launches in front of the lists where routing takes several kernels: histogram, boundaries, per-row counts, and
// the scans over the rows with the lists' offsets and (`ordered`) the launch order.
int rank_rows(const anemoi_sm100_shape& s, const void* probability, int64_t n16, int64_t n8, int64_t n4,
              int prefix_phase, bool ordered, void* scratch, int32_t* row_offset, int32_t* row_counts, RouteScratch& sc,
              cudaStream_t st) {
  const int H = s.heads, R = s.video_blocks;
  const int64_t items = (int64_t)R * R;
  sc.hist = static_cast<int*>(scratch);
  sc.thr = sc.hist + (int64_t)H * kBins;
  sc.stat = sc.thr + (int64_t)H * 8;
  if (cudaMemsetAsync(sc.hist, 0, (size_t)H * kBins * 4, st) != cudaSuccess)
    return ANEMOI_SM100_ELAUNCH;
  const unsigned short* prob = static_cast<const unsigned short*>(probability);
  // Function attributes belong to a device: the opt-in is made at every call (a cheap host-side
  // driver call), so a process that routes on several GPUs, or from several host threads,
  // never launches the kernel without the opt-in for its dynamic shared memory.
  if (cudaFuncSetAttribute(hist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kHalfBins * 4) !=
      cudaSuccess)
    return ANEMOI_SM100_ELAUNCH;
  // about two waves of histogram CTAs per key-range half, each with at least 8192 items
  const int chunks = (int)max((int64_t)1, min(min((int64_t)16, items / 8192), (int64_t)((296 + H / 2) / H)));
  const int factor = s.query_block / 64, prefix_stages = rec::prefix_stages(s);
  const dim3 rows((R + kRowWarps - 1) / kRowWarps, H);
  hist_kernel<<<dim3(chunks, H, 2), kHistThreads, kHalfBins * 4, st>>>(prob, items, chunks, sc.hist);
  threshold_kernel<<<H, 1024, 0, st>>>(sc.hist, nullptr, sc.thr, 8, 0, n16, n16 + n8, n16 + n8 + n4);
  rowstat_kernel<<<rows, kRowWarps * 32, 0, st>>>(prob, R, sc.thr, sc.stat);
  headscan_kernel<<<H, 1024, 0, st>>>(R, sc.thr, sc.stat, factor, prefix_stages, prefix_phase, ordered,
                                      row_offset, row_counts);
  return cudaGetLastError() == cudaSuccess ? ANEMOI_SM100_OK : ANEMOI_SM100_ELAUNCH;
}

}  // namespace

bool layer::routes_pairs(const anemoi_sm100_shape& s) {
  return fused_fits(s.heads, s.video_blocks) && rec::stages(s) < (1 << 30);
}

extern "C" int64_t anemoi_sm100_route_anchored_scratch_bytes(const anemoi_sm100_shape* shape) {
  if (rec::validate_shape(shape) != ANEMOI_SM100_OK) return ANEMOI_SM100_EINVAL;
  return (int64_t)shape->heads * (2 * kBins + 16 + kAnchorStat * (int64_t)shape->video_blocks) * 4;
}

extern "C" int anemoi_sm100_route_anchored(const anemoi_sm100_shape* shape, const void* probability,
                                           int64_t n16, int64_t n8, int64_t n4, int prefix_phase,
                                           const uint8_t* anchors, const int32_t* anchor_ids,
                                           int32_t anchor_count, void* scratch, int64_t scratch_bytes,
                                           int32_t* row_offset, int32_t* row_counts,
                                           int32_t* stage_ids, int64_t list_capacity, void* stream) {
  if (rec::validate_shape(shape) != ANEMOI_SM100_OK || !probability || !scratch || !row_offset ||
      !row_counts || !stage_ids || !anchors || !anchor_ids || anchor_count <= 0)
    return ANEMOI_SM100_EINVAL;
  const int H = shape->heads, R = shape->video_blocks;
  const int64_t items = (int64_t)R * R, retained = n16 + n8 + n4;
  if (n16 < 0 || n8 < 0 || n4 < 0 || retained > items || retained <= 0) return ANEMOI_SM100_EINVAL;
  // as the reference: the anchors must fit into the lowest active precision
  const int64_t lowest = n4 ? n4 : (n8 ? n8 : n16);
  if (anchor_count > lowest) return ANEMOI_SM100_EINVAL;
  if (prefix_phase < -1 || prefix_phase > 2) return ANEMOI_SM100_EINVAL;
  if (prefix_phase >= 0 && shape->prefix_tokens == 0) prefix_phase = -1;
  if (scratch_bytes < anemoi_sm100_route_anchored_scratch_bytes(shape)) return ANEMOI_SM100_EINVAL;
  if (list_capacity < anemoi_sm100_route_list_capacity(shape, n16, n8, n4, prefix_phase))
    return ANEMOI_SM100_EINVAL;
  if (R > 65535 || items * H >= (1ll << 40)) return ANEMOI_SM100_ELIMIT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int* hist = static_cast<int*>(scratch);
  int* hist_anchor = hist + (int64_t)H * kBins;
  int* thr = hist_anchor + (int64_t)H * kBins;
  int* stat = thr + (int64_t)H * 16;
  if (cudaMemsetAsync(hist, 0, (size_t)H * kBins * 8, st) != cudaSuccess) return ANEMOI_SM100_ELAUNCH;
  if (cudaFuncSetAttribute(hist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kHalfBins * 4) !=
      cudaSuccess)
    return ANEMOI_SM100_ELAUNCH;
  const unsigned short* prob = static_cast<const unsigned short*>(probability);
  const int chunks = (int)max((int64_t)1, min(min((int64_t)16, items / 8192), (int64_t)((296 + H / 2) / H)));
  const int factor = shape->query_block / 64, prefix_stages = rec::prefix_stages(*shape);
  const int lowest_code = n4 ? 1 : (n8 ? 2 : 3);
  const dim3 rows((R + kRowWarps - 1) / kRowWarps, H);
  hist_kernel<<<dim3(chunks, H, 2), kHistThreads, kHalfBins * 4, st>>>(prob, items, chunks, hist);
  anchor_hist_kernel<<<dim3((anchor_count + 255) / 256, H), 256, 0, st>>>(prob, items, anchor_ids,
                                                                           anchor_count, hist_anchor);
  threshold_kernel<<<H, 1024, 0, st>>>(hist, nullptr, thr, 16, 0, n16, n16 + n8, retained);
  const int64_t others = retained - anchor_count;  // pairs kept that are not anchors
  threshold_kernel<<<H, 1024, 0, st>>>(hist, hist_anchor, thr, 16, 8, others, others, others);
  anchor_rowstat_kernel<<<rows, kRowWarps * 32, 0, st>>>(prob, anchors, R, thr, stat);
  anchor_tiescan_kernel<<<H, 1024, 0, st>>>(R, stat);
  anchor_count_kernel<<<rows, kRowWarps * 32, 0, st>>>(prob, anchors, R, thr, stat, lowest_code,
                                                       row_counts);
  anchor_offsets_kernel<<<H, 1024, 0, st>>>(R, factor, prefix_stages, prefix_phase, row_offset,
                                            row_counts);
  anchor_emit_kernel<<<rows, kRowWarps * 32, 0, st>>>(prob, anchors, R, thr, stat, lowest_code, factor,
                                                      prefix_stages, prefix_phase, list_capacity,
                                                      row_offset, row_counts, stage_ids);
  return cudaGetLastError() == cudaSuccess ? ANEMOI_SM100_OK : ANEMOI_SM100_ELAUNCH;
}

extern "C" int anemoi_sm100_pair_lists(const anemoi_sm100_shape* shape, const int32_t* row_offset,
                                       const int32_t* row_counts, const int32_t* stage_ids,
                                       int64_t list_capacity, int32_t* pair_counts,
                                       int32_t* pair_ids, void* stream) {
  if (rec::validate_shape(shape) != ANEMOI_SM100_OK || !row_offset || !row_counts || !stage_ids ||
      !pair_counts || !pair_ids || list_capacity <= 0 || shape->query_block != 64)
    return ANEMOI_SM100_EINVAL;
  if (rec::stages(*shape) >= (1 << 30)) return ANEMOI_SM100_ELIMIT;  // two flag bits per entry
  const int R = shape->video_blocks, H = shape->heads, pairs = (R + 1) / 2;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  pair_kernel<<<dim3((pairs + kRowWarps - 1) / kRowWarps, H), kRowWarps * 32, 0, st>>>(
      R, list_capacity, row_offset, row_counts, stage_ids, pair_counts, pair_ids);
  if (pairs <= kOrderMaxBlocks) pair_order_kernel<<<H, 1024, 0, st>>>(pairs, pair_counts);
  return cudaGetLastError() == cudaSuccess ? ANEMOI_SM100_OK : ANEMOI_SM100_ELAUNCH;
}

extern "C" int64_t anemoi_sm100_route_scratch_bytes(const anemoi_sm100_shape* shape) {
  if (rec::validate_shape(shape) != ANEMOI_SM100_OK) return ANEMOI_SM100_EINVAL;
  return scratch_ints(shape->heads, shape->video_blocks) * 4;
}

extern "C" int64_t anemoi_sm100_route_list_capacity(const anemoi_sm100_shape* shape, int64_t n16,
                                                    int64_t n8, int64_t n4, int prefix_phase) {
  if (rec::validate_shape(shape) != ANEMOI_SM100_OK) return ANEMOI_SM100_EINVAL;
  const int64_t f = shape->query_block / 64;
  const int64_t p = prefix_phase >= 0 ? rec::prefix_stages(*shape) : 0;
  return (n16 + n8 + n4) * f + (int64_t)shape->video_blocks * p;
}

extern "C" int anemoi_sm100_route(const anemoi_sm100_shape* shape, const void* probability,
                                  int64_t n16, int64_t n8, int64_t n4, int prefix_phase,
                                  void* scratch, int64_t scratch_bytes, int32_t* row_offset,
                                  int32_t* row_counts, int32_t* stage_ids, int64_t list_capacity,
                                  void* stream) {
  if (rec::validate_shape(shape) != ANEMOI_SM100_OK || !probability || !scratch || !row_offset ||
      !row_counts || !stage_ids)
    return ANEMOI_SM100_EINVAL;
  const int H = shape->heads, R = shape->video_blocks;
  const int64_t items = (int64_t)R * R;
  if (n16 < 0 || n8 < 0 || n4 < 0 || n16 + n8 + n4 > items || n16 + n8 + n4 <= 0)
    return ANEMOI_SM100_EINVAL;
  if (prefix_phase < -1 || prefix_phase > 2) return ANEMOI_SM100_EINVAL;
  if (prefix_phase >= 0 && shape->prefix_tokens == 0) prefix_phase = -1;
  if (scratch_bytes < scratch_ints(H, R) * 4) return ANEMOI_SM100_EINVAL;
  if (list_capacity < anemoi_sm100_route_list_capacity(shape, n16, n8, n4, prefix_phase))
    return ANEMOI_SM100_EINVAL;
  if (R > 65535 || items * H >= (1ll << 40)) return ANEMOI_SM100_ELIMIT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (R <= kShortBlocks)
    return launch_short<false, 0>(*shape, DraftPools{}, probability, n16, n8, n4, prefix_phase, row_offset, row_counts,
                                  stage_ids, list_capacity, nullptr, nullptr, st);
  if (fused_fits(H, R))
    return launch_fused<kLists>(*shape, probability, n16, n8, n4, prefix_phase, row_offset, row_counts, stage_ids,
                               list_capacity, nullptr, nullptr, st);
  RouteScratch sc;
  const int code = rank_rows(*shape, probability, n16, n8, n4, prefix_phase, true, scratch, row_offset, row_counts, sc, st);
  if (code != ANEMOI_SM100_OK) return code;
  emit_kernel<<<dim3((R + kRowWarps - 1) / kRowWarps, H), kRowWarps * 32, 0, st>>>(
      static_cast<const unsigned short*>(probability), R, sc.thr, sc.stat, shape->query_block / 64,
      rec::prefix_stages(*shape), prefix_phase, list_capacity, row_offset, row_counts, stage_ids);
  return cudaGetLastError() == cudaSuccess ? ANEMOI_SM100_OK : ANEMOI_SM100_ELAUNCH;
}

extern "C" int anemoi_sm100_route_pairs(const anemoi_sm100_shape* shape, const void* probability, int64_t n16,
                                        int64_t n8, int64_t n4, int prefix_phase, int32_t* row_offset,
                                        int32_t* row_counts, int32_t* pair_counts, int32_t* pair_ids,
                                        int64_t list_capacity, void* stream) {
  if (rec::validate_shape(shape) != ANEMOI_SM100_OK || !probability || !row_offset || !row_counts ||
      !pair_counts || !pair_ids || shape->query_block != 64)
    return ANEMOI_SM100_EINVAL;
  const int64_t items = (int64_t)shape->video_blocks * shape->video_blocks;
  if (n16 < 0 || n8 < 0 || n4 < 0 || n16 + n8 + n4 > items || n16 + n8 + n4 <= 0)
    return ANEMOI_SM100_EINVAL;
  if (prefix_phase < -1 || prefix_phase > 2) return ANEMOI_SM100_EINVAL;
  if (prefix_phase >= 0 && shape->prefix_tokens == 0) prefix_phase = -1;
  if (list_capacity < anemoi_sm100_route_list_capacity(shape, n16, n8, n4, prefix_phase))
    return ANEMOI_SM100_EINVAL;
  if (!fused_fits(shape->heads, shape->video_blocks) || rec::stages(*shape) >= (1 << 30)) return ANEMOI_SM100_ELIMIT;
  if (shape->video_blocks <= kShortBlocks)
    return launch_short<true, 0>(*shape, DraftPools{}, probability, n16, n8, n4, prefix_phase, row_offset, row_counts,
                                 nullptr, list_capacity, pair_counts, pair_ids, static_cast<cudaStream_t>(stream));
  return launch_fused<kNeighbours>(*shape, probability, n16, n8, n4, prefix_phase, row_offset, row_counts, nullptr,
                            list_capacity, pair_counts, pair_ids, static_cast<cudaStream_t>(stream));
}

int layer::route_bits(const anemoi_sm100_shape& s, const void* probability, int64_t n16, int64_t n8, int64_t n4,
                      int prefix_phase, void* scratch, int32_t* row_offset, int32_t* row_counts, const PairBits& bits,
                      int64_t capacity, cudaStream_t st) {
  // (the conditions of draft_probability's map, route and pair_lists)
  const int H = s.heads, R = s.video_blocks;
  const int64_t items = (int64_t)R * R;
  if (n16 < 0 || n8 < 0 || n4 < 0 || n16 + n8 + n4 > items || n16 + n8 + n4 <= 0) return ANEMOI_SM100_EINVAL;
  if (prefix_phase < -1 || prefix_phase > 2) return ANEMOI_SM100_EINVAL;
  if (capacity < anemoi_sm100_route_list_capacity(&s, n16, n8, n4, prefix_phase)) return ANEMOI_SM100_EINVAL;
  if (fused_fits(H, R))
    return launch_fused<kBits>(s, probability, n16, n8, n4, prefix_phase, row_offset, row_counts,
                                  nullptr, 0, nullptr, nullptr, st, bits);
  RouteScratch sc;
  const int code = rank_rows(s, probability, n16, n8, n4, prefix_phase, false, scratch, row_offset, row_counts, sc, st);
  if (code != ANEMOI_SM100_OK) return code;
  emit_bits_kernel<<<dim3((R + kRowWarps - 1) / kRowWarps, H), kRowWarps * 32, 0, st>>>(
      static_cast<const unsigned short*>(probability), R, sc.thr, sc.stat, bits);
  return cudaGetLastError() == cudaSuccess ? ANEMOI_SM100_OK : ANEMOI_SM100_ELAUNCH;
}

bool layer::drafts_in_routing(const anemoi_sm100_shape& s) {
  // (one CTA per head, and one kernel for lists and pairs, whatever the number of heads)
  static_assert(kDraftBlocks == 32 && 2 * kShortWarps >= kDraftBlocks, "a column per lane, two rows per warp");
  return s.prefix_tokens == 0 && s.video_blocks <= kDraftBlocks;
}

int layer::draft_and_route(const anemoi_sm100_shape& s, const anemoi_sm100_operands& ops, float maxpool_weight,
                           void* probability, int64_t n16, int64_t n8, int64_t n4, int prefix_phase,
                           int32_t* row_offset, int32_t* row_counts, int32_t* stage_ids, int32_t* pair_counts,
                           int32_t* pair_ids, int64_t capacity, cudaStream_t st) {
  // (the conditions of draft_probability, route and route_pairs)
  const int64_t items = (int64_t)s.video_blocks * s.video_blocks;
  const bool pairs = pair_counts != nullptr;
  if (!ops.q_pool || !ops.k_pool || !probability || !row_offset || !row_counts || !(pairs ? pair_ids : stage_ids))
    return ANEMOI_SM100_EINVAL;
  if (!(maxpool_weight >= 0.0f && maxpool_weight <= 1.0f)) return ANEMOI_SM100_EINVAL;
  if (maxpool_weight != 0.0f && (!ops.q_max_pool || !ops.k_max_pool)) return ANEMOI_SM100_EINVAL;
  if (n16 < 0 || n8 < 0 || n4 < 0 || n16 + n8 + n4 > items || n16 + n8 + n4 <= 0) return ANEMOI_SM100_EINVAL;
  if (prefix_phase < -1 || prefix_phase > 2) return ANEMOI_SM100_EINVAL;
  if (prefix_phase >= 0 && s.prefix_tokens == 0) prefix_phase = -1;
  if (capacity < anemoi_sm100_route_list_capacity(&s, n16, n8, n4, prefix_phase)) return ANEMOI_SM100_EINVAL;
  DraftPools d = {};
  const bool most = maxpool_weight == 1.0f;  // max pools only
  d.q[0] = static_cast<const __half*>(most ? ops.q_max_pool : ops.q_pool);
  d.k[0] = static_cast<const __half*>(most ? ops.k_max_pool : ops.k_pool);
  d.q[1] = static_cast<const __half*>(ops.q_max_pool);
  d.k[1] = static_cast<const __half*>(ops.k_max_pool);
  d.maps = maxpool_weight != 0.0f && !most ? 2 : 1;
  d.weight = maxpool_weight;
  d.map = static_cast<unsigned short*>(probability);
#define ANEMOI_LAUNCH(PAIRS, D)                                                                                      \
  launch_short<PAIRS, D>(s, d, probability, n16, n8, n4, prefix_phase, row_offset, row_counts, stage_ids, capacity, \
                         pair_counts, pair_ids, st)
  if (pairs) return s.head_dim == 64 ? ANEMOI_LAUNCH(true, 64) : ANEMOI_LAUNCH(true, 128);
  return s.head_dim == 64 ? ANEMOI_LAUNCH(false, 64) : ANEMOI_LAUNCH(false, 128);
#undef ANEMOI_LAUNCH
}

// ------------------------------------------------------------------------------------------
// Routing without any allocation by the caller
// ------------------------------------------------------------------------------------------
// Some hosts of this library cannot hand it scratch memory: a serving loop whose memory
// pool is frozen after start-up, or code that must not call cudaMalloc because it runs
// between other streams' work and cannot afford the implicit device synchronisation.
// For them the scratch of anemoi_sm100_route lives in this file-scope device array.
// Every GPU that loads the library holds these 8 MiB until the process exits.
constexpr int64_t kStaticScratchInts = 2 * 1024 * 1024;  // 8 MiB of int32
static __device__ __align__(256) int g_route_scratch[kStaticScratchInts];

namespace {
constexpr int kMaxDevices = 64;
int* g_route_scratch_address[kMaxDevices];  // device address of the array, per device ordinal
}  // namespace

extern "C" int64_t anemoi_sm100_route_static_max_bytes(void) { return kStaticScratchInts * 4; }

extern "C" int anemoi_sm100_route_static(const anemoi_sm100_shape* shape, const void* probability,
                                         int64_t n16, int64_t n8, int64_t n4, int prefix_phase,
                                         int32_t* row_offset, int32_t* row_counts,
                                         int32_t* stage_ids, int64_t list_capacity,
                                         void* stream) {
  if (rec::validate_shape(shape) != ANEMOI_SM100_OK) return ANEMOI_SM100_EINVAL;
  const int64_t need = scratch_ints(shape->heads, shape->video_blocks);
  if (need > kStaticScratchInts) return ANEMOI_SM100_ELIMIT;  // heads*(32776 + 6*blocks) ints
  int device = -1;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kMaxDevices)
    return ANEMOI_SM100_ELAUNCH;
  // In host code the array's name is only a stand-in for the symbol, not a device address.
  // The address is looked up once per device, with that device current (the first call on
  // a device does it, so make that call before any stream capture), and then reused.
  int* scratch = g_route_scratch_address[device];
  if (scratch == nullptr) {
    if (cudaGetSymbolAddress(reinterpret_cast<void**>(&scratch), g_route_scratch) != cudaSuccess ||
        scratch == nullptr)
      return ANEMOI_SM100_ELAUNCH;
    g_route_scratch_address[device] = scratch;
  }
  // Same kernels as anemoi_sm100_route; the bins that must start at zero are cleared there on
  // `stream` at every call, the rest is overwritten before it is read.
  return anemoi_sm100_route(shape, probability, n16, n8, n4, prefix_phase, scratch, need * 4,
                            row_offset, row_counts, stage_ids, list_capacity, stream);
}
