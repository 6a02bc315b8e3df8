// Apps over directed graphs: symbiosity (apps/symbiosity.cpp) and the n_path
// breadth-first search (apps/n_path.cpp).
//
// symbiosity: for each row i, out(i) (the row matrix) is intersected with in(i)
// (the column matrix) and the Jaccard ratio tested as symbiosity.cpp:46-58 does in
// double precision (here exactly, in integers).  Short rows take a lane each, longer
// ones a warp; rows too long for a warp (hubs) are listed first and taken one per CTA, a
// slice per warp.
//
// n_path: level-synchronous BFS on a visited bitset of (n + 64) / 64 words,
// the reference's bs_size (n_path.cpp:45-53).  A level is two launches:
//   expand  ORs the frontier's rows into `seen`, which starts as the visited set
//           (set_union, union.hpp:6-127); a bitset row is ORed word by word;
//   collect takes seen AND NOT visited as the new frontier (set_difference,
//           difference.hpp:5-84) and merges it into visited.
// Frontier rows longer than kBfsHeavy entries are split over the warps of the
// grid, rows above kBfsGroup over a CTA, and shorter ones take 8 lanes.  Levels are launched
// kBfsChunk at a time: each kernel reads its frontier size from device memory
// and does nothing once a frontier is empty, so the host checks the sizes
// once per chunk instead of once per level.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#include "eh_internal.h"
#include "eh_kernels.cuh"
#include "eh_matrix.cuh"

namespace eh {
namespace {

constexpr uint32_t kBfsHeavy = 4096;
constexpr uint32_t kBfsGroup = 256;
constexpr uint32_t kBfsListed = 1024;
constexpr uint32_t kBfsChunk = 8;
constexpr int kBfsThreads = 256;

// A row pair whose intersection is too long for one warp: streamed side (the
// smaller row) above kSymLight entries (two uint rows of sizes within 32x: the
// larger above kSymMerge), or two bitsets sharing more than 8 * kSymLight words.  Such rows go
// to a list that whole CTAs work through.
constexpr uint32_t kSymLight = 256;
constexpr uint32_t kSymMerge = 2048;

__device__ __forceinline__ bool sym_heavy(const RowView& A, const RowView& B) {
  if (!A.card || !B.card) return false;
  if (A.type == TY_BITSET && B.type == TY_BITSET) {
    const int64_t lo = max(A.aux, B.aux), hi = min((int64_t)A.aux + A.len, (int64_t)B.aux + B.len);
    return hi - lo > 8 * (int64_t)kSymLight;
  }
  const uint32_t lo = min(A.card, B.card), hi = max(A.card, B.card);
  if (A.type == TY_UINT && B.type == TY_UINT && hi <= 32u * lo) return hi > kSymMerge;
  return lo > kSymLight;
}

constexpr uint32_t kSymChunk = 32;  // rows a warp takes per grab (one per lane)
constexpr uint32_t kSymTiny = 32;   // uint rows a single lane intersects by merging

// The test both / (|A| + |B| - both) > threshold, the quotient rounded to double
// as the reference rounds it, without FP64 (a division took 30-odd instructions of
// a pipe with two lanes per SM: two divisions a row were 170 us for 2^21 rows).  For
// 2^-30 <= threshold < 1, threshold = m 2^-s' with 2^52 <= m < 2^53, the rounded
// quotient is above it when the quotient is above the middle (2m + 1) 2^-(s' + 1) to
// the next double, or on it when that rounds up (m odd, ties to even): an exact
// 128-bit comparison of both 2^shift with m2 (|A| + |B| - both).
struct SymTest {
  double threshold;
  unsigned long long m2;  // 2m + 1, 0: outside the range above
  int shift;              // s' + 1: 54 .. 84
  bool tie;               // m odd
};
SymTest sym_test(double threshold) {
  SymTest t{threshold, 0, 0, false};
  if (threshold >= 0x1p-30 && threshold < 1.0) {
    int e = 0;
    const unsigned long long m = (unsigned long long)std::ldexp(std::frexp(threshold, &e), 53);
    t.m2 = 2 * m + 1;
    t.shift = 53 - e + 1;
    t.tie = m & 1;
  }
  return t;
}
__device__ __forceinline__ bool sym_above(uint32_t both, const RowView& A, const RowView& B, const SymTest& t) {
  const unsigned long long all = (unsigned long long)A.card + B.card - both;
  if (!t.m2) return (double)both / (double)all > t.threshold;  // 0 / 0 is NaN, above nothing (as in the reference)
  if (!both) return false;
  const unsigned long long rl = t.m2 * all, rh = __umul64hi(t.m2, all);
  // shift is 54 .. 84: both << shift as two words.
  const unsigned long long ll = t.shift < 64 ? (unsigned long long)both << t.shift : 0ull;
  const unsigned long long lh = t.shift < 64 ? (unsigned long long)both >> (64 - t.shift)
                                             : (unsigned long long)both << (t.shift - 64);
  return lh != rh ? lh > rh : ll != rl ? ll > rl : t.tie;
}

// |A ∩ B| of two sorted uint rows by one thread (a merge).
__device__ __forceinline__ uint32_t merge_count(const uint32_t* a, uint32_t na, const uint32_t* b, uint32_t nb) {
  uint32_t i = 0, j = 0, c = 0;
  while (i < na && j < nb) {
    const uint32_t x = a[i], y = b[j];
    c += x == y;
    i += x <= y;
    j += y <= x;
  }
  return c;
}

// Per-lane part of |A ∩ B| of two ascending uint lists, by a warp.  A block of 32
// entries of each list is held one per lane; each a is looked up in the b block
// by a binary search over the lanes (shuffles), then the block with the smaller
// last entry is replaced (both when equal), so that overlapping blocks meet
// exactly once.  Loads are coalesced and
// the next three blocks of each list are in flight; a merge path per lane read
// one entry at a time.
__device__ __forceinline__ uint32_t block_merge(const uint32_t* A, uint32_t na, const uint32_t* B, uint32_t nb,
                                                uint32_t lane) {
  uint32_t ia = 0, ib = 0, c = 0;
  const auto at = [&](const uint32_t* p, uint32_t n, uint32_t k) { return k < n ? __ldg(p + k) : kUintPad; };
  uint32_t x = at(A, na, lane), x1 = at(A, na, 32 + lane), x2 = at(A, na, 64 + lane), x3 = at(A, na, 96 + lane);
  uint32_t y = at(B, nb, lane), y1 = at(B, nb, 32 + lane), y2 = at(B, nb, 64 + lane), y3 = at(B, nb, 96 + lane);
  while (ia < na && ib < nb) {
    uint32_t pos = 0;
#pragma unroll
    for (int h = 16; h; h >>= 1) pos += __shfl_sync(FULL, y, pos + h - 1) < x ? h : 0;
    c += __shfl_sync(FULL, y, pos) == x && x != kUintPad;
    const uint32_t xm = __shfl_sync(FULL, x, 31), ym = __shfl_sync(FULL, y, 31);
    if (xm <= ym) {
      ia += 32;
      x = x1;
      x1 = x2;
      x2 = x3;
      x3 = at(A, na, ia + 96 + lane);
    }
    if (ym <= xm) {
      ib += 32;
      y = y1;
      y1 = y2;
      y2 = y3;
      y3 = at(B, nb, ib + 96 + lane);
    }
  }
  return c;
}

// Lists the rows whose intersection CTAs take (sym_heavy).  A kernel of its own, so that
// those rows come first and k_symbiosity fills the GPU as they run out: with the list made
// by k_symbiosity the two ran one after the other (half-reciprocal R-MAT scale 21, hybrid:
// 328 against 299 us a call, 50,000 vertices 65 against 56).  Bound by reading the row
// descriptors; the column matrix is only looked at where the row's own size allows a heavy pair.
__global__ void k_symbiosity_find(uint32_t n, const RowDesc* __restrict__ dr, const uint4* __restrict__ ar,
                                  const RowDesc* __restrict__ dc, const uint4* __restrict__ ac, SymTest test,
                                  uint32_t* heavy, uint32_t* n_heavy) {
  for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < n; r += (uint64_t)gridDim.x * blockDim.x) {
    const RowView A = load_view(dr, ar, (uint32_t)r);
    // Uint rows: the larger above kSymMerge and within 32 x of the smaller, or the smaller above kSymLight.
    if (A.type != TY_BITSET && A.card <= kSymMerge / 32) continue;
    const RowView B = load_view(dc, ac, (uint32_t)r);
    if (sym_heavy(A, B) && sym_above(min(A.card, B.card), A, B, test)) heavy[atomicAdd(n_heavy, 1u)] = (uint32_t)r;
  }
}

// Rows are taken kSymChunk at a time from a shared cursor, one row per lane.  A
// row that could not pass with min(|out|, |in|) common entries is not read (the
// ratio grows with their number).  Two uint rows of at most kSymTiny entries are
// merged by the lane alone, longer ones and the other layouts go to the warp,
// rows too long for a warp are k_symbiosity_heavy's.  Half-reciprocal R-MAT scale 21,
// hybrid: 223 us here (latency of the lane merges and of the warp rows' first
// blocks, about equal) and 74 us for the listed rows, where binary searches in a
// staged row took 335 us; 541 -> 279 us a call with the two overlapped (six CTAs
// an SM; five: 299).
__global__ void __launch_bounds__(256, 6) k_symbiosity(uint32_t n, const RowDesc* __restrict__ dr,
                                                    const uint4* __restrict__ ar, const RowDesc* __restrict__ dc,
                                                    const uint4* __restrict__ ac, SymTest test,
                                                    unsigned long long* out, uint32_t* cursor) {
  __shared__ PshortHdr s_hdr[8];
  overlap_begin();
  const uint32_t lane = threadIdx.x & 31;
  unsigned long long acc = 0;
  const uint32_t chunks = (n + kSymChunk - 1) / kSymChunk;
  const uint32_t turn = (uint32_t)(((lane >> 1) * 2654435761ull) % chunks);  // this lane's 16th starts here
  for (;;) {
    uint32_t q = 0;
    if (lane == 0) q = atomicAdd(cursor, 1u);
    q = __shfl_sync(FULL, q, 0);
    if (q >= chunks) break;
    // Pairs of rows, one from each 16th of the matrix at a different place in it: the long
    // rows at the front of a degree-ordered graph spread over the chunks, and so do those
    // of raw R-MAT ids, which sit at the same places of every 16th (scale 22, directed: 493 us a call, 1,015
    // with the pairs 2 * chunks apart).
    uint32_t at = q + turn;
    if (at >= chunks) at -= chunks;
    const uint64_t r = 2 * at + (lane & 1) + (uint64_t)(lane >> 1) * 2 * chunks;
    bool warp_row = false;
    RowView A, B;
    A.p = B.p = nullptr;
    A.card = B.card = 0;
    A.type = B.type = TY_UINT;
    if (r < n) {
      A = load_view(dr, ar, (uint32_t)r);
      B = load_view(dc, ac, (uint32_t)r);
      const uint32_t most = max(A.card, B.card);
      const bool both_uint = A.type == TY_UINT && B.type == TY_UINT;
      if (!A.card || !B.card) {  // ratio 0, or 0/0 (NaN, never above)
        acc += sym_above(0, A, B, test);
      } else if (!sym_above(min(A.card, B.card), A, B, test)) {
        // not even with every entry of the shorter row
      } else if (both_uint && most <= kSymTiny) {
        const uint32_t both = merge_count(static_cast<const uint32_t*>(A.p), A.card,
                                          static_cast<const uint32_t*>(B.p), B.card);
        acc += sym_above(both, A, B, test);
      } else if (sym_heavy(A, B)) {
        // in the list
      } else {
        warp_row = true;
      }
    }
    const bool mergeable =
        A.type == TY_UINT && B.type == TY_UINT && max(A.card, B.card) <= 32u * min(A.card, B.card);
    for (uint32_t m = __ballot_sync(FULL, warp_row && mergeable); m; m &= m - 1) {
      const uint32_t src = __ffs(m) - 1;
      RowView A2, B2;
      A2.card = __shfl_sync(FULL, A.card, src);
      B2.card = __shfl_sync(FULL, B.card, src);
      const uint32_t* a = reinterpret_cast<const uint32_t*>(
          __shfl_sync(FULL, reinterpret_cast<unsigned long long>(A.p), src));
      const uint32_t* b = reinterpret_cast<const uint32_t*>(
          __shfl_sync(FULL, reinterpret_cast<unsigned long long>(B.p), src));
      const uint32_t both = warp_sum_u32(block_merge(a, A2.card, b, B2.card, lane));
      if (lane == 0) acc += sym_above(both, A2, B2, test);
    }
    for (uint32_t wm = __ballot_sync(FULL, warp_row && !mergeable); wm; wm &= wm - 1) {
      const uint32_t r2 = __shfl_sync(FULL, (uint32_t)r, __ffs(wm) - 1);
      const RowView A2 = load_view(dr, ar, r2);
      const RowView B2 = load_view(dc, ac, r2);
      const uint32_t both = warp_intersect_size(A2, B2, lane, &s_hdr[threadIdx.x >> 5]);  // header table: pshort rows
      if (lane == 0) acc += sym_above(both, A2, B2, test);
    }
  }
  acc = warp_sum_u64(acc);
  if (lane == 0 && acc) atomicAdd(out, acc);
  overlap_end();
}

// The listed rows, one CTA per row taken from a shared cursor.
__global__ void __launch_bounds__(256) k_symbiosity_heavy(const RowDesc* __restrict__ dr, const uint4* __restrict__ ar,
                                                          const RowDesc* __restrict__ dc, const uint4* __restrict__ ac,
                                                          SymTest test, unsigned long long* out,
                                                          const uint32_t* __restrict__ heavy,
                                                          const uint32_t* n_heavy, uint32_t* cursor) {
  __shared__ uint32_t s_sum[8];
  __shared__ uint32_t s_idx;
  overlap_begin();
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  const uint32_t nh = *n_heavy;
  unsigned long long acc = 0;
  for (;;) {
    __syncthreads();  // the previous row is finished with s_sum / s_idx
    if (tid == 0) s_idx = atomicAdd(cursor, 1u);
    __syncthreads();
    const uint32_t idx = s_idx;
    if (idx >= nh) break;
    const uint32_t r = heavy[idx];
    RowView A = load_view(dr, ar, r);
    RowView B = load_view(dc, ac, r);
    const RowView A0 = A, B0 = B;
    uint32_t c = 0;
    if (A.type == TY_BITSET && B.type == TY_BITSET) {
      const unsigned long long* a = static_cast<const unsigned long long*>(A.p);
      const unsigned long long* b = static_cast<const unsigned long long*>(B.p);
      const uint32_t lo = max(A.aux, B.aux), hi = min(A.aux + A.len, B.aux + B.len);
      for (uint32_t w = lo + tid; w < hi; w += blockDim.x) c += __popcll(a[w - A.aux] & b[w - B.aux]);
    } else {
      if (A.card > B.card) {
        const RowView T = A;
        A = B;
        B = T;
      }
      if (A.type == TY_UINT && B.type == TY_UINT && B.card <= 32u * A.card) {
        // Each warp merges a slice of the larger row with the part of the other in its range.
        const uint32_t* p = static_cast<const uint32_t*>(A.p);
        const uint32_t* q = static_cast<const uint32_t*>(B.p);
        const uint32_t nwarp = blockDim.x >> 5, per = (B.card + nwarp - 1) / nwarp;
        const uint32_t b0 = min(B.card, (tid >> 5) * per), b1 = min(B.card, b0 + per);
        const uint32_t a0 = b0 < b1 ? lower_bound_u32(p, 0, A.card, q[b0]) : 0u;
        const uint32_t a1 = b0 < b1 ? (b1 < B.card ? lower_bound_u32(p, a0, A.card, q[b1]) : A.card) : 0u;
        c = block_merge(p + a0, a1 - a0, q + b0, b1 - b0, lane);
      } else {
        cta_for_each(A, [&](uint32_t y) { c += row_contains(B, y); });
      }
    }
    c = warp_sum_u32(c);
    if (lane == 0) s_sum[tid >> 5] = c;
    __syncthreads();
    if (tid == 0) {
      uint32_t both = 0;
      for (uint32_t w = 0; w < (blockDim.x >> 5); w++) both += s_sum[w];
      both -= (uint32_t)pshort_pair_drop(A0, B0, ~0ull);
      if (sym_above(both, A0, B0, test)) acc++;
    }
  }
  if (tid == 0 && acc) atomicAdd(out, acc);
}

struct LevelCount {
  uint32_t light, heavy;
};

struct BfsArgs {
  const RowDesc* desc;
  const uint4* arena;
  uint32_t n;
  uint64_t words;
  unsigned long long* vis;   // visited up to the current frontier
  unsigned long long* seen;  // and what the current expansion has reached
  uint32_t* lists;     // two frontier lists of n entries: light rows from the front, heavy from the back
  LevelCount* counts;  // counts[j]: frontier sizes of the j-th level of the current chunk
  unsigned long long* reached;
};

// A word of `seen` through L1, possibly an older value of it: bits are only ever
// set, so a set bit is never wrong and a clear one is looked up again in L2.
__device__ __forceinline__ unsigned long long ld_seen(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.global.ca.u64 %0, [%1];" : "=l"(v) : "l"(p));
  return v;
}
// Sets x's bit in `seen` unless it is set.
__device__ __forceinline__ void visit(unsigned long long* seen, uint32_t x) {
  unsigned long long* at = seen + (x >> 6);
  const unsigned long long bit = 1ull << (x & 63);
  if (!(ld_seen(at) & bit) && !(__ldcg(at) & bit)) atomicOr(at, bit);
}

// Sets the bits of slice `part` (of `nparts`) of row V in `seen`; a group of W
// lanes (lane: the index in the group) shares the slice.
template <uint32_t W>
__device__ __forceinline__ void expand_slice(unsigned long long* seen, uint32_t n, const RowView& V, uint32_t part,
                                             uint32_t nparts, uint32_t lane) {
  if (V.type == TY_UINT) {
    const uint4* e4 = static_cast<const uint4*>(V.p);
    const uint32_t n4 = (V.card + 3) >> 2;
    for (uint32_t k = part * W + lane; k < n4; k += nparts * W) {
      const uint4 v = __ldg(e4 + k);
      const uint32_t x[4] = {v.x, v.y, v.z, v.w};
      unsigned long long w[4];
#pragma unroll
      for (int h = 0; h < 4; h++) w[h] = x[h] < n ? ld_seen(seen + (x[h] >> 6)) : ~0ull;  // padding: kUintPad
#pragma unroll
      for (int h = 0; h < 4; h++) {
        const unsigned long long bit = 1ull << (x[h] & 63);
        unsigned long long* at = seen + (x[h] >> 6);
        if (!(w[h] & bit) && !(__ldcg(at) & bit)) atomicOr(at, bit);
      }
    }
  } else if (V.type == TY_BITSET) {
    const unsigned long long* w = static_cast<const unsigned long long*>(V.p);
    for (uint32_t k = part * W + lane; k < V.len; k += nparts * W) {
      unsigned long long* at = seen + V.aux + k;
      const unsigned long long x = w[k];
      if ((x & ~ld_seen(at)) && (x & ~__ldcg(at))) atomicOr(at, x);
    }
  } else {
    const uint16_t* s = static_cast<const uint16_t*>(V.p);
    uint32_t i = 0, p = 0;
    while (i < V.len) {
      const uint32_t hb = (uint32_t)s[i] << 16, cnt = (uint32_t)s[i + 1] + 1;
      if (p % nparts == part)
        for (uint32_t k = lane; k < cnt; k += W) visit(seen, hb | s[i + 2 + k]);
      i += cnt + 2;
      p++;
    }
  }
}

__global__ void k_bfs_init(BfsArgs a, uint32_t start) {
  a.vis[start >> 6] = a.seen[start >> 6] = 1ull << (start & 63);
  if (a.desc[start].card > kBfsHeavy) {
    a.lists[a.n - 1] = start;
    a.counts[0] = LevelCount{0, 1};
  } else {
    a.lists[0] = start;
    a.counts[0] = LevelCount{1, 0};
  }
  *a.reached = 1;
}

// Level j of the chunk: frontier F (sizes counts[j]) -> seen.  Most entries lead to
// the same few hubs, whose words every SM asked the same L2 slice for (423 of
// 520 us at R-MAT scale 21 were one level's): the words now come through L1
// first, and no row is longer than its group of lanes, CTA or grid can share:
// 520 -> 260 us for all levels.
__global__ void __launch_bounds__(kBfsThreads) k_bfs_expand(BfsArgs a, uint32_t j, const uint32_t* __restrict__ F) {
  const LevelCount c = a.counts[j];
  if (c.light + c.heavy == 0) return;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t nw = gridDim.x * (blockDim.x / 32);
  const uint32_t gw = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  if (c.heavy) {
    // Warps form min(heavy, nw) groups; group g takes heavy rows g, g + groups, ...
    // and its gsz warps split each of them.
    const uint32_t groups = min(c.heavy, nw), gsz = nw / groups, g = gw / gsz;
    if (g < groups)
      for (uint32_t h = g; h < c.heavy; h += groups)
        expand_slice<32>(a.seen, a.n, load_view(a.desc, a.arena, F[a.n - 1 - h]), gw % gsz, gsz, lane);
  }
  // Light rows: 8 lanes each up to kBfsGroup entries; longer ones wait in a list
  // that the whole CTA shares at the end.  The ids and descriptors of a group's
  // next rows are fetched ahead.
  __shared__ uint32_t s_row[kBfsListed], s_n;
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  const uint32_t step = 4 * nw;
  const auto id = [&](uint32_t f) { return f < c.light ? F[f] : 0u; };
  const uint32_t f0 = 4 * gw + (lane >> 3);
  uint32_t r1 = id(f0), r2 = id(f0 + step);
  RowView next = load_view(a.desc, a.arena, r1);
  for (uint32_t f = f0; f < c.light; f += step) {
    const RowView V = next;
    const uint32_t row = r1;
    r1 = r2;
    next = load_view(a.desc, a.arena, r1);
    r2 = id(f + 2 * step);
    uint32_t at = kBfsListed;
    if (V.card > kBfsGroup) {
      if ((lane & 7) == 0) at = atomicAdd(&s_n, 1u);
      at = __shfl_sync(0xffu << (lane & 24), at, 0, 8);
      if (at < kBfsListed && (lane & 7) == 0) s_row[at] = row;
    }
    if (at >= kBfsListed) expand_slice<8>(a.seen, a.n, V, 0, 1, lane & 7);
  }
  __syncthreads();
  const uint32_t listed = min(s_n, kBfsListed);
  for (uint32_t k = 0; k < listed; k++)
    expand_slice<32>(a.seen, a.n, load_view(a.desc, a.arena, s_row[k]), threadIdx.x >> 5, kBfsThreads / 32, lane);
}

// Level j of the chunk: seen AND NOT visited -> frontier F (sizes counts[j + 1]).
__global__ void __launch_bounds__(kBfsThreads) k_bfs_collect(BfsArgs a, uint32_t j, uint32_t* __restrict__ F) {
  const LevelCount c = a.counts[j];
  if (c.light + c.heavy == 0) return;
  LevelCount* out = a.counts + j + 1;
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t nw = (uint64_t)gridDim.x * (blockDim.x / 32);
  unsigned long long found = 0;
  // One byte of the bitsets per lane, so that a lane has at most 8 vertices to
  // look up; whole warps step together (the appends below use warp collectives).
  const unsigned char* seen8 = reinterpret_cast<const unsigned char*>(a.seen);
  unsigned char* vis8 = reinterpret_cast<unsigned char*>(a.vis);
  const uint64_t bytes = a.words * 8;
  for (uint64_t w0 = ((uint64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5)) * 32; w0 < bytes; w0 += nw * 32) {
    const uint64_t w = w0 + lane;
    uint32_t x = 0, heavy = 0;
    if (w < bytes) {
      const uint32_t now = seen8[w];
      x = now & ~(uint32_t)vis8[w];
      if (x) vis8[w] = (unsigned char)now;
    }
    if (!__any_sync(FULL, x)) continue;
    uint32_t card[8];
#pragma unroll
    for (int h = 0; h < 8; h++) card[h] = (x >> h) & 1u ? a.desc[8 * w + h].card : 0u;
#pragma unroll
    for (int h = 0; h < 8; h++) heavy |= (card[h] > kBfsHeavy ? 1u : 0u) << h;
    found += __popc(x);
    const uint32_t nh = __popc(heavy), nl = __popc(x) - nh;
    const uint32_t il = warp_exclusive_scan(nl, lane), ih = warp_exclusive_scan(nh, lane);
    uint32_t base_l = 0, base_h = 0;
    if (lane == 31) {
      if (il + nl) base_l = atomicAdd(&out->light, il + nl);
      if (ih + nh) base_h = atomicAdd(&out->heavy, ih + nh);
    }
    uint32_t pl = __shfl_sync(FULL, base_l, 31) + il, ph = __shfl_sync(FULL, base_h, 31) + ih;
    for (uint32_t y = x; y; y &= y - 1) {
      const uint32_t v = (uint32_t)(8 * w) + (__ffs(y) - 1);
      if (heavy & y & (0u - y)) F[a.n - 1 - ph++] = v;
      else F[pl++] = v;
    }
  }
  found = warp_sum_u64(found);
  if (lane == 0 && found) atomicAdd(a.reached, found);
}

}  // namespace
}  // namespace eh

using eh::Matrix;

static eh_status cuda_err(cudaError_t e, const char* what) {
  return eh::set_error(EH_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

extern "C" eh_status eh_symbiosity_async(eh_matrix_t rh, eh_matrix_t ch, double threshold, uint64_t* d_count,
                                         void* stream) {
  using namespace eh;
  if (!rh || !ch) return set_error(EH_ERR_INVALID_ARGUMENT, "matrix is NULL");
  EH_CHECK_ARG(d_count, "d_count is NULL");
  Matrix* r = reinterpret_cast<Matrix*>(rh);
  Matrix* c = reinterpret_cast<Matrix*>(ch);
  if (r->n != c->n)
    return set_error(EH_ERR_INVALID_ARGUMENT, "row and column matrices differ in size (%llu vs %llu)",
                     (unsigned long long)r->n, (unsigned long long)c->n);
  if (r->device != c->device) return set_error(EH_ERR_INVALID_ARGUMENT, "row and column matrices are on different GPUs");
  cudaSetDevice(r->device);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemsetAsync(d_count, 0, sizeof(uint64_t), st);
  if (e != cudaSuccess) return cuda_err(e, "memset");
  if (r->n == 0) return EH_OK;
  // Heavy-row list: n entries, then its length, the CTAs' cursor and the warps' cursor.
  uint32_t* scratch = nullptr;
  e = pool_alloc((void**)&scratch, (r->n + 3) * sizeof(uint32_t), st);
  if (e != cudaSuccess) return set_error(EH_ERR_OUT_OF_MEMORY, "symbiosity scratch: %s", cudaGetErrorString(e));
  uint32_t* counts = scratch + r->n;
  e = cudaMemsetAsync(counts, 0, 3 * sizeof(uint32_t), st);
  int sms = 0, per = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, r->device);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_symbiosity_heavy, 256, 0);
  if (e == cudaSuccess) {
    const uint64_t g = std::min<uint64_t>((r->n + 8 * kSymChunk - 1) / (8 * kSymChunk), (uint64_t)sms * 8);
    unsigned long long* out = reinterpret_cast<unsigned long long*>(d_count);
    const SymTest test = sym_test(threshold);
    const unsigned blocks = (unsigned)std::min<uint64_t>((r->n + 255) / 256, (uint64_t)sms * 8);
    k_symbiosity_find<<<blocks, 256, 0, st>>>((uint32_t)r->n, r->desc, r->arena, c->desc, c->arena, test, scratch,
                                              counts);
    k_symbiosity_heavy<<<(unsigned)(sms * std::max(per, 1)), 256, 0, st>>>(r->desc, r->arena, c->desc, c->arena,
                                                                           test, out, scratch, counts,
                                                                           counts + 1);
    e = launch_overlapped(k_symbiosity, (unsigned)std::max<uint64_t>(g, 1), 256, 0, st, true, 0, (uint32_t)r->n,
                          r->desc, r->arena, c->desc, c->arena, test, out, counts + 2);
    const cudaError_t el = cudaGetLastError();
    if (e == cudaSuccess) e = el;
  }
  const cudaError_t ef = cudaFreeAsync(scratch, st);
  if (e == cudaSuccess) e = ef;
  note_use(r, st);
  note_use(c, st);
  return e == cudaSuccess ? EH_OK : cuda_err(e, "symbiosity kernels");
}

extern "C" eh_status eh_symbiosity(eh_matrix_t rh, eh_matrix_t ch, double threshold, uint64_t* count,
                                   void* stream) {
  using namespace eh;
  EH_CHECK_ARG(count, "count is NULL");
  if (!rh) return set_error(EH_ERR_INVALID_ARGUMENT, "matrix is NULL");
  Matrix* r = reinterpret_cast<Matrix*>(rh);
  eh_status s = eh_symbiosity_async(rh, ch, threshold, reinterpret_cast<uint64_t*>(r->result), stream);
  if (s != EH_OK) return s;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemcpyAsync(count, r->result, sizeof(uint64_t), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  return e == cudaSuccess ? EH_OK : cuda_err(e, "symbiosity");
}

extern "C" eh_status eh_bfs_path_length(eh_matrix_t mh, uint32_t start, uint64_t max_depth, uint64_t* path_length,
                                        uint64_t* reached, void* stream) {
  using namespace eh;
  if (!mh) return set_error(EH_ERR_INVALID_ARGUMENT, "matrix is NULL");
  EH_CHECK_ARG(path_length, "path_length is NULL");
  Matrix* m = reinterpret_cast<Matrix*>(mh);
  EH_CHECK_ARG(start < m->n, "start row %u >= matrix size %llu", start, (unsigned long long)m->n);
  cudaSetDevice(m->device);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const uint64_t n = m->n;
  // No BFS has more than n levels, so a deeper limit never binds.
  const uint64_t depth = std::min<uint64_t>(max_depth, n);
  const uint64_t words = (n + 64) / 64;
  const size_t bytes = 2 * words * 8 + 2 * n * 4 + (kBfsChunk + 1) * sizeof(LevelCount) + 8;
  char* base = nullptr;
  cudaError_t e = pool_alloc((void**)&base, bytes, st);
  if (e != cudaSuccess) return set_error(EH_ERR_OUT_OF_MEMORY, "BFS scratch (%zu bytes): %s", bytes, cudaGetErrorString(e));
  BfsArgs a;
  a.desc = m->desc;
  a.arena = m->arena;
  a.n = (uint32_t)n;
  a.words = words;
  a.vis = reinterpret_cast<unsigned long long*>(base);
  a.seen = a.vis + words;
  a.reached = a.seen + words;
  a.counts = reinterpret_cast<LevelCount*>(a.reached + 1);
  a.lists = reinterpret_cast<uint32_t*>(a.counts + kBfsChunk + 1);
  auto done = [&](eh_status s) {
    cudaFreeAsync(base, st);
    return s;
  };
  // vis, seen, reached, counts: everything before the lists starts at zero.
  if ((e = cudaMemsetAsync(base, 0, reinterpret_cast<char*>(a.lists) - base, st)) != cudaSuccess)
    return done(cuda_err(e, "memset"));
  k_bfs_init<<<1, 1, 0, st>>>(a, start);
  int sms = 0, per = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, m->device);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_bfs_expand, kBfsThreads, 0);
  const unsigned grid = (unsigned)std::max(1, sms * std::max(per, 1));
  const unsigned cgrid = (unsigned)std::min<uint64_t>((words * 8 + kBfsThreads - 1) / kBfsThreads, grid);
  struct {  // as on the device
    unsigned long long reached;
    LevelCount counts[kBfsChunk + 1];
  } h;
  const LevelCount* hc = h.counts;
  uint64_t level = 0, path = 0;
  for (;;) {
    // Expansions level .. level + k - 1; expansion L produces the frontier of level L + 1.
    const uint32_t k = (uint32_t)std::min<uint64_t>(kBfsChunk, depth + 1 - level);
    for (uint32_t j = 0; j < k; j++) {
      uint32_t* cur = a.lists + ((level + j) & 1) * n;
      uint32_t* nxt = a.lists + ((level + j + 1) & 1) * n;
      k_bfs_expand<<<grid, kBfsThreads, 0, st>>>(a, j, cur);
      k_bfs_collect<<<cgrid, kBfsThreads, 0, st>>>(a, j, nxt);
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return done(cuda_err(e, "BFS kernels"));
    if ((e = cudaMemcpyAsync(&h, a.reached, sizeof(h), cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
        (e = cudaStreamSynchronize(st)) != cudaSuccess)
      return done(cuda_err(e, "BFS level sizes"));
    bool stop = false;
    for (uint32_t j = 0; j < k && !stop; j++)
      if (hc[j + 1].light + hc[j + 1].heavy == 0) {
        path = level + j;
        stop = true;
      }
    if (!stop && level + k - 1 >= depth) {
      path = depth;
      stop = true;
    }
    if (stop) break;
    level += k;
    // The last frontier size of this chunk becomes the first of the next.
    if ((e = cudaMemcpyAsync(a.counts, a.counts + k, sizeof(LevelCount), cudaMemcpyDeviceToDevice, st)) != cudaSuccess ||
        (e = cudaMemsetAsync(a.counts + 1, 0, kBfsChunk * sizeof(LevelCount), st)) != cudaSuccess)
      return done(cuda_err(e, "BFS level sizes"));
  }
  *path_length = path;
  if (reached) *reached = h.reached;
  return done(EH_OK);
}

// ---- diagnostics: the bounded mbarrier wait used by the bulk-copy staging ----
namespace eh {
namespace {
// Waits on an mbarrier that nothing arrives on; the wait must give up after
// `tries` polls and the kernel report it instead of hanging.
__global__ void k_selftest_bounded_wait(uint32_t tries, uint32_t* status) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) mbar_init(&bar);
  __syncthreads();
  const bool done = mbar_wait(&bar, 0, tries);
  if (threadIdx.x == 0) *status = done ? 1u : 2u;
}
}  // namespace
}  // namespace eh

extern "C" eh_status eh_selftest_bounded_wait(uint32_t tries, uint32_t* timed_out) {
  using namespace eh;
  EH_CHECK_ARG(timed_out, "timed_out is NULL");
  EH_CHECK_ARG(tries > 0 && tries <= (1u << 16), "tries must be in [1, 65536]");
  uint32_t* d = nullptr;
  cudaError_t e = cudaMalloc((void**)&d, sizeof(uint32_t));
  if (e != cudaSuccess) return cuda_err(e, "selftest allocation");
  uint32_t h = 0;
  e = cudaMemset(d, 0, sizeof(uint32_t));
  if (e == cudaSuccess) {
    k_selftest_bounded_wait<<<1, 32>>>(tries, d);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(&h, d, sizeof(uint32_t), cudaMemcpyDeviceToHost);
  cudaFree(d);
  if (e != cudaSuccess) return cuda_err(e, "selftest");
  *timed_out = h == 2u;
  return h ? EH_OK : set_error(EH_ERR_DEVICE_CHECK, "self-test kernel did not report");
}
