// k-clique counting: the reference's n_clique<T,R>::run / apply_function
// (apps/n_clique.cpp:30-101).
//
// The reference walks, for every pivot i and j in A_i = row(i) (rows pruned to
// nbr < node), the materialized intersection C = A_i ∩ row(j), then for each
// k in C the intersection C ∩ row(k), and so on to depth n, returning |C| at
// the last level.  Every set on that path is a subset of A_i, so here each is a
// bitmask over the positions of A_i: M[e] = {t < e : A_i[t] in row(A_i[e])} is
// A_i ∩ row(A_i[e]) (row(j) only holds ids below j), and the reference's
// C ∩ row(k) for k = A_i[t] is M[e] & M[t].  The masks are built with the same
// layout-aware choice as the triangle kernel (probe each A_i[t] into row(j), or
// stream row(j) and look each element up in A_i); the counting is popcounts of
// ANDs:
//   k = 3: sum_e popc(M[e])
//   k = 4: sum_e sum_{t in M[e]} popc(M[e] & M[t])
//   k > 4: depth-first over the same masks.
// Tiers by |A_i| (rows sorted by descending size): one warp per pivot with
// two-word masks (|A_i| <= 64); one CTA per pivot with masks in shared memory
// (up to clique_smem_cap(k), about 1,650-1,850 entries), launched in size bands
// so that each launch's shared memory (and so its CTAs per SM) fits its own
// largest pivot; one CTA per pivot with masks in a global scratch slot (larger
// pivots).  The masks are stored as a packed lower-triangular bit matrix.
#include <algorithm>
#include <atomic>
#include <map>
#include <mutex>
#include <cstdint>

#include "eh_kernels.cuh"

namespace eh {

namespace {

constexpr int NW = kCtaThreads / 32;
constexpr uint32_t kCliqueWideMin = 1024;  // k <= 4 pivots above this run 1,024-thread CTAs

__device__ __forceinline__ uint32_t ilog2p1_c(uint32_t x) { return 32u - __clz(x | 1u); }

// Packed lower-triangular masks: row e holds bits < e in mask_len(e) words
// (ceil(e/32), made odd so that lanes reading rows e, e+1, ... at the same word
// index fall in different shared-memory banks); mask_off(e) = sum of the
// lengths of rows 0 .. e-1.  A c-entry pivot needs mask_off(c) words, about
// half of a c x c bit matrix.
__host__ __device__ __forceinline__ uint32_t mask_len(uint32_t e) { return ((e + 31) >> 5) | 1u; }
// 32-bit arithmetic: exact below kCliqueMaxPivot = 2^18 entries, the largest
// pivot a clique count accepts (mask_off(2^18 - 1) = 1,073,987,583 < 2^32).
__host__ __device__ __forceinline__ uint32_t mask_off(uint32_t e) {
  if (e == 0) return 0;
  const uint32_t A = (e - 1) >> 5, r = (e - 1) & 31;
  // row 0: 1 word; rows 32a+1 .. 32a+32: (a+1)|1 words each.
  return 1 + 32 * (A * (A + 1) / 2 + A / 2) + r * ((A + 1) | 1);
}

// Tuple output: the k ids of one clique (pivot row, then pivot entries in
// descending order) at the position the cursor a.out[0] hands out, if it is
// below the capacity.
__device__ __forceinline__ void put_tuple(const CliqueArgs& a, unsigned long long pos, uint32_t row, uint32_t x1,
                                          uint32_t x2, uint32_t x3) {
  if (pos >= a.capacity) return;
  uint32_t* o = a.tuples + pos * a.k;
  o[0] = row;
  o[1] = x1;
  o[2] = x2;
  if (a.k == 4) o[3] = x3;
}

// ---- warp tier: |A_i| <= kCliqueWarpMax (64), one warp per pivot, two-word masks ----
// Phase 1 sets bit t of M[e] for every pair with A_i[t] in row(A_i[e]); it has two forms,
// find_masks by work area.  HashArea, for a matrix with a core:
//  * j = A_i[e] < core_k: one lane per pair, two pairs in flight, a word of
//    core row j each;
//  * j >= core_k, a uint row: the row is streamed, 8 lanes per row and 16 bytes
//    per lane, each element tested in a 4,096-bit hash of the pivot; a set bit
//    is looked up in the list, which gives t;
//  * other rows, and rows longer than kCliqueProbe e: the e elements below j
//    are probed, 8 lanes per row.
// RowsArea, for a batch of graphs, which has no core and all its pivots here.  The
// rows are gathered by kind first, so that a warp's lanes stay together:
//  * bitset rows: a lane per t, a row per step, four in flight: the row's word under
//    x_t, a ballot, and a lane in 32 keeps it;
//  * uint rows are streamed as one sequence of 16-byte quads, two per lane and step
//    (rows of 17 entries on average, but of any length side by side), and each element
//    x looked up in a hash table of the pivot: kSlots 16-bit entries, ten bits of the
//    element stored there over its position, so that one shared-memory word answers
//    nearly every miss and gives t for a hit (the list confirms it).  Entries whose
//    slot another one took (18 entries: 0.15 of them) are compared with every x;
//  * other rows, and uint rows longer than kCliqueProbe e: the e elements below j
//    are probed, 4 lanes per row.
// Both are bound by instruction issue (80% of the slots with RowsArea).  A batch of
// 256 graphs (37 M entries, rows of 18 on average): 2.24 ms with HashArea, 15.7 of 32
// lanes active, as nearly every step met a bitset row beside a uint one and a hit to
// look up; 1.70 ms with RowsArea, 26.7 lanes (2.50 and 1.80 ms alone under ncu).  Where a core answers most pairs HashArea
// is the better one: 4-cliques of an R-MAT graph of 1 M vertices 0.340 against 0.347 ms
// in this kernel, of 21,288 vertices 34 against 51 us in all, as the table's shared
// memory (158 KB per SM against 51) keeps it from starting beside the larger pivots'
// kernel.
// Phase 2 counts (or lists) from the masks.  With `tri` set the same masks also
// give the pivot's triangles (sum of popc M[e]).
constexpr uint32_t kCliqueHash = 4096;
constexpr uint32_t kCliqueProbe = 24;
constexpr uint32_t kSlots = 1024;
constexpr uint32_t kFreeSlot = 0x803fu;  // no t: bit 63 is past every row's masks
__device__ __forceinline__ uint32_t slot_of(uint32_t x) { return (x * 0x9e3779b1u) >> 22; }
__device__ __forceinline__ uint32_t slot_tag(uint32_t x) { return (x >> 4) & 0xffc0u; }

// A warp's work area.
struct HashArea {
  // Draws from the queue a chunk ahead?  Not where that would set large pivots aside:
  // planted cliques 2.33 against 2.25 ms, 4-cliques of 21,288 vertices 37 against 34 us.
  static constexpr bool kAhead = false;
  uint32_t bm[kCliqueHash / 32];
  __device__ __forceinline__ void clear(uint32_t lane) {
    for (uint32_t k = lane; k < kCliqueHash / 32; k += 32) bm[k] = 0u;
  }
};
struct RowsArea {
  static constexpr bool kAhead = true;
  uint4 src[kCliqueWarpMax + 3];
  uint16_t tab[kSlots];
  uint8_t bit_e[kCliqueWarpMax];
  __device__ __forceinline__ void clear(uint32_t lane) {
    for (uint32_t k = lane; k < kSlots; k += 32) tab[k] = kFreeSlot;
  }
};

// The masks of the pivot whose c entries are in list; the work area is clear again on return.
__device__ __forceinline__ void find_masks(const CliqueArgs& a, HashArea& w, const uint32_t* list,
                                           unsigned long long* mask, uint32_t c, uint32_t lane) {
  uint32_t* bm = w.bm;
  uint32_t* mask32 = reinterpret_cast<uint32_t*>(mask);
  uint32_t ea = 0;  // entries below core_k
#pragma unroll
  for (uint32_t h = 0; h < kCliqueWarpMax; h += 32) {
    const uint32_t e = h + lane, x = e < c ? list[e] : 0xffffffffu;
    if (e < c) {
      mask[e] = 0ull;
      atomicOr(&bm[(x & (kCliqueHash - 1)) >> 5], 1u << (x & 31));
    }
    ea += __popc(__ballot_sync(FULL, x < a.core_k));
  }
  __syncwarp();
  // j < core_k
  const uint32_t pairs = ea * (ea - 1) / 2;
  uint32_t e = 1, t = lane;
  while (t >= e) { t -= e; e++; }
  for (uint32_t q = lane; q < pairs; q += 64) {
    const uint32_t e0 = e, t0 = t, j0 = list[e], x0 = list[t];
    t += 32;
    while (t >= e && e < c) { t -= e; e++; }
    const bool two = q + 32 < pairs;
    const uint32_t e1 = e, t1 = t, j1 = two ? list[e] : 0u, x1 = two ? list[t] : 0u;
    t += 32;
    while (t >= e && e < c) { t -= e; e++; }
    const unsigned long long v0 = __ldg(a.core + core_row_offset(j0) + (x0 >> 6));
    const unsigned long long v1 = two ? __ldg(a.core + core_row_offset(j1) + (x1 >> 6)) : 0ull;
    if ((v0 >> (x0 & 63)) & 1ull) atomicOr(&mask32[2 * e0 + (t0 >> 5)], 1u << (t0 & 31));
    if ((v1 >> (x1 & 63)) & 1ull) atomicOr(&mask32[2 * e1 + (t1 >> 5)], 1u << (t1 & 31));
  }
  // j >= core_k
  const uint32_t sl = lane & 7, first = max(1u, ea) + (lane >> 3);
  const auto source = [&](uint32_t r) { return __ldg(reinterpret_cast<const uint4*>(a.desc) + list[r]); };
  uint4 next = make_uint4(0u, 0u, 0u, 0u);
  if (first < c) next = source(first);
  for (uint32_t r = first; r < c; r += 4) {
    const uint4 d = next;
    if (r + 4 < c) next = source(r + 4);
    if ((d.w >> 30) == TY_UINT && d.y <= kCliqueProbe * r) {
      const uint4* p4 = a.arena + d.x;
      const uint32_t n4 = (d.y + 3) >> 2;  // padded with kUintPad
      for (uint32_t q0 = sl; q0 < n4; q0 += 16) {
        const uint4 pad = make_uint4(kUintPad, kUintPad, kUintPad, kUintPad);
        const uint4 va = __ldg(p4 + q0), vb = q0 + 8 < n4 ? __ldg(p4 + q0 + 8) : pad;
        const uint32_t y[8] = {va.x, va.y, va.z, va.w, vb.x, vb.y, vb.z, vb.w};
        uint32_t hits = 0;
#pragma unroll
        for (int h = 0; h < 8; h++)
          hits |= ((bm[(y[h] & (kCliqueHash - 1)) >> 5] >> (y[h] & 31)) & 1u) << h;
        for (; hits; hits &= hits - 1) {
          const uint32_t h = __ffs(hits) - 1;
          uint32_t yy = y[0];
#pragma unroll
          for (int u = 1; u < 8; u++) yy = h == (uint32_t)u ? y[u] : yy;
          const uint32_t pos = lower_bound_u32(list, 0, r, yy);
          if (pos < r && list[pos] == yy) atomicOr(&mask32[2 * r + (pos >> 5)], 1u << (pos & 31));
        }
      }
    } else {
      RowView B;
      B.p = a.arena + d.x;
      B.card = d.y;
      B.aux = d.z;
      B.type = d.w >> 30;
      B.len = d.w & 0x3fffffffu;
      for (uint32_t u = sl; u < r; u += 8)
        if (row_contains(B, list[u])) atomicOr(&mask32[2 * r + (u >> 5)], 1u << (u & 31));
    }
  }
  __syncwarp();
  for (uint32_t u = lane; u < c; u += 32) bm[(list[u] & (kCliqueHash - 1)) >> 5] = 0u;
}

__device__ __forceinline__ void find_masks(const CliqueArgs& a, RowsArea& w, const uint32_t* list,
                                           unsigned long long* mask, uint32_t c, uint32_t lane) {
  uint4* src = w.src;
  uint16_t* tab = w.tab;
  uint8_t* bit_e = w.bit_e;
  uint32_t* mask32 = reinterpret_cast<uint32_t*>(mask);
  // The entries by kind: uint rows in src[0, ns) (payload, first quad in the sequence, e),
  // bitset rows in src[np, nr) (payload, first 32-bit word, words) and three empty ones, the others between (e).
  uint4 d[2];
  uint32_t kind[2] = {0u, 0u}, quads[2] = {0u, 0u}, lost[2] = {0u, 0u};  // entries whose slot another one took
#pragma unroll
  for (uint32_t h = 0; h < 2; h++) {
    const uint32_t e = 32 * h + lane;
    if (e < c) {
      const uint32_t x = list[e];
      mask[e] = 0ull;
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(a.desc) + x);
      const uint32_t type = v.w >> 30;
      if (type == TY_BITSET) {
        d[h] = make_uint4(v.x, 0u, 2 * v.z, 2 * (v.w & 0x3fffffffu));
        kind[h] = 3;
      } else {
        d[h] = make_uint4(v.x, v.y, e, 0u);
        kind[h] = type == TY_UINT && v.y <= kCliqueProbe * e ? 1 : 2;
        if (kind[h] == 1) quads[h] = (v.y + 3) >> 2;  // padded with kUintPad
      }
      if (e == 0 || (kind[h] == 1 && quads[h] == 0)) kind[h] = quads[h] = 0;
    }
    if (c <= 32) break;
  }
  // The hash table and the sequence of quads, if there are uint rows.
  uint32_t start[2] = {0xffffffffu, 0xffffffffu}, total = 0;
  if (__any_sync(FULL, quads[0] + quads[1])) {
#pragma unroll
    for (uint32_t h = 0; h < 2; h++) {
      const uint32_t e = 32 * h + lane;
      if (e < c) {
        const uint32_t x = list[e];
        tab[slot_of(x)] = (uint16_t)(slot_tag(x) | e);
      }
      const uint32_t s = total + warp_exclusive_scan(quads[h], lane);
      total = __shfl_sync(FULL, s + quads[h], 31);
      if (quads[h]) start[h] = d[h].y = s;
      if (c <= 32) break;
    }
    __syncwarp();
#pragma unroll
    for (uint32_t h = 0; h < 2; h++) {
      const uint32_t e = 32 * h + lane;
      lost[h] = __ballot_sync(FULL, e < c && (tab[slot_of(list[e])] & 63u) != e);
      if (c <= 32) break;
    }
  }
  uint32_t ns = 0, np = 0, np1 = 0, nr = 0;  // np1: the first bit row of an entry past 31
#pragma unroll
  for (uint32_t k = 1; k <= 3; k++) {
#pragma unroll
    for (uint32_t h = 0; h < 2; h++) {
      const uint32_t bits = __ballot_sync(FULL, kind[h] == k), at = nr + __popc(bits & ((1u << lane) - 1u));
      if (kind[h] == k) {
        src[at] = d[h];
        if (k == 3) bit_e[at] = (uint8_t)(32 * h + lane);
      }
      nr += __popc(bits);
      if (k == 3 && h == 0) np1 = nr;
      if (c <= 32) break;
    }
    if (k == 1) ns = nr;
    if (k == 2) np = nr;
  }
  if (lane < 3) src[nr + lane] = make_uint4(0u, 0u, 0u, 0u);
  __syncwarp();
  // bitset rows
#pragma unroll 1
  for (uint32_t h = 0; h < 2 && 32 * h < c; h++) {
    const uint32_t t = 32 * h + lane, x = t < c ? list[t] : 0u, xw = x >> 5, sh = x & 31;
#pragma unroll 1
    for (uint32_t i0 = h ? np1 : np; i0 < nr; i0 += 32) {
      uint32_t keep = 0;
      const uint32_t iend = min(nr - i0, 32u);
      for (uint32_t i = 0; i < iend; i += 4) {
        uint32_t v[4];
#pragma unroll
        for (uint32_t u = 0; u < 4; u++) {
          const uint4 b = src[i0 + i + u];
          const uint32_t* words = reinterpret_cast<const uint32_t*>(a.arena + b.x);
          v[u] = xw - b.z < b.w ? __ldg(words + (xw - b.z)) : 0u;
        }
#pragma unroll
        for (uint32_t u = 0; u < 4; u++) {
          const uint32_t m = __ballot_sync(FULL, (v[u] >> sh) & 1u);
          if (lane == i + u) keep = m;
        }
      }
      if (lane < iend) {
        const uint32_t e = bit_e[i0 + lane];  // bits t < e
        if (h) mask32[2 * e + 1] = keep & ((1u << (e - 32)) - 1u);
        else mask32[2 * e] = e < 32 ? keep & ((1u << e) - 1u) : keep;
      }
    }
  }
  // uint rows
  const uint32_t upto = (2u << lane) - 1u;
  uint32_t rows = 0xffffffffu;  // the last row that starts before the step
  for (uint32_t q0 = 0; q0 < total; q0 += 64) {
    uint32_t e[2], y[8], at[8], least = 64;
#pragma unroll
    for (int v = 0; v < 2; v++) {
      const uint32_t first = q0 + 32 * v, q = first + lane;
      const uint32_t begins = __reduce_or_sync(FULL, __funnelshift_lc(0u, 1u, start[0] - first) |
                                                         __funnelshift_lc(0u, 1u, start[1] - first));
      const uint4 b = src[rows + __popc(begins & upto)];
      rows += __popc(begins);
      uint4 w = make_uint4(kUintPad, kUintPad, kUintPad, kUintPad);
      if (q < total) w = __ldg(a.arena + b.x + (q - b.y));
      e[v] = b.z;
      y[4 * v] = w.x;
      y[4 * v + 1] = w.y;
      y[4 * v + 2] = w.z;
      y[4 * v + 3] = w.w;
    }
#pragma unroll
    for (int h = 0; h < 8; h++) {
      at[h] = tab[slot_of(y[h])] ^ slot_tag(y[h]);
      least = min(least, at[h]);
    }
    uint32_t m[4] = {0u, 0u, 0u, 0u};  // the quads' masks, low and high words
    if (least < 64) {
#pragma unroll
      for (int h = 0; h < 8; h++)
        if (at[h] < 64 && list[at[h]] == y[h]) {
          m[h >> 2] |= __funnelshift_lc(0u, 1u, at[h]);  // 0 from 32 on
          m[2 + (h >> 2)] |= __funnelshift_lc(0u, 1u, at[h] - 32u);
        }
    }
#pragma unroll
    for (int g = 0; g < 2; g++) {
      for (uint32_t o = lost[g]; o; o &= o - 1) {
        const uint32_t pos = __ffs((int)o) - 1, x = list[32 * g + pos];
#pragma unroll
        for (int h = 0; h < 8; h++) m[2 * g + (h >> 2)] |= y[h] == x ? 1u << pos : 0u;
      }
    }
#pragma unroll
    for (int v = 0; v < 2; v++) {  // bits t < e
      if (m[v]) atomicOr(&mask32[2 * e[v]], m[v] & (__funnelshift_lc(0u, 1u, e[v]) - 1u));
      if (m[2 + v] && e[v] > 32) atomicOr(&mask32[2 * e[v] + 1], m[2 + v] & ((1u << (e[v] - 32)) - 1u));
    }
  }
  // the other rows, eight at a time
  const uint32_t sl = lane & 3;
  for (uint32_t i0 = ns; i0 < np; i0 += 8) {
    const uint32_t i = i0 + (lane >> 2);
    unsigned long long m = 0;
    uint32_t r = 0;
    if (i < np) {
      r = src[i].z;
      const RowView B = load_view(a.desc, a.arena, list[r]);
      for (uint32_t u = sl; u < r; u += 4)
        if (row_contains(B, list[u])) m |= 1ull << u;
    }
    m |= __shfl_xor_sync(FULL, m, 1);
    m |= __shfl_xor_sync(FULL, m, 2);
    if (sl == 0 && r) mask[r] = m;
  }
  __syncwarp();
  if (total)
    for (uint32_t u = lane; u < c; u += 32) tab[slot_of(list[u])] = kFreeSlot;
}

// LIST: write the k = 3 or 4 cliques as tuples instead of counting them.
template <bool LIST, class Area>
__global__ void __launch_bounds__(kCtaThreads, 5) k_clique_warp(CliqueArgs a, uint32_t pos_begin, uint32_t pos_end,
                                                                uint32_t grab, uint32_t* counter) {
  __shared__ unsigned long long s_mask[NW][kCliqueWarpMax];
  __shared__ uint32_t s_list[NW][kCliqueWarpMax];
  __shared__ Area s_work[NW];
  overlap_begin();
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t* list = s_list[warp];
  Area& work = s_work[warp];
  unsigned long long* mask = s_mask[warp];
  uint32_t* mask32 = reinterpret_cast<uint32_t*>(mask);
  const int top = (int)a.k - 3;  // DFS depth at which a popcount finishes the count
  work.clear(lane);
  unsigned long long acc = 0, tacc = 0;
  const bool ahead = Area::kAhead && grab > 1;
  uint32_t drawn = 0;
  if (lane == 0 && ahead) drawn = atomicAdd(counter, grab);
  for (;;) {
    if (lane == 0 && !ahead) drawn = atomicAdd(counter, grab);
    const uint32_t base = __shfl_sync(FULL, drawn, 0) + pos_begin;
    if (base >= pos_end) break;
    if (lane == 0 && ahead) drawn = atomicAdd(counter, grab);
    const uint32_t end = min(pos_end, base + grab);
    const uint32_t my_row = base + lane < end ? a.order[base + lane] : a.order[base];
    const uint4 my_desc = __ldg(reinterpret_cast<const uint4*>(a.desc) + my_row);
    for (uint32_t p = base; p < end; p++) {
      const uint32_t row = __shfl_sync(FULL, my_row, p - base);
      RowView A;
      A.p = a.arena + __shfl_sync(FULL, my_desc.x, p - base);
      A.card = __shfl_sync(FULL, my_desc.y, p - base);
      A.aux = __shfl_sync(FULL, my_desc.z, p - base);
      A.len = __shfl_sync(FULL, my_desc.w, p - base);
      A.type = A.len >> 30;
      A.len &= 0x3fffffffu;
      const uint32_t c = A.card;
      warp_decode(A, list, lane);
      find_masks(a, work, list, mask, c, lane);
      // phase 2: a lane takes the cliques whose two largest members are i and A_i[e]
      if (LIST) {
        for (uint32_t h = 0; h < c; h += 32) {
          // (i, A_i[e], A_i[t]) for t in M[e], or (i, A_i[e], A_i[t], A_i[u]) for
          // u in M[e] & M[t]; one cursor atomic per warp and 32 entries.
          const unsigned long long m0 = h + lane < c ? mask[h + lane] : 0ull;
          uint32_t n = 0;
          if (top == 0) {
            n = __popcll(m0);
          } else {
            for (unsigned long long m = m0; m; m &= m - 1) n += __popcll(m0 & mask[__ffsll((long long)m) - 1]);
          }
          const uint32_t ex = warp_exclusive_scan(n, lane);
          unsigned long long at = 0;
          if (lane == 31 && ex + n) at = atomicAdd(a.out, (unsigned long long)(ex + n));
          at = __shfl_sync(FULL, at, 31) + ex;
          for (unsigned long long m = at < a.capacity ? m0 : 0ull; m; m &= m - 1) {  // past the capacity: counted only
            const uint32_t tt = __ffsll((long long)m) - 1;
            if (top == 0) {
              put_tuple(a, at++, row, list[h + lane], list[tt], 0u);
            } else {
              for (unsigned long long r = m0 & mask[tt]; r; r &= r - 1)
                put_tuple(a, at++, row, list[h + lane], list[tt], list[__ffsll((long long)r) - 1]);
            }
          }
        }
        __syncwarp();
        continue;
      }
      unsigned long long pc = 0;
      uint32_t tc = 0;
      if (c <= 32 && top <= 1) {
        const uint32_t m0 = lane < c ? mask32[2 * lane] : 0u;
        tc = __popc(m0);
        uint32_t n = 0;
        for (uint32_t m = top == 1 ? m0 : 0u; m; m &= m - 1) n += __popc(m0 & mask32[2 * (__ffs(m) - 1)]);
        pc = n;
      }
      for (uint32_t ee = c <= 32 && top <= 1 ? c : lane; ee < c; ee += 32) {
        const unsigned long long m0 = mask[ee];
        tc += __popcll(m0);
        if (top == 1) {
          uint32_t n = 0;
          for (unsigned long long m = m0; m; m &= m - 1) n += __popcll(m0 & mask[__ffsll((long long)m) - 1]);
          pc += n;
        } else if (top > 1) {
          unsigned long long S[kCliqueMaxK], R[kCliqueMaxK];
          S[0] = R[0] = m0;
          int d = 0;
          while (d >= 0) {
            if (d == top) {
              pc += __popcll(S[d]);
              d--;
              continue;
            }
            if (!R[d]) {
              d--;
              continue;
            }
            const uint32_t tt = __ffsll((long long)R[d]) - 1;
            R[d] &= R[d] - 1;
            const unsigned long long nx = S[d] & mask[tt];
            if (__popcll(nx) >= top - d) {  // enough candidates left
              S[d + 1] = R[d + 1] = nx;
              d++;
            }
          }
        }
      }
      if (top == 0) pc = tc;
      if (a.graph_rows) {  // batch: this pivot's cliques (and triangles) go to its graph
        tc = warp_sum_u32(tc);
        if (tc) {  // no clique without a triangle
          pc = top <= 1 ? warp_sum_u32((uint32_t)pc) : warp_sum_u64(pc);
          const uint32_t g = warp_graph_of(a.graph_rows, a.num_graphs, row, lane);
          if (lane == 0 && pc) atomicAdd(&a.out[g], pc);
          if (lane == 0 && a.tri) atomicAdd(&a.tri[g], (unsigned long long)tc);
        }
      } else {
        acc += pc;
        tacc += tc;
      }
      __syncwarp();
    }
  }
  if (!LIST && !a.graph_rows) {
    acc = warp_sum_u64(acc);
    if (lane == 0 && acc) atomicAdd(a.out, acc);
    tacc = a.tri ? warp_sum_u64(tacc) : 0ull;
    if (lane == 0 && tacc) atomicAdd(a.tri, tacc);
  }
  overlap_end();
}

// ---- mid tier, k = 4: kCliqueWarpMax < |A_i| <= kCliqueMidMax, one CTA per pivot ----
// The masks in shared memory as rows of 16-byte quads: row e holds bits < e in
// ceil(e / 128) quads, from quad quad_off(e) on.
//  Phase 1, j = A_i[e] < core_k: a lane keeps one t of 32 (its element's word and
//    bit in a core row) and walks the e's, eight words in flight; a ballot per e
//    gives a mask word, which lane e - e0 keeps and stores once per 16 e's.  That
//    is about half the instructions of a warp per e, which recomputed every
//    element's address for every e.  j >= core_k: 8 lanes stream row(j) and find
//    each element's position in a chained hash of the list (two or three words of
//    shared memory, where a binary search took eight), or probe a longer row or
//    another layout at the e elements.
//  Phase 2: the sum over e and t in M[e] of popc(M[e] & M[t]).  A lane keeps the
//    quad of M[t] for one t of 32, and the e's quads are broadcast: three LDS and
//    a masked AND per word into a carry-save counter, whatever the density, no
//    bank conflicts, and the popcount unit (16 lanes per cycle and SM) sees one
//    word in eight.
// Bound by instruction issue.  Tensor cores do not help: the one-bit mma.sync
// (m16n8k256, and.popc) takes 520 to 545 cycles a warp on this chip, fewer bits per cycle
// than the AND loop.  R-MAT, 1 M vertices, 4-cliques: phase 1 / phase 2 took 1.49 /
// 2.73 ms with a warp per e in both.
__host__ __device__ __forceinline__ uint32_t quad_off(uint32_t e) {
  if (e == 0) return 0;
  const uint32_t m = (e - 1) >> 7, r = (e - 1) & 127;
  return (64 * m + r) * (m + 1);
}

__host__ __device__ constexpr uint32_t mid_slots(uint32_t c) { return (c + 31) & ~31u; }
// Heads of the list's hash chains: two per entry at least.
__host__ __device__ inline uint32_t mid_heads(uint32_t cmax) {
  uint32_t h = 128;
  while (h < 2 * cmax) h *= 2;
  return h;
}
static uint32_t mid_bytes(uint32_t cmax) {
  return quad_off(cmax) * 16 + mid_slots(cmax) * (4 + 4 + 2 + 2) + mid_heads(cmax) * 4;
}

struct MaskSum {  // carry-save counter of 32-bit words
  uint32_t one, two, four, eights;
  __device__ __forceinline__ void clear() { one = two = four = eights = 0; }
  __device__ __forceinline__ void add8(const uint32_t (&x)[8]) {
    const uint32_t a = csa(one, x[0], x[1]), b = csa(one, x[2], x[3]), f = csa(two, a, b);
    const uint32_t c = csa(one, x[4], x[5]), d = csa(one, x[6], x[7]), g = csa(two, c, d);
    eights += __popc(csa(four, f, g));
  }
  __device__ __forceinline__ uint32_t total() const {
    return 8 * eights + 4 * __popc(four) + 2 * __popc(two) + __popc(one);
  }
};

// Phase 2 for one quad of 32 t's (mt: this lane's, W words of it in use), e = e0,
// e0 + NW, ... < c: quad q of M[e] against mt where bit `lane` of M[e]'s word r is set.
template <int W>
__device__ __forceinline__ void and_quads(const uint4* m4, const uint16_t* ro, uint4 mt, uint32_t q, uint32_t r,
                                          uint32_t e0, uint32_t c, uint32_t lane, MaskSum& sum) {
  constexpr int E = W == 1 ? 8 : W == 2 ? 4 : 2;  // e's per step: eight words or six
  const uint32_t m[4] = {mt.x, mt.y, mt.z, mt.w};
  for (uint32_t e = e0; e < c; e += E * NW) {
    uint32_t x[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int u = 0; u < E; u++) {
      const uint32_t eu = e + u * NW;
      const bool in = eu < c;
      const uint4* row = m4 + ro[in ? eu : e];
      const uint32_t bits = in ? reinterpret_cast<const uint32_t*>(row)[r] : 0u;
      const uint32_t sel = (uint32_t)((int32_t)(bits << (31 - lane)) >> 31);
      const uint4 v = row[q];
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int k = 0; k < W; k++) x[u * W + k] = w[k] & m[k] & sel;
    }
    sum.add8(x);
  }
}

__global__ void __launch_bounds__(kCtaThreads, 5) k_clique_mid(CliqueArgs a, uint32_t pos_begin, uint32_t pos_end,
                                                               uint32_t* counter, uint32_t cmax) {
  extern __shared__ __align__(16) uint4 m4[];
  __shared__ uint32_t s_unit, s_scan[NW];
  overlap_begin();
  uint32_t* m32 = reinterpret_cast<uint32_t*>(m4);
  uint32_t* list = reinterpret_cast<uint32_t*>(m4 + quad_off(cmax));
  uint32_t* off = list + mid_slots(cmax);  // word (32-bit) offset of core row A_i[e]
  constexpr uint32_t kNone = 0xffffu;
  const uint32_t hmask = mid_heads(cmax) - 1;
  uint32_t* head = off + mid_slots(cmax);  // first position of each chain (positions are below 2^16), or kNone
  uint16_t* ro = reinterpret_cast<uint16_t*>(head + hmask + 1);
  uint16_t* next = ro + mid_slots(cmax);
  const uint32_t* core32 = reinterpret_cast<const uint32_t*>(a.core);
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long acc = 0;
  MaskSum sum;
  sum.clear();
  for (;;) {
    if (threadIdx.x == 0) s_unit = atomicAdd(counter, 1u) + pos_begin;
    __syncthreads();  // also: every thread is done with the previous pivot's masks
    const uint32_t unit = s_unit;
    if (unit >= pos_end) break;
    const uint32_t row = a.order[unit];
    const RowView A = load_view(a.desc, a.arena, row);
    const uint32_t c = A.card;
    cta_decode_to<kCtaThreads>(A, s_scan, [&](uint32_t k, uint32_t x) {
      list[k] = x;
      off[k] = x < a.core_k ? 2 * core_offset32(x) : 0u;
    });
    const uint32_t quads = quad_off(c);
    for (uint32_t k = threadIdx.x; k < quads; k += kCtaThreads) m4[k] = make_uint4(0u, 0u, 0u, 0u);
    for (uint32_t k = threadIdx.x; k < c; k += kCtaThreads) ro[k] = (uint16_t)quad_off(k);
    __syncthreads();
    const uint32_t ea = lower_bound_u32(list, 0, c, a.core_k);
    if (ea < c) {  // rows to stream: hash the list
      for (uint32_t k = threadIdx.x; k <= hmask; k += kCtaThreads) head[k] = kNone;
      __syncthreads();
      for (uint32_t k = threadIdx.x; k < c; k += kCtaThreads)
        next[k] = (uint16_t)atomicExch(&head[list[k] & hmask], k);
      __syncthreads();
    }
    // phase 1, j < core_k: tasks (32 t's from 32 r, 16 e's from 16 b), b >= 2 r
    const uint32_t nb = (ea + 15) >> 4;
    for (uint32_t r = 0, id = warp;;) {
      while (2 * r < nb && id >= nb - 2 * r) {
        id -= nb - 2 * r;
        r++;
      }
      if (2 * r >= nb) break;
      const uint32_t e0 = 16 * (2 * r + id), t = 32 * r + lane;
      const uint32_t x = t < ea ? list[t] : 0u;
      const uint32_t* col = core32 + (x >> 5);
      const uint32_t bit = 1u << (x & 31);
      uint32_t word = 0;
      const bool whole = e0 >= 32 * (r + 1) && e0 + 16 <= ea;  // every t < e
#pragma unroll
      for (int h = 0; h < 16; h += 8) {
        uint32_t v[8];
        if (whole) {
#pragma unroll
          for (int u = 0; u < 8; u++) v[u] = __ldg(col + off[e0 + h + u]);
        } else {
#pragma unroll
          for (int u = 0; u < 8; u++) {
            const uint32_t e = e0 + h + u;
            v[u] = (t < e && e < ea) ? __ldg(col + off[e]) : 0u;
          }
        }
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const uint32_t bal = __ballot_sync(FULL, v[u] & bit);
          if (lane == (uint32_t)(h + u)) word = bal;
        }
      }
      const uint32_t e = e0 + lane;
      if (lane < 16 && e < ea && e > 32 * r) m32[4 * (uint32_t)ro[e] + r] = word;
      id += NW;
    }
    // phase 1, j >= core_k: 8 lanes per e
    const uint32_t sl = lane & 7;
    for (uint32_t e = max(1u, ea) + 4 * warp + (lane >> 3); e < c; e += 4 * NW) {
      uint32_t* Me = m32 + 4 * (uint32_t)ro[e];
      const RowView B = load_view(a.desc, a.arena, list[e]);
      if (B.type == TY_UINT && B.card <= kCliqueProbe * e) {
        const uint4* p4 = static_cast<const uint4*>(B.p);
        const uint32_t n4 = (B.card + 3) >> 2;  // padded with kUintPad
        for (uint32_t q0 = sl; q0 < n4; q0 += 16) {
          const uint4 pad = make_uint4(kUintPad, kUintPad, kUintPad, kUintPad);
          const uint4 va = __ldg(p4 + q0), vb = q0 + 8 < n4 ? __ldg(p4 + q0 + 8) : pad;
          const uint32_t y[8] = {va.x, va.y, va.z, va.w, vb.x, vb.y, vb.z, vb.w};
          uint32_t at[8];
#pragma unroll
          for (int h = 0; h < 8; h++) at[h] = head[y[h] & hmask];
#pragma unroll
          for (int h = 0; h < 8; h++) {
            uint32_t k = at[h];
            while (k != kNone && list[k] != y[h]) k = next[k];
            if (k < e) atomicOr(&Me[k >> 5], 1u << (k & 31));
          }
        }
      } else {
        for (uint32_t t = sl; t < e; t += 8)
          if (row_contains(B, list[t])) atomicOr(&Me[t >> 5], 1u << (t & 31));
      }
    }
    __syncthreads();
    // phase 2
    for (uint32_t r = 0; 32 * r < c; r++) {
      const uint32_t t = 32 * r + lane, e0 = 32 * r + 1 + warp, last = r >> 2;
      for (uint32_t q = 0; q <= last; q++) {
        const uint4 mt = (t < c && 128 * q < t) ? m4[ro[t] + q] : make_uint4(0u, 0u, 0u, 0u);
        const uint32_t words = q < last ? 4u : (r & 3) + 1;
        if (words == 1) and_quads<1>(m4, ro, mt, q, r, e0, c, lane, sum);
        else if (words == 2) and_quads<2>(m4, ro, mt, q, r, e0, c, lane, sum);
        else if (words == 3) and_quads<3>(m4, ro, mt, q, r, e0, c, lane, sum);
        else and_quads<4>(m4, ro, mt, q, r, e0, c, lane, sum);
      }
    }
    if (a.graph_rows) {  // batch: each warp's share of this pivot goes to its graph
      const uint32_t pc = warp_sum_u32(sum.total());  // below 2^28
      sum.clear();
      if (pc) {
        const uint32_t g = warp_graph_of(a.graph_rows, a.num_graphs, row, lane);
        if (lane == 0) atomicAdd(&a.out[g], (unsigned long long)pc);
      }
    } else {
      acc += 8ull * sum.eights;
      sum.eights = 0;
    }
  }
  acc = warp_sum_u64(acc + sum.total());
  if (lane == 0 && acc) atomicAdd(a.out, acc);
  overlap_end();
}

// ---- CTA tiers: one pivot per CTA; masks in shared memory or a global slot ----
// Per CTA working set (words): list[cmax] | masks[mask_off(cmax)] | stacks[NW][2 * (k-2) * W]
// (stacks only for k >= 5); W = mask_len(cmax) is the DFS stack row length.
// NT threads per CTA: 256, or 1,024 for the largest pivots at k <= 4, whose
// masks leave room for one CTA per SM (more warps to hide latency).
template <bool GLOBAL, int NT, bool LIST>
__global__ void __launch_bounds__(NT, NT == 1024 ? 1 : (GLOBAL ? 2 : 8)) k_clique_cta(CliqueArgs a, uint32_t pos_begin, uint32_t pos_end,
                                                            uint32_t* counter, uint32_t cmax, uint32_t W,
                                                            uint32_t* gscratch, uint64_t slot_words) {
  extern __shared__ __align__(16) uint32_t dyn[];
  __shared__ uint32_t s_unit;
  constexpr int NW = NT / 32;
  __shared__ uint32_t s_scan[NT];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t* base = GLOBAL ? gscratch + (uint64_t)blockIdx.x * slot_words : dyn;
  uint32_t* list = base;
  uint32_t* masks = base + cmax;
  const uint32_t stack_words = 2u * (a.k - 2) * W;
  uint32_t* stack = masks + mask_off(cmax) + (uint64_t)warp * stack_words;
  const int top = (int)a.k - 3;
  unsigned long long acc = 0;
  for (;;) {
    if (threadIdx.x == 0) s_unit = atomicAdd(counter, 1u) + pos_begin;
    __syncthreads();
    const uint32_t unit = s_unit;
    if (unit >= pos_end) break;
    const uint32_t row = a.order[unit];
    const RowView A = load_view(a.desc, a.arena, row);
    const uint32_t c = A.card;
    const unsigned long long acc_before = acc;
    cta_decode<NT>(A, list, s_scan);
    for (uint64_t x = threadIdx.x; x < mask_off(c); x += NT) masks[x] = 0;
    __syncthreads();
    // phase 1: warp per e builds M[e]
    for (uint32_t e = 1 + warp; e < c; e += NW) {
      const uint32_t j = list[e];
      uint32_t* Me = masks + mask_off(e);
      if (j < a.core_k) {  // core row j = row(j) ∩ [0, j): one word per probe, L2-resident
        const unsigned long long* row = a.core + core_row_offset(j);
        for (uint32_t b = 0; b < e; b += 32) {
          const uint32_t t = b + lane;
          const bool hit = t < e && ((__ldg(row + (list[t] >> 6)) >> (list[t] & 63)) & 1ull);
          const uint32_t word = __ballot_sync(FULL, hit);
          if (lane == 0) Me[b >> 5] = word;
        }
        continue;
      }
      const RowView B = load_view(a.desc, a.arena, j);
      if (B.card == 0) continue;
      bool stream = false;
      if (B.type == TY_UINT) stream = (uint64_t)B.card * ilog2p1_c(e) < (uint64_t)e * ilog2p1_c(B.card) * 4u;
      else if (B.type == TY_PSHORT) stream = (uint64_t)B.card * ilog2p1_c(e) < (uint64_t)e * (B.aux + ilog2p1_c(B.card)) * 4u;
      if (!stream) {
        for (uint32_t b = 0; b < e; b += 32) {
          const uint32_t t = b + lane;
          const bool hit = t < e && row_contains(B, list[t]);
          const uint32_t word = __ballot_sync(FULL, hit);
          if (lane == 0) Me[b >> 5] = word;
        }
      } else {
        warp_for_each(B, j, lane, [&](uint32_t y) {
          const uint32_t t = lower_bound_u32(list, 0, e, y);
          if (t < e && list[t] == y) atomicOr(&Me[t >> 5], 1u << (t & 31));
        });
      }
    }
    __syncthreads();
    // k = 3, pshort pivots of >= 65,536 entries: M[e] without what the reference's u16
    // counts drop.  (Not for larger k, whose later levels need the whole of M[t].)
    if (GLOBAL && top == 0 && A.type == TY_PSHORT && c >= 65536u) {
      for (uint32_t e = 1 + warp; e < c; e += NW) {
        const RowView B = load_view(a.desc, a.arena, list[e]);
        if (!pshort_pair_drop(A, B, list[e])) continue;
        uint32_t* Me = masks + mask_off(e);
        for (uint32_t w = lane; 32 * w < e; w += 32)
          for (uint32_t r = Me[w]; r; r &= r - 1) {
            const uint32_t h = list[32 * w + __ffs(r) - 1] >> 16;
            if (pshort_full_block(A, h) && pshort_full_block(B, h)) Me[w] &= ~(r & (0u - r));
          }
      }
      __syncthreads();
    }
    // phase 2: warp per e
    for (uint32_t e = 1 + warp; e < c; e += NW) {
      const uint32_t* Me = masks + mask_off(e);
      const uint32_t we = (e + 31) >> 5;  // words that can hold bits < e
      if (LIST) {
        // Lane t of each word of M[e] lists (i, A_i[e], A_i[t]) or, for k = 4,
        // (i, A_i[e], A_i[t], A_i[u]) for u in M[e] & M[t], one cursor atomic per word of M[e].
        // Tuples past the capacity are counted, not enumerated.
        const uint32_t je = list[e];
        for (uint32_t w = 0; w < we; w++) {
          const uint32_t bits = Me[w];
          if (top == 0) {  // one cursor atomic per word of M[e]
            if (!bits) continue;
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(a.out, (unsigned long long)__popc(bits));
            base = __shfl_sync(FULL, base, 0);
            if ((bits >> lane) & 1u)
              put_tuple(a, base + __popc(bits & ((1u << lane) - 1u)), row, je, list[32 * w + lane], 0u);
            continue;
          }
          if (!bits) continue;  // k = 4: lane t of the word counts M[e] & M[t], one cursor atomic per word
          const bool has = (bits >> lane) & 1u;
          const uint32_t t = 32 * w + lane;
          const uint32_t* Mt = masks + mask_off(t);
          const uint32_t lt = (t + 31) >> 5;
          uint32_t n = 0;
          if (has)
            for (uint32_t x = 0; x < lt; x++) n += __popc(Me[x] & Mt[x]);
          const uint32_t ex = warp_exclusive_scan(n, lane);
          const uint32_t sum = __shfl_sync(FULL, ex + n, 31);
          unsigned long long pos = 0;
          if (lane == 0 && sum) pos = atomicAdd(a.out, (unsigned long long)sum);
          pos = __shfl_sync(FULL, pos, 0) + ex;
          if (has)
            for (uint32_t x = 0; x < lt && pos < a.capacity; x++)
              for (uint32_t r = Me[x] & Mt[x]; r; r &= r - 1) put_tuple(a, pos++, row, je, list[t], list[32 * x + __ffs(r) - 1]);
        }
        continue;
      }
      if (top == 0) {
        for (uint32_t w = lane; w < we; w += 32) acc += __popc(Me[w]);
      } else if (top == 1) {
        // k = 4: sum over t in M[e] of popc(M[e] & M[t]); M[t] has bits below t only,
        // in its ceil(t/32) words.
        if (GLOBAL && we > 8) {
          // Long rows in global memory: the warp walks the set bits t together and
          // lanes take consecutive words of the two rows (coalesced reads).
          for (uint32_t w0 = 0; w0 < we; w0++) {
            uint32_t bits = Me[w0];
            while (bits) {
              const uint32_t t = 32 * w0 + (__ffs(bits) - 1);
              bits &= bits - 1;
              const uint32_t* Mt = masks + mask_off(t);
              for (uint32_t x = lane; x < ((t + 31) >> 5); x += 32) acc += __popc(Me[x] & Mt[x]);
            }
          }
        } else {
          // Each lane takes one t of a word of M[e]; odd row lengths keep the
          // lanes' rows in different shared-memory banks.
          for (uint32_t w = 0; w < we; w++) {
            const uint32_t bits = Me[w];
            if (!((bits >> lane) & 1u)) continue;
            const uint32_t t = 32 * w + lane;
            // mask_off(t) from the word's first row: rows 32w+1 .. 32w+31 are (w+1)|1
            // words long, row 32w is w|1 words long.
            const uint32_t first = mask_off(32 * w + 1);
            const uint32_t* Mt = masks + (lane ? first + (lane - 1) * ((w + 1) | 1u) : first - (w | 1u));
            for (uint32_t x = 0; x < ((t + 31) >> 5); x++) acc += __popc(Me[x] & Mt[x]);
          }
        }
      } else {
        // Warp-cooperative depth-first search; S[d], R[d] live in the warp's stack.
        uint32_t* S = stack;
        uint32_t* R = stack + (a.k - 2) * W;
        for (uint32_t w = lane; w < W; w += 32) S[w] = R[w] = (w < we) ? Me[w] : 0u;
        __syncwarp();
        int d = 0;
        while (d >= 0) {
          uint32_t* Sd = S + (uint64_t)d * W;
          uint32_t* Rd = R + (uint64_t)d * W;
          if (d == top) {
            for (uint32_t w = lane; w < W; w += 32) acc += __popc(Sd[w]);  // summed over lanes at the end
            d--;
            continue;
          }
          // lowest remaining candidate t in Rd
          uint32_t t = 0xffffffffu;
          for (uint32_t w0 = 0; w0 < W && t == 0xffffffffu; w0 += 32) {
            const uint32_t w = w0 + lane;
            const uint32_t v = w < W ? Rd[w] : 0u;
            const uint32_t nz = __ballot_sync(FULL, v != 0);
            if (nz) {
              const uint32_t src = __ffs(nz) - 1;
              const uint32_t vw = __shfl_sync(FULL, v, src);
              t = 32 * (w0 + src) + (__ffs(vw) - 1);
            }
          }
          if (t == 0xffffffffu) {
            d--;
            continue;
          }
          __syncwarp();
          if (lane == 0) Rd[t >> 5] &= ~(1u << (t & 31));
          const uint32_t* Mt = masks + mask_off(t);
          const uint32_t lt = (t + 31) >> 5;  // words of M[t]; the rest are 0
          uint32_t* Sn = S + (uint64_t)(d + 1) * W;
          uint32_t* Rn = R + (uint64_t)(d + 1) * W;
          uint32_t cnt = 0;
          for (uint32_t w = lane; w < W; w += 32) {
            const uint32_t v = w < lt ? Sd[w] & Mt[w] : 0u;
            Sn[w] = v;
            Rn[w] = v;
            cnt += __popc(v);
          }
          cnt = warp_sum_u32(cnt);
          __syncwarp();
          if (cnt >= (uint32_t)(top - d)) d++;
        }
      }
    }
    if (a.graph_rows) {  // batch: each warp's share of this pivot goes to its graph
      const unsigned long long pc = warp_sum_u64(acc - acc_before);
      acc = acc_before;
      if (lane == 0 && pc) atomicAdd(&a.out[graph_of(a.graph_rows, a.num_graphs, row)], pc);
    }
    __syncthreads();
  }
  acc = warp_sum_u64(acc);
  if (!LIST && lane == 0 && acc) atomicAdd(a.out, acc);
}

}  // namespace

uint64_t clique_slot_words(uint32_t cmax, uint32_t k) {
  const uint64_t W = mask_len(cmax);
  // DFS stacks (k >= 5) are sized for the 256-thread CTAs that run those k.
  return (uint64_t)cmax + (uint64_t)mask_off(cmax) + (k >= 5 ? (uint64_t)NW * 2 * (k - 2) * W : 0);
}

uint32_t clique_smem_cap(uint32_t k, int device) {
  static std::atomic<int> optin[64];
  int o = (device >= 0 && device < 64) ? optin[device].load() : 0;
  if (o <= 0) {
    cudaDeviceGetAttribute(&o, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    if (device >= 0 && device < 64) optin[device].store(o);
  }
  // Leave room for the kernel's static shared memory (s_unit, s_scan: 4,112 bytes
  // in the 1,024-thread variant).
  const uint64_t budget = o > 4608 ? (uint64_t)o - 4608 : 0;
  uint32_t lo = 32, hi = kCliqueSmemMax;
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1) / 2;
    if (clique_slot_words(mid, k) * 4 <= budget) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// SMs x resident CTAs of the shared-memory clique kernel with `bytes` of
// dynamic shared memory; looked up once per (device, size), so that launches
// captured into a CUDA graph after a direct run make no occupancy query.
template <int NT, bool LIST>
static int resident_ctas(int dev, size_t bytes) {
  static std::mutex mu;
  static std::map<std::pair<int, size_t>, int> cache;
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find({dev, bytes});
  if (it != cache.end()) return it->second;
  int sms = 0, per = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_clique_cta<false, NT, LIST>, NT, bytes);
  const int g = std::max(sms, 1) * std::max(per, 1);
  cache[{dev, bytes}] = g;
  return g;
}

// Shared-memory launch with NT threads per CTA.
template <int NT, bool LIST>
static cudaError_t launch_shared(const CliqueArgs& a, uint32_t pos_begin, uint32_t pos_end, uint32_t* counter,
                                 uint32_t cmax, uint32_t W, uint64_t slot, int grid, cudaStream_t st) {
  const size_t bytes = slot * 4;
  // Raise the kernel's dynamic shared-memory limit only when a launch needs more
  // than any before it (so replays of captured launches never call this).
  static std::atomic<int> set_bytes[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if ((int)bytes > set_bytes[dev].load()) {
    cudaError_t e = cudaFuncSetAttribute(k_clique_cta<false, NT, LIST>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)bytes);
    if (e != cudaSuccess) return e;
    int prev = set_bytes[dev].load();
    while ((int)bytes > prev && !set_bytes[dev].compare_exchange_weak(prev, (int)bytes)) {
    }
  }
  if (grid <= 0)  // fill the GPU: SMs x resident CTAs at this shared-memory size, at most one per pivot
    grid = (int)std::min<uint64_t>(pos_end - pos_begin, (uint64_t)resident_ctas<NT, LIST>(dev, bytes));
  k_clique_cta<false, NT, LIST><<<grid, NT, bytes, st>>>(a, pos_begin, pos_end, counter, cmax, W, nullptr, slot);
  return cudaGetLastError();
}

cudaError_t launch_clique_warp(const CliqueArgs& a, uint32_t pos_begin, uint32_t pos_end, uint32_t* counter,
                               int sms, cudaStream_t st, bool list, bool overlap) {
  if (pos_end <= pos_begin) return cudaSuccess;
  // Grabs of up to four pivots, small enough that every resident warp gets several.
  const uint32_t n = pos_end - pos_begin, warps = 5u * NW * (uint32_t)std::max(1, sms);
  const uint32_t grab = std::max(1u, std::min(4u, n / (16 * warps)));
  const unsigned grid = std::max(1u, std::min(5u * (uint32_t)std::max(1, sms), (n + NW * grab - 1) / (NW * grab)));
  // The batch's form where there is no core (see above).
  const auto kernel = list ? k_clique_warp<true, HashArea>
                           : a.core ? k_clique_warp<false, HashArea> : k_clique_warp<false, RowsArea>;
  return launch_overlapped(kernel, grid, kCtaThreads, 0, st, overlap, 0, a,
                           pos_begin, pos_end, grab, counter);
}

cudaError_t launch_clique_mid(const CliqueArgs& a, uint32_t pos_begin, uint32_t pos_end, uint32_t* counter,
                              uint32_t cmax, int sms, cudaStream_t st, bool overlap) {
  if (pos_end <= pos_begin) return cudaSuccess;
  static std::atomic<bool> allowed[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!allowed[dev].load()) {
    const cudaError_t e = cudaFuncSetAttribute(k_clique_mid, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)mid_bytes(kCliqueMidMax));
    if (e != cudaSuccess) return e;
    allowed[dev].store(true);
  }
  const uint32_t bytes = mid_bytes(cmax), per = std::max(1u, std::min(5u, (228u << 10) / (bytes + 2048)));
  const unsigned grid = std::min<unsigned>(pos_end - pos_begin, per * (unsigned)std::max(1, sms));
  return launch_overlapped(k_clique_mid, grid, kCtaThreads, bytes, st, overlap, 0, a, pos_begin, pos_end, counter, cmax);
}

template <bool LIST>
static cudaError_t launch_cta(const CliqueArgs& a, uint32_t pos_begin, uint32_t pos_end, uint32_t* counter,
                              uint32_t cmax, uint32_t* gscratch, int grid, cudaStream_t st) {
  const uint32_t W = mask_len(cmax);
  const uint64_t slot = clique_slot_words(cmax, a.k);
  const bool wide = a.k <= 4 && cmax > kCliqueWideMin;
  if (gscratch) {
    if (wide) {
      // One 1,024-thread CTA per SM in place of two 256-thread ones.
      int sms = 0, dev = 0;
      cudaGetDevice(&dev);
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      grid = std::max(1, std::min(grid, sms));
      k_clique_cta<true, 1024, LIST><<<grid, 1024, 0, st>>>(a, pos_begin, pos_end, counter, cmax, W, gscratch,
                                                            slot);
    } else {
      k_clique_cta<true, kCtaThreads, LIST><<<grid, kCtaThreads, 0, st>>>(a, pos_begin, pos_end, counter, cmax, W,
                                                                          gscratch, slot);
    }
    return cudaGetLastError();
  }
  return wide ? launch_shared<1024, LIST>(a, pos_begin, pos_end, counter, cmax, W, slot, grid, st)
              : launch_shared<kCtaThreads, LIST>(a, pos_begin, pos_end, counter, cmax, W, slot, grid, st);
}

cudaError_t launch_clique_cta(const CliqueArgs& a, uint32_t pos_begin, uint32_t pos_end, uint32_t* counter,
                              uint32_t cmax, uint32_t* gscratch, int grid, cudaStream_t st, bool list) {
  if (pos_end <= pos_begin) return cudaSuccess;
  return list ? launch_cta<true>(a, pos_begin, pos_end, counter, cmax, gscratch, grid, st)
              : launch_cta<false>(a, pos_begin, pos_end, counter, cmax, gscratch, grid, st);
}

}  // namespace eh
