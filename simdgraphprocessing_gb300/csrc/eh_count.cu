// Pattern-count kernels over an encoded matrix.
//
// Triangles (apps/undirected_triangle_counting.cpp:27-65) sum, over every pivot
// row i and every j in A_i = row(i), the intersection |A_i ∩ row(j)|.  Rows are
// pruned (nbr < node), so row(j) only holds ids below j and the count for the
// pair equals |{a in A_i : a < j} ∩ row(j)|; with A_i sorted and j = A_i[e]
// those are exactly A_i[0..e).  Lollipops (apps/undirected_lollipop_counting.cpp:
// 27-77) run on the full rows and count, for y = A_x[e], the z in A_x ∩ row(y)
// with z < y -- the same bounded intersection -- each weighted by |A_x|.
//
// The same kernels do both.  Pivots go by size, largest first, handed out
// dynamically with atomic counters (the GPU form of par_for_range's block
// stealing, src/common.hpp:214-276): above 2,048 entries in units of unit_span
// positions to k_pivots_heavy; above kMidMax in units, and from there down to
// light_max whole, to a CTA of k_pivots_cta; up to light_max to a warp of
// k_pivots_warp, which takes the tiniest sixteen at a time.  The per-pair
// choices stand for the reference's intersection kernels: ANDs of words + popc
// (bitset ∩ bitset, intersection.hpp:880-955), probes of A_i[t], t < e, into
// row(j) (uint ∩ bitset, :1023-1058, or the galloping search of :393-584) and
// streams of row(j) tested against the staged pivot (merge, :696-771).
// Per-lane counts stay in registers; one u64 atomic per CTA at the end replaces
// the reference's per-thread padded t_count array.
#include <algorithm>
#include <atomic>
#include <cstdint>

#include "eh_kernels.cuh"

namespace eh {

namespace {

constexpr int NWARPS = kCtaThreads / 32;
constexpr int kLargeWarps = 8, kMidWarps = 4;  // warps of a k_pivots_cta CTA for the two tiers
constexpr uint32_t kStreamMinE = 256;  // core rows: consider streaming row(j) only past this many probes

struct __align__(16) HeavySmem {
  unsigned long long words[kCtaWordCap];
  unsigned long long abits[kCoreAndMax / 64];  // pivot ∩ [0, min(core_k, kCoreAndMax)) as bits
  uint64_t bar;  // completion of the unit's bulk copy
  uint32_t unit;
};
// Device error flag (PivotArgs::flags): a bulk copy's wait ran out.
constexpr uint32_t kErrBulkWait = 1u;

// Warp, CTA, then one u64 atomic per CTA into the single count; the last CTA of
// the call's kernels writes the result and resets the queue, so that a call needs
// no memset before it and a blocking call no copy after it (out is then host memory).
template <int NW = NWARPS>
__device__ __forceinline__ void cta_add(unsigned long long acc, const PivotArgs& a) {
  __shared__ unsigned long long s_red[NW];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  acc = warp_sum_u64(acc);
  if (lane == 0) s_red[warp] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long tot = 0;
    for (int w = 0; w < NW; w++) tot += s_red[w];
    unsigned long long* sum = reinterpret_cast<unsigned long long*>(a.queue + 6);
    if (tot && !a.graph_rows) atomicAdd(sum, tot);
    __threadfence();
    if (atomicAdd(&a.queue[5], 1u) == a.ctas - 1) {
      __threadfence();
      if (!a.graph_rows) a.out[0] = atomicExch(sum, 0ull);
      if (a.report) a.out[1] = atomicExch(a.flags, 0u);
      for (int k = 0; k < 6; k++) a.queue[k] = 0u;
    }
  }
}

__device__ __forceinline__ uint32_t ilog2p1(uint32_t x) { return 32u - __clz(x | 1u); }

// |{t < e : L[t] in B}| with j = L[e]; warp-uniform result.  A is the pivot row
// (shared or global payload), L its sorted elements.
__device__ uint32_t pair_count_warp(const uint32_t* L, uint32_t e, const RowView& A, const RowView& B,
                                    uint32_t j, uint32_t lane) {
  if (B.card == 0 || e == 0) return 0;
  uint32_t c = 0;
  if (A.type == TY_BITSET && B.type == TY_BITSET) {
    const uint32_t lo = max(A.aux, B.aux);
    const uint32_t hi = min(min(A.aux + A.len, B.aux + B.len), (j >> 6) + 1);
    if (hi <= lo) return 0;
    if (hi - lo <= 2 * e) {  // 128-bit AND + popcount over the overlapping words below j
      c = bitset_and_lane(A.p, A.aux, B.p, B.aux, B.len, lo, hi, j >> 6, (1ull << (j & 63)) - 1ull, lane);
      return warp_sum_u32(c);
    }
  }
  // Probe cost: e lookups into B.  Stream cost: |B| lookups into the pivot.
  // Merge cost (uint rows): e + |B| steps of a merge path.
  bool stream = false;
  if (B.type == TY_UINT) {
    const uint32_t look = (A.type == TY_BITSET) ? 1u : ilog2p1(e);
    const uint64_t probe_cost = (uint64_t)e * ilog2p1(B.card) * 4u, stream_cost = (uint64_t)B.card * look;
    if (A.type != TY_BITSET && e >= 64 && (uint64_t)e + B.card < min(probe_cost, stream_cost)) {
      const uint32_t* b = static_cast<const uint32_t*>(B.p);
      const uint32_t nb = lower_bound_u32(b, 0, B.card, j);  // full rows hold elements >= j too
      return warp_sum_u32(merge_path_lane(L, e, b, nb, lane));
    }
    stream = stream_cost < probe_cost;
  } else if (B.type == TY_PSHORT) {
    stream = (uint64_t)B.card * ilog2p1(e) < (uint64_t)e * (B.aux + ilog2p1(B.card)) * 4u;
  }
  if (!stream) {
    for (uint32_t t = lane; t < e; t += 32) c += row_contains(B, L[t]);
  } else if (A.type == TY_BITSET) {
    warp_for_each(B, j, lane, [&](uint32_t y) { c += row_contains(A, y); });
  } else {
    warp_for_each(B, j, lane, [&](uint32_t y) {
      const uint32_t p = lower_bound_u32(L, 0, e, y);
      c += (p < e && L[p] == y);
    });
  }
  return warp_sum_u32(c);
}

// Per-lane part of |{t < e : L[t] in B}| by streaming B's elements below j and
// looking each up in the pivot (a bit test for a bitset pivot, else a binary
// search of L[0, e)); the caller sums over the warp.
__device__ __forceinline__ uint32_t pair_count_stream(const uint32_t* L, uint32_t e, const RowView& A,
                                                      const RowView& B, uint32_t j, uint32_t lane) {
  uint32_t c = 0;
  if (A.type == TY_BITSET) {
    warp_for_each(B, j, lane, [&](uint32_t y) { c += row_contains(A, y); });
  } else {
    warp_for_each(B, j, lane, [&](uint32_t y) {
      const uint32_t p = lower_bound_u32(L, 0, e, y);
      c += (p < e && L[p] == y);
    });
  }
  return c;
}

// Pivots above kCtaListCap entries (decoded lists in global memory): 6 resident
// CTAs per SM, 40 registers per thread (the per-pair choice keeps many values
// live, and at 32 registers it spilled).
template <bool LOLLI>
__global__ void __launch_bounds__(kCtaThreads, 6) k_pivots_heavy(PivotArgs a, const uint2* __restrict__ units,
                                                              uint32_t n_units) {
  __shared__ HeavySmem s;
  overlap_begin();
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long acc = 0;
  uint32_t phase = 0;
  if (threadIdx.x == 0) mbar_init(&s.bar);

  for (;;) {
    if (threadIdx.x == 0) s.unit = atomicAdd(&a.queue[0], 1u);
    __syncthreads();  // also: every thread is done with the previous unit's staging
    const uint32_t unit = s.unit;
    if (unit >= n_units) break;
    const uint2 uu = units[unit];
    if (uu.x >= a.n_giant) break;  // units come in pivot order, the largest first
    const uint32_t i = a.order[uu.x];
    RowView A = load_view(a.desc, a.arena, i);
    // Bitset words are staged by one bulk (TMA) copy: row payloads start on
    // 16-byte boundaries and are padded to 16 bytes.
    const bool bulk_words = A.type == TY_BITSET && A.len <= kCtaWordCap;
    if (bulk_words) {
      if (threadIdx.x == 0) bulk_copy_g2s(s.words, A.p, (8 * A.len + 15) & ~15u, &s.bar);
      if (!mbar_wait(&s.bar, phase)) {
        // Record the failure, then give the copy in flight a second bounded
        // wait before the buffer is used or the CTA exits.
        if (threadIdx.x == 0) atomicOr(a.flags, kErrBulkWait);
        mbar_wait(&s.bar, phase);
      }
      phase ^= 1u;
    }
    const uint32_t* L =
        (A.type == TY_UINT) ? static_cast<const uint32_t*>(A.p) : a.giant_lists + a.giant_off[uu.x];
    if (bulk_words) A.p = s.words;
    const bool use_core = a.core_k != 0;
    const uint32_t and_k = min(a.core_k, kCoreAndMax);
    if (use_core) {
      for (uint32_t k = threadIdx.x; k < (and_k >> 6); k += kCtaThreads) s.abits[k] = 0ull;
      __syncthreads();
      for (uint32_t k = threadIdx.x; k < A.card; k += kCtaThreads) {
        const uint32_t x = L[k];
        if (x < and_k) atomicOr(&s.abits[x >> 6], 1ull << (x & 63));
      }
    }
    __syncthreads();
    const uint32_t c = A.card;
    const uint32_t e0 = 1 + uu.y * a.unit_span;
    const uint32_t e1 = min(c, e0 + a.unit_span);
    unsigned long long uacc = 0;
    for (uint32_t e = e0 + warp; e < e1; e += NWARPS) {
      const uint32_t j = L[e];
      uint32_t cnt;
      if (use_core && j < a.core_k) {
        // Core row j holds row(j) ∩ [0, j).  Cheapest of: AND it with the pivot's
        // bits (j within the staged bits; wj words), probe it at the e pivot
        // elements below j (e words), or stream row(j) itself and look each
        // element up in the pivot (|row(j)| lookups; rows past the highest-degree
        // ones are short while e grows with the pivot).
        const unsigned long long* row = a.core + core_row_offset(j);
        const uint32_t wj = (j + 63) >> 6;
        cnt = 0;
        if (j <= and_k && wj <= e) {
          // 8-byte words: padding the core rows to 16-byte pairs for 128-bit
          // loads here measured 0.15 ms slower per count at scale 22.
          for (uint32_t w = lane; w < wj; w += 32) cnt += __popcll(s.abits[w] & __ldg(row + w));
        } else {
          bool stream = false;
          RowView B;
          if (e > kStreamMinE) {
            B = load_view(a.desc, a.arena, j);
            stream = (uint64_t)B.card * (A.type == TY_BITSET ? 1u : ilog2p1(e)) < e;
          }
          if (stream) {
            cnt = pair_count_stream(L, e, A, B, j, lane);
          } else {
            for (uint32_t t = lane; t < e; t += 32) {
              const uint32_t x = L[t];
              cnt += (uint32_t)((__ldg(row + (x >> 6)) >> (x & 63)) & 1ull);
            }
          }
        }
        cnt = warp_sum_u32(cnt);
      } else {
        const RowView B = load_view(a.desc, a.arena, j);
        cnt = pair_count_warp(L, e, A, B, j, lane);
      }
      if (lane == 0) uacc += LOLLI ? (unsigned long long)cnt * c : (unsigned long long)cnt;
    }
    // Pshort pivots of >= 65,536 entries: less what the reference's u16 counts drop of the
    // same pairs (a loop of its own: in the one above it spills registers).
    if (A.type == TY_PSHORT && c >= 65536u) {
      unsigned long long drop = 0;
      for (uint32_t e = e0 + threadIdx.x; e < e1; e += kCtaThreads)
        drop += pshort_pair_drop(A, load_view(a.desc, a.arena, L[e]), L[e]);
      drop = warp_sum_u64(drop);
      if (lane == 0) uacc -= LOLLI ? drop * c : drop;
    }
    if (a.graph_rows) {  // batch: this unit's count goes to its graph
      if (lane == 0 && uacc) atomicAdd(&a.out[graph_of(a.graph_rows, a.num_graphs, i)], uacc);
    } else {
      acc += uacc;
    }
    __syncthreads();
  }

  cta_add(acc, a);
  overlap_end();
}

// What the kernels below count: triangles; lollipops by the definition (full
// rows, each hit weighted by its pivot's card); or lollipops of a symmetric
// matrix without self-loops, where every triangle {i > j > k} counts |A_i| +
// |A_j| + |A_k|: pivots then hold only their entries below i (PivotArgs::lcard),
// so hubs are no pivots of 10^5 entries (R-MAT scale 20: 4.8 ms by definition).
enum Mode { kTri = 0, kFull = 1, kSym = 2 };

// ---- pivots of up to kCtaListCap entries: one warp or one CTA each ----
// Per pivot, staged in the group's shared-memory slice:
//  * jc[e] = (word offset of core row j, j) for j = A_i[e];
//  * word / widx: the non-zero 64-bit words of the pivot's elements below
//    core_k and their word indices, cfirst[ch] the position of the first
//    element of word 32 ch;
//  * bm: the elements of [base, base + win) as bits, base = A_i[0] rounded
//    down to 64, then kHashBits bits with bit x mod kHashBits set for the
//    elements x past the window.
// The pairs (i, j) then take one of two paths, split at the first e with
// A_i[e] >= core_k (the list is ascending):
//  * j < core_k: a lane keeps one pivot word of 32 in registers and walks the
//    e's: core row j's word under it is loaded, ANDed and added to a
//    carry-save counter.  Nothing is reduced per pair and four pairs' loads are
//    in flight; only the pivot's non-zero words are touched.  (One warp per
//    pair, with the whole overlap ANDed or every element probed and a warp sum
//    per pair, took 6.76 ms for the heavy pivots of an R-MAT scale-22 graph.)
//  * j >= core_k: row(j) is streamed, 8 lanes per row and 16 bytes per lane,
//    and each element is tested in bm; a hashed hit past the window is
//    confirmed by a binary search.  A bitset row of at most 2 e words is ANDed
//    with the window word by word.  Longer bitset rows, pshort rows and rows of
//    more than kProbeRatio e entries are probed at the e pivot elements instead.
// What bounds it: instruction issue (about 11 instructions per 32 words and
// per 16 streamed entries), and for the core's words the L1: a load in flight
// holds an L1 line, so shared memory a slice does not need is left to it (at R-MAT
// scale 22 the warp tier took 4.08 ms with a 32,768-bit window, which leaves
// L1 28 KB per SM, 2.61 ms with 8,192 + 16,384 hashed bits).
constexpr uint32_t kProbeRatio = 24;
constexpr uint32_t kHashBits = 16384;

struct Slice {
  uint2* jc;
  unsigned long long* word;
  uint16_t* widx;
  uint16_t* cfirst;
  uint32_t* rcnt;  // CTA groups: per 32 entries, word starts | elements below core_k << 16
  uint32_t* bm;
  // kSym: |A_i| + |A_j| of entry e, and its word's position mod 32.
  uint32_t* wt;
  uint8_t* wp;
};
// Bytes of a slice for pivots of up to cap entries (a multiple of 32) and a
// window of win bits (a multiple of 4,096).
template <int NW, int MODE>
__host__ __device__ constexpr uint32_t slice_bytes(uint32_t cap, uint32_t win) {
  return (cap * (MODE == kSym ? 23 : 18) + (cap / 32 + 1) * 2 + (NW > 1 ? cap / 32 * 4 : 0) + (win + kHashBits) / 8 + 31) & ~15u;
}
template <int NW, int MODE>
__device__ __forceinline__ Slice make_slice(char* p, uint32_t cap, uint32_t win) {
  Slice s;
  s.bm = reinterpret_cast<uint32_t*>(p);
  s.jc = reinterpret_cast<uint2*>(p + (win + kHashBits) / 8);
  s.word = reinterpret_cast<unsigned long long*>(s.jc + cap);
  s.rcnt = reinterpret_cast<uint32_t*>(s.word + cap);
  s.wt = s.rcnt + (NW > 1 ? cap / 32 : 0);
  s.widx = reinterpret_cast<uint16_t*>(s.wt + (MODE == kSym ? cap : 0));
  s.cfirst = s.widx + cap;
  s.wp = reinterpret_cast<uint8_t*>(s.cfirst + cap / 32 + 1);
  return s;
}
template <int NW>
__device__ __forceinline__ void group_sync() {
  if (NW == 1) __syncwarp();
  else __syncthreads();
}

// Carry-save counter of 64-bit words, eight at a time: the popcount unit (16
// lanes per cycle and SM) sees one word in eight.
struct WordSum {
  uint32_t one[2], two[2], four[2], eights;
  __device__ __forceinline__ void clear() { one[0] = one[1] = two[0] = two[1] = four[0] = four[1] = eights = 0; }
  __device__ __forceinline__ void add8(const unsigned long long (&v)[8], const uint32_t (&w)[2]) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
      uint32_t x[8];
#pragma unroll
      for (int u = 0; u < 8; u++) x[u] = (uint32_t)(v[u] >> (32 * h)) & w[h];
      const uint32_t a = csa(one[h], x[0], x[1]), b = csa(one[h], x[2], x[3]), f = csa(two[h], a, b);
      const uint32_t c = csa(one[h], x[4], x[5]), d = csa(one[h], x[6], x[7]), g = csa(two[h], c, d);
      eights += __popc(csa(four[h], f, g));
    }
  }
  __device__ __forceinline__ uint32_t total() const {
    return 8 * eights + 4 * (__popc(four[0]) + __popc(four[1])) + 2 * (__popc(two[0]) + __popc(two[1])) +
           __popc(one[0]) + __popc(one[1]);
  }
};

// Bit-sliced counters of hits per bit of a lane's word over a chunk's e's: at most
// 256 per warp (a CTA tier's e's are shared by its warps, a warp's pivot has 160).
constexpr int kPlanes = 9;
__device__ __forceinline__ void add_planes(uint32_t (&plane)[2][kPlanes], const unsigned long long (&v)[8],
                                           const uint32_t (&w)[2]) {
#pragma unroll
  for (int h = 0; h < 2; h++) {
    uint32_t x[8];
#pragma unroll
    for (int u = 0; u < 8; u++) x[u] = (uint32_t)(v[u] >> (32 * h)) & w[h];
    uint32_t* p = plane[h];
    const uint32_t a = csa(p[0], x[0], x[1]), b = csa(p[0], x[2], x[3]), f = csa(p[1], a, b);
    const uint32_t c = csa(p[0], x[4], x[5]), d = csa(p[0], x[6], x[7]), g = csa(p[1], c, d);
    uint32_t carry = csa(p[2], f, g);
#pragma unroll
    for (int q = 3; q < kPlanes; q++) {
      const uint32_t t = p[q] & carry;
      p[q] ^= carry;
      carry = t;
    }
  }
}

// This lane's part (of 8: sl) of the members of a pivot, as bm and jc hold them, in a
// pshort row of u16 stream h, below j unless kTri; kSym: the sum of we + |A_y| over
// them.  Partition by partition, where a probe walks the headers for each of the
// pivot's elements (R-MAT scale 22, pshort: 8.06 -> 7.05 ms a count).  Out of line: in
// it, the uint rows' loop loses 2%.
template <int MODE>
__device__ __noinline__ unsigned long long pshort_hits(const uint16_t* h, uint32_t len, uint32_t sl, uint32_t j,
                                                       const uint32_t* bm, const uint2* jc, uint32_t c, uint32_t base,
                                                       uint32_t win, uint32_t we, const RowDesc* desc) {
  unsigned long long sum = 0;
  for (uint32_t i = 0; i < len;) {
    const uint32_t hb = (uint32_t)h[i] << 16, m = (uint32_t)h[i + 1] + 1;
    if (MODE != kTri && hb >= j) break;
    for (uint32_t k = sl; k < m; k += 8) {
      const uint32_t y = hb | h[i + 2 + k], dy = y - base, at = dy < win ? dy : win + (y & (kHashBits - 1));
      if (!((bm[at >> 5] >> (y & 31)) & 1u) || (MODE != kTri && y >= j)) continue;
      if (dy >= win) {
        uint32_t lo = 0, hi = c;
        while (lo < hi) {
          const uint32_t mid = (lo + hi) >> 1;
          if (jc[mid].y < y) lo = mid + 1;
          else hi = mid;
        }
        if (lo == c || jc[lo].y != y) continue;
      }
      sum += MODE == kSym ? (unsigned long long)we + desc[y].card : 1ull;
    }
    i += m + 2;
  }
  return sum;
}

// This lane's part of the count of pivot i's pairs e in [e0, e1), by a group
// of NW warps (gw: this warp's index in it): the returned count plus what went
// into `sum`; kSym: everything goes into `wsum`, weighted.  But for kTri the rows
// are full ones, which hold elements >= j too.  The group's slice is free for the
// next pivot on return, bm zero.
template <int NW, int MODE, bool LONG>
__device__ __forceinline__ uint32_t pivot_count(const PivotArgs& a, const RowView& A, uint32_t e0, uint32_t e1,
                                                const Slice& s, uint32_t win, uint32_t* scan, uint32_t lane,
                                                uint32_t gw, WordSum& sum, uint32_t card_i,
                                                unsigned long long& wsum) {
  constexpr bool LOLLI = MODE != kTri, SYM = MODE == kSym;
  const uint32_t c = A.card, core_k = a.core_k, lt = (1u << lane) - 1u, tid = gw * 32 + lane;
  const auto put = [&](uint32_t k, uint32_t x) {
    if (SYM && k >= c) return;  // entries past the pivot itself
    s.jc[k] = make_uint2(x < core_k ? core_offset32(x) : 0u, x);
    if (SYM) s.wt[k] = card_i + a.desc[x].card;
  };
  if (NW == 1) warp_decode_to<LONG>(A, lane, put);
  else cta_decode_to<NW * 32>(A, scan, put);
  uint32_t* word32 = reinterpret_cast<uint32_t*>(s.word);
  if (NW > 1)
    for (uint32_t k = tid; k < c; k += NW * 32) s.word[k] = 0ull;
  group_sync<NW>();

  const uint32_t base = s.jc[0].y & ~63u, last = s.jc[c - 1].y;
  const bool stream_any = last >= core_k, wide = last - base >= win;
  const uint32_t rounds = (c + 31) >> 5;
  uint32_t nw = 0, ea = 0, pre0 = 0, pre1 = 0;  // non-zero words; elements below core_k
  if (NW > 1) {
    for (uint32_t r = gw; r < rounds; r += NW) {
      const uint32_t k = 32 * r + lane, x = k < c ? s.jc[k].y : 0xffffffffu;
      const bool in = x < core_k;  // false past c: core_k <= kCoreMaxK
      const uint32_t hb = __ballot_sync(FULL, in && (k == 0 || (s.jc[k - 1].y >> 6) != (x >> 6)));
      const uint32_t ab = __ballot_sync(FULL, in);
      if (lane == 0) s.rcnt[r] = __popc(hb) | ((uint32_t)__popc(ab) << 16);
    }
    group_sync<NW>();
    const uint32_t v0 = lane < rounds ? s.rcnt[lane] : 0u, v1 = lane + 32 < rounds ? s.rcnt[lane + 32] : 0u;
    pre0 = warp_exclusive_scan(v0, lane);  // 16-bit halves: sums stay below 2^12
    const uint32_t t0 = __shfl_sync(FULL, pre0 + v0, 31);
    pre1 = t0 + warp_exclusive_scan(v1, lane);
    const uint32_t tot = __shfl_sync(FULL, pre1 + v1, 31);
    nw = tot & 0xffffu;
    ea = tot >> 16;
  }
  uint32_t run = 0;  // NW == 1: words before this round
  for (uint32_t r = gw; r < rounds; r += NW) {
    const uint32_t k = 32 * r + lane, x = k < c ? s.jc[k].y : 0xffffffffu;
    const bool in = x < core_k;
    const bool head = in && (k == 0 || (s.jc[k - 1].y >> 6) != (x >> 6));
    const uint32_t hb = __ballot_sync(FULL, head);
    if (NW > 1) run = (r < 32 ? __shfl_sync(FULL, pre0, r) : __shfl_sync(FULL, pre1, r - 32)) & 0xffffu;
    const uint32_t pos = run + __popc(hb & (lt | (1u << lane))) - 1;
    if (head) {
      if (NW == 1) s.word[pos] = 0ull;
      s.widx[pos] = (uint16_t)(x >> 6);
      if (!(pos & 31)) s.cfirst[pos >> 5] = (uint16_t)k;
    }
    if (NW == 1) {
      ea += __popc(__ballot_sync(FULL, in));
      run += __popc(hb);
      __syncwarp();
    }
    if (in) atomicOr(&word32[2 * pos + ((x >> 5) & 1)], 1u << (x & 31));
    if (SYM && in) s.wp[k] = (uint8_t)(pos & 31);
    if (stream_any && k < c) {
      const uint32_t d = x - base;
      atomicOr(&s.bm[(d < win ? d : win + (x & (kHashBits - 1))) >> 5], 1u << (x & 31));
    }
  }
  if (NW == 1) nw = run;
  group_sync<NW>();

  // ---- j < core_k ----
  uint32_t cnt = 0;
  const uint32_t ee = min(e1, ea);
  for (uint32_t ch = 0; 32 * ch < nw; ch++) {
    const uint32_t p = 32 * ch + lane;
    const bool live = p < nw;
    const unsigned long long word = live ? s.word[p] : 0ull;
    const uint32_t w[2] = {(uint32_t)word, (uint32_t)(word >> 32)};
    const uint32_t idx = live ? s.widx[p] : 0u;
    const uint32_t first = live ? idx << 6 : 0xffffffffu;  // smallest id under this lane's word
    const unsigned long long* col = a.core + idx;
    uint32_t e = max(e0, (uint32_t)s.cfirst[ch]) + 8 * gw;
    unsigned long long v[8];
    uint32_t plane[2][kPlanes];  // kSym: hits per bit of this lane's word, bit-sliced
    if (SYM) {
#pragma unroll
      for (int q = 0; q < kPlanes; q++) plane[0][q] = plane[1][q] = 0;
    }
    const auto add = [&](uint32_t eb) {
      if (!SYM) {
        sum.add8(v, w);
        return;
      }
#pragma unroll
      for (int u = 0; u < 8; u++)
        wsum += (unsigned long long)(__popc((uint32_t)v[u] & w[0]) + __popc((uint32_t)(v[u] >> 32) & w[1])) * s.wt[eb + u];
      add_planes(plane, v, w);
    };
    for (; e + 7 < ee; e += 8 * NW) {
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const uint2 q = s.jc[e + u];
        v[u] = first < q.y ? __ldg(col + q.x) : 0ull;
      }
      add(e);
    }
    if (e < ee) {  // the last block of fewer than eight belongs to one warp
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const uint2 q = s.jc[e + u];
        v[u] = (e + u < ee && first < q.y) ? __ldg(col + q.x) : 0ull;
      }
      add(e);
    }
    if (SYM) {
      // Each element under the chunk's words takes its hits from the lane that holds its word.
      const uint32_t k1 = 32 * (ch + 1) < nw ? s.cfirst[ch + 1] : ea;
      for (uint32_t k0 = s.cfirst[ch]; k0 < k1; k0 += 32) {
        const uint32_t k = k0 + lane;
        const bool has = k < k1;
        const uint32_t owner = has ? s.wp[k] : 0u, x = has ? s.jc[k].y : 0u;
        uint32_t hits = 0;
#pragma unroll
        for (int q = 0; q < kPlanes; q++) {
          const uint32_t p0 = __shfl_sync(FULL, plane[0][q], owner), p1 = __shfl_sync(FULL, plane[1][q], owner);
          hits |= (((x & 32 ? p1 : p0) >> (x & 31)) & 1u) << q;
        }
        if (has) wsum += (unsigned long long)hits * (s.wt[k] - card_i);
      }
    }
  }

  // ---- j >= core_k ----
  if (stream_any && ea < e1) {
    // Whether L holds y, which lies past the window.
    // (Hits of kSym are weighed as they are found: wt of the row's entry plus |A_y|.)
    const auto weigh = [&](uint32_t e, uint32_t y) { wsum += (unsigned long long)s.wt[e] + a.desc[y].card; };
    const auto search = [&](uint32_t y) -> uint32_t {
      uint32_t lo = 0, hi = c;
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (s.jc[mid].y < y) lo = mid + 1;
        else hi = mid;
      }
      return lo < c && s.jc[lo].y == y;
    };
    const uint32_t sl = lane & 7, begin = max(e0, ea) + 4 * gw;
    const auto source = [&](uint32_t e) { return __ldg(reinterpret_cast<const uint4*>(a.desc) + s.jc[e].y); };
    uint4 next = make_uint4(0u, 0u, 0u, 0u);
    if (begin + (lane >> 3) < e1) next = source(begin + (lane >> 3));
    for (uint32_t eb = begin; eb < e1; eb += 4 * NW) {
      const uint32_t e = eb + (lane >> 3);
      const uint4 d = next;
      if (e + 4 * NW < e1) next = source(e + 4 * NW);
      uint32_t n = 0, j = 0;
      const uint32_t* p = nullptr;
      if (e < e1) {
        j = s.jc[e].y;
        const uint32_t type = d.w >> 30;
        p = reinterpret_cast<const uint32_t*>(a.arena + d.x);
        n = d.y;
        if (type == TY_BITSET && (d.w & 0x3fffffffu) <= 2 * e) {
          // Word pairs of row(j) against the window; words past it element by element.
          const uint32_t np = ((d.w & 0x3fffffffu) + 1) >> 1, bw = base >> 6, jw = j >> 6, ww = win >> 6;
          const unsigned long long* bm64 = reinterpret_cast<const unsigned long long*>(s.bm);
          for (uint32_t q = sl; q < np; q += 8) {
            const uint32_t w0 = d.z + 2 * q;
            if (LOLLI && w0 > jw) break;
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(p) + q);
            const unsigned long long x[2] = {lo64(v), hi64(v)};
#pragma unroll
            for (int h = 0; h < 2; h++) {
              const uint32_t wi = w0 + h;
              unsigned long long y = x[h];
              if (LOLLI && wi >= jw) y = wi > jw ? 0ull : y & ((1ull << (j & 63)) - 1ull);
              if (wi - bw < ww) {
                y &= bm64[wi - bw];
                if (!SYM) cnt += __popcll(y);
                else
                  for (; y; y &= y - 1ull) weigh(e, 64 * wi + (uint32_t)(__ffsll((long long)y) - 1));
              } else if (wide && wi > bw) {
                for (; y; y &= y - 1ull) {
                  const uint32_t id = 64 * wi + (uint32_t)(__ffsll((long long)y) - 1), hit = search(id);
                  if (!SYM) cnt += hit;
                  else if (hit) weigh(e, id);
                }
              }
            }
          }
          n = 0;
        } else if (LONG && type == TY_PSHORT && n <= kProbeRatio * e) {
          const unsigned long long hits =
              pshort_hits<MODE>(reinterpret_cast<const uint16_t*>(p), d.w & 0x3fffffffu, sl, j, s.bm, s.jc, c, base, win,
                                SYM ? s.wt[e] : 0u, a.desc);
          if (SYM) wsum += hits;
          else cnt += (uint32_t)hits;
          n = 0;
        } else if (type != TY_UINT || n > kProbeRatio * e) {
          const RowView B = load_view(a.desc, a.arena, j);
          for (uint32_t t = sl; t < e; t += 8) {
            const bool hit = row_contains(B, s.jc[t].y);
            if (!SYM) cnt += hit;
            else if (hit) wsum += s.wt[e] + (unsigned long long)(s.wt[t] - card_i);
          }
          n = 0;
        }
      }
      // Four 16-byte loads per lane in flight (128 entries of each of the four
      // rows): the rows come from L2 or DRAM and a lane's chain is one list.
      const uint32_t most = __reduce_max_sync(FULL, n);
      for (uint32_t k0 = 0; k0 < most; k0 += 128) {
        uint4 v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const uint32_t k = k0 + 32 * u + 4 * sl;
          // uint rows are padded to 16 bytes with an id no row holds (kUintPad).
          v[u] = k < n ? __ldg(reinterpret_cast<const uint4*>(p + k)) : make_uint4(kUintPad, kUintPad, kUintPad, kUintPad);
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
          if (k0 + 32 * u >= most) break;
          const uint32_t y[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
          uint32_t near = 0;  // kSym: hits in the window
          uint32_t past = 0;  // elements past the window whose hashed bit is set
#pragma unroll
          for (int h = 0; h < 4; h++) {
            const uint32_t dy = y[h] - base;
            const bool in = dy < win;
            const uint32_t at = in ? dy : win + (y[h] & (kHashBits - 1));
            uint32_t bit = (s.bm[at >> 5] >> (y[h] & 31)) & 1u;
            if (LOLLI) bit = y[h] < j ? bit : 0u;
            if (!SYM) cnt += in ? bit : 0u;
            else near |= (in ? bit : 0u) << h;
            past += in ? 0u : bit;
          }
          if (SYM)
            for (; near; near &= near - 1) {
              const uint32_t h = __ffs(near) - 1;
              weigh(e, h == 0 ? y[0] : h == 1 ? y[1] : h == 2 ? y[2] : y[3]);
            }
          if (past)
#pragma unroll
            for (int h = 0; h < 4; h++)
              if (y[h] - base >= win && (!LOLLI || y[h] < j)) {
                const uint32_t hit = search(y[h]);
                if (!SYM) cnt += hit;
                else if (hit) weigh(e, y[h]);
              }
        }
      }
    }
  }
  group_sync<NW>();
  if (stream_any) {
    for (uint32_t k = tid; k < c; k += NW * 32) {
      const uint32_t x = s.jc[k].y, d = x - base;
      s.bm[(d < win ? d : win + (x & (kHashBits - 1))) >> 5] = 0u;
    }
    group_sync<NW>();
  }
  return cnt;
}

// A warp's part of a finished pivot (or unit): into its graph's count in a
// batch (returns 0), weighted by the pivot's card for lollipops, else this
// lane's part of the one sum, where the carry-save counter may run on.
template <int MODE>
__device__ __forceinline__ unsigned long long finish_pivot(const PivotArgs& a, uint32_t i, uint32_t card, uint32_t cnt,
                                                           WordSum& sum, uint32_t lane) {
  constexpr bool LOLLI = MODE != kTri;
  if (MODE == kSym) return 0;
  if (!LOLLI && !a.graph_rows) {
    const unsigned long long pc = (unsigned long long)cnt + 8ull * sum.eights;
    sum.eights = 0;
    return pc;
  }
  if (a.core_k) {
    cnt += sum.total();
    sum.clear();
  }
  if (!a.graph_rows) return (unsigned long long)cnt * card;
  cnt = warp_sum_u32(cnt);  // below kCtaListCap^2 / 2
  if (cnt) {
    const uint32_t g = warp_graph_of(a.graph_rows, a.num_graphs, i, lane);
    if (lane == 0) atomicAdd(&a.out[g], (unsigned long long)cnt * (LOLLI ? card : 1u));
  }
  return 0;
}

// kSym: cuts a pivot's view to its entries below i (bitset rows: the words that
// hold some; what a word or a pshort row holds past them is dropped as it is decoded).
__device__ __forceinline__ void keep_below(const PivotArgs& a, RowView& A, uint32_t i) {
  A.card = a.lcard[i];
  if (A.type == TY_BITSET) A.len = min(A.len, (i >> 6) + 1 - A.aux);
}

// Pivots above the warp tier and up to kCtaListCap entries, one CTA each, in
// two launches so that the many mid-sized ones leave their shared memory to
// L1 and have few warps at a barrier: large pivots as units of unit_span
// positions (units; the giants' are k_pivots_heavy's) where some have more, or
// a range of the order from pos0 on whole (units null).
template <int NW, int MODE, bool LONG>
__global__ void __launch_bounds__(NW * 32, (MODE == kSym ? 24 : 32) / NW) k_pivots_cta(PivotArgs a, const uint2* __restrict__ units,
                                                               uint32_t n_units, uint32_t pos0, uint32_t* counter,
                                                               uint32_t cap, uint32_t win) {
  extern __shared__ __align__(16) char dyn[];
  __shared__ uint32_t s_unit, s_scan[NW];
  overlap_begin();
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Slice s = make_slice<NW, MODE>(dyn, cap, win);
  for (uint32_t k = threadIdx.x; k < (win + kHashBits) / 32; k += NW * 32) s.bm[k] = 0u;
  unsigned long long acc = 0;
  WordSum sum;
  sum.clear();
  for (;;) {
    if (threadIdx.x == 0) s_unit = atomicAdd(counter, 1u);
    __syncthreads();
    const uint32_t unit = s_unit;
    __syncthreads();
    if (unit >= n_units) break;
    const uint2 uu = units ? units[unit] : make_uint2(pos0 + unit, 0u);
    if (units && uu.x < a.n_giant) continue;
    const uint32_t i = a.order[uu.x];
    RowView A = load_view(a.desc, a.arena, i);
    const uint32_t card = A.card;
    if (MODE == kSym) keep_below(a, A, i);
    const uint32_t e0 = 1 + uu.y * a.unit_span, e1 = units ? min(A.card, e0 + a.unit_span) : A.card;
    const uint32_t cnt = pivot_count<NW, MODE, LONG>(a, A, e0, e1, s, win, s_scan, lane, warp, sum, card, acc);
    acc += finish_pivot<MODE>(a, i, card, cnt, sum, lane);
  }
  cta_add<NW>(acc + sum.total(), a);
  overlap_end();
}

// A chunk of pivots of at most kTinyMax entries as one pair space: the pivots'
// descriptors and rows are loaded by one lane each, and lane q of a step takes
// pair q of the whole chunk, so a pivot of a few pairs does not hold the warp
// for a step of its own.  A probe reads one word of core row j when
// j < core_k, else row(j).  Returns the chunk's count (each hit weighted by its
// pivot's card for lollipops).
constexpr uint32_t kTinyMax = 8;
constexpr uint32_t kTinyChunk = 16;
template <int MODE, bool LONG>
__device__ __noinline__ unsigned long long tiny_chunk(const PivotArgs& a, uint32_t base, uint32_t g, uint32_t* mem,
                                                      uint32_t lane) {
  uint32_t* list = mem;                               // kTinyChunk * kTinyMax
  uint32_t* pstart = mem + kTinyChunk * kTinyMax;     // kTinyChunk + 1
  uint32_t* poff = pstart + kTinyChunk + 1;
  uint32_t* pcard = poff + kTinyChunk;
  RowView V;
  uint32_t cl = 0, card = 0;
  if (lane < g) {
    const uint32_t i = a.order[base + lane];
    V = load_view(a.desc, a.arena, i);
    card = V.card;
    if (MODE == kSym) keep_below(a, V, i);
    cl = V.card;
  }
  const uint32_t pl = cl * (cl - 1) / 2;
  const uint32_t off = warp_exclusive_scan(cl, lane), pex = warp_exclusive_scan(pl, lane);
  const uint32_t total = __shfl_sync(FULL, pex + pl, 31);
  if (lane < g) {
    pstart[lane] = pex;
    poff[lane] = off;
    pcard[lane] = card;
  }
  if (lane == 0) pstart[g] = total;
  if (lane < g && V.type == TY_UINT)
    for (uint32_t u = 0; u < cl; u++) list[off + u] = static_cast<const uint32_t*>(V.p)[u];
  __syncwarp();
  for (uint32_t rest = __ballot_sync(FULL, lane < g && V.type != TY_UINT); rest; rest &= rest - 1) {
    const uint32_t p = __ffs(rest) - 1;
    const uint32_t i = a.order[base + p];
    RowView W = load_view(a.desc, a.arena, i);
    if (MODE == kSym) keep_below(a, W, i);
    uint32_t* to = list + poff[p];
    warp_decode_to<LONG>(W, lane, [&](uint32_t k, uint32_t x) {
      if (k < W.card) to[k] = x;
    });
    __syncwarp();
  }
  unsigned long long tcnt = 0;
  for (uint32_t q = lane; q < total; q += 32) {
    uint32_t p = 0;
    while (pstart[p + 1] <= q) p++;
    uint32_t e = 1, t = q - pstart[p];
    while (t >= e) { t -= e; e++; }
    const uint32_t j = list[poff[p] + e], x = list[poff[p] + t];
    bool hit;
    if (j < a.core_k) hit = (__ldg(a.core + core_offset32(j) + (x >> 6)) >> (x & 63)) & 1ull;
    else hit = row_contains(load_view(a.desc, a.arena, j), x);
    if (hit && MODE == kSym) tcnt += (unsigned long long)pcard[p] + a.desc[j].card + a.desc[x].card;
    else if (hit) tcnt += MODE == kFull ? pcard[p] : 1u;
  }
  __syncwarp();  // the tables are reused by the next chunk
  return tcnt;
}

// Pivots up to light_max entries, one warp each: order[mid0, mid1) in grabs of
// mid_chunk, then the tiny ones order[mid1, n_order) in chunks of tiny_chunk.
template <int MODE, bool LONG>
__global__ void __launch_bounds__(kCtaThreads, MODE == kSym ? 3 : 4) k_pivots_warp(PivotArgs a, uint32_t mid1, uint32_t mid_chunk,
                                                                uint32_t tiny, uint32_t cap, uint32_t win) {
  extern __shared__ __align__(16) char dyn[];
  overlap_begin();
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  char* mem = dyn + warp * slice_bytes<1, MODE>(cap, win);
  const Slice s = make_slice<1, MODE>(mem, cap, win);
  for (uint32_t k = lane; k < (win + kHashBits) / 32; k += 32) s.bm[k] = 0u;
  __syncwarp();
  unsigned long long acc = 0;
  WordSum sum;
  sum.clear();
  for (;;) {
    uint32_t base = 0;
    if (lane == 0) base = a.n_heavy + atomicAdd(&a.queue[1], mid_chunk);
    base = __shfl_sync(FULL, base, 0);
    if (base >= mid1) break;
    const uint32_t end = min(mid1, base + mid_chunk);
    for (uint32_t k = base; k < end; k++) {
      const uint32_t i = a.order[k];
      RowView A = load_view(a.desc, a.arena, i);
      const uint32_t card = A.card;
      if (MODE == kSym) keep_below(a, A, i);
      const uint32_t cnt = pivot_count<1, MODE, LONG>(a, A, 1, A.card, s, win, nullptr, lane, 0, sum, card, acc);
      acc += finish_pivot<MODE>(a, i, card, cnt, sum, lane);
    }
  }
  __syncwarp();
  const uint32_t tiny0 = max(mid1, a.n_heavy);
  for (;;) {
    uint32_t base = 0;
    if (lane == 0) base = tiny0 + atomicAdd(&a.queue[3], tiny);
    base = __shfl_sync(FULL, base, 0);
    if (base >= a.n_order) break;
    acc += tiny_chunk<MODE, LONG>(a, base, min(tiny, a.n_order - base), reinterpret_cast<uint32_t*>(mem), lane);
  }
  cta_add(acc + sum.total(), a);
  overlap_end();
}

// Dense core build: one warp per row j < core_k writes row(j) ∩ [0, j) as bits.
__global__ void __launch_bounds__(256) k_core_build(const RowDesc* __restrict__ desc, const uint4* __restrict__ arena,
                                                    uint32_t core_k, unsigned long long* __restrict__ core) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t nw = gridDim.x * (blockDim.x / 32);
  for (uint32_t j = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); j < core_k; j += nw) {
    unsigned long long* row = core + core_row_offset(j);
    const uint32_t wj = (j + 63) >> 6;
    for (uint32_t w = lane; w < wj; w += 32) row[w] = 0ull;
    __syncwarp();
    const RowView B = load_view(desc, arena, j);
    if (B.type == TY_BITSET) {
      const unsigned long long* bw = static_cast<const unsigned long long*>(B.p);
      for (uint32_t w = lane; w < B.len; w += 32) {
        const uint32_t gw = B.aux + w;
        if (gw >= wj) break;
        unsigned long long x = bw[w];
        if (gw == wj - 1 && (j & 63)) x &= (1ull << (j & 63)) - 1ull;
        row[gw] = x;
      }
    } else {
      warp_for_each(B, j, lane, [&](uint32_t x) { atomicOr(&row[x >> 6], 1ull << (x & 63)); });
    }
    __syncwarp();
  }
}

// Heavy units: for order position u < n_heavy, ceil((card-1)/span) units (u, part).
__global__ void k_unit_counts(const RowDesc* __restrict__ desc, const uint32_t* __restrict__ order,
                              uint32_t n_heavy, uint32_t span, uint32_t* __restrict__ cnt) {
  const uint32_t u = blockIdx.x * blockDim.x + threadIdx.x;
  if (u < n_heavy) {
    const uint32_t c = desc[order[u]].card;
    cnt[u] = (c - 1 + span - 1) / span;
  }
}
__global__ void k_unit_fill(const uint32_t* __restrict__ cnt, const uint32_t* __restrict__ start,
                            uint32_t n_heavy, uint2* __restrict__ units) {
  const uint32_t u = blockIdx.x * blockDim.x + threadIdx.x;
  if (u < n_heavy)
    for (uint32_t p = 0; p < cnt[u]; p++) units[start[u] + p] = make_uint2(u, p);
}

// bits = row(v) as a bitmap over all n ids (zeroed before).
__global__ void __launch_bounds__(256) k_row_bits(const RowDesc* __restrict__ desc, const uint4* __restrict__ arena,
                                                  uint32_t v, unsigned long long* __restrict__ bits) {
  const RowView V = load_view(desc, arena, v);
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  if (V.type == TY_UINT) {
    const uint32_t* e = static_cast<const uint32_t*>(V.p);
    for (uint32_t k = tid; k < V.card; k += nt) atomicOr(bits + (e[k] >> 6), 1ull << (e[k] & 63));
  } else if (V.type == TY_BITSET) {
    const unsigned long long* w = static_cast<const unsigned long long*>(V.p);
    for (uint32_t k = tid; k < V.len; k += nt) bits[V.aux + k] = w[k];
  } else {  // warps take partitions round-robin
    const uint16_t* e = static_cast<const uint16_t*>(V.p);
    for (uint32_t i = 0, p = 0; i < V.len; p++) {
      const uint32_t hb = (uint32_t)e[i] << 16, cnt = (uint32_t)e[i + 1] + 1;
      if (p % (nt / 32) == tid / 32)
        for (uint32_t k = tid & 31; k < cnt; k += 32) {
          const uint32_t x = hb | e[i + 2 + k];
          atomicOr(bits + (x >> 6), 1ull << (x & 63));
        }
      i += cnt + 2;
    }
  }
}

// similar_nodes: rows i with |row(v*) ∩ row(i)| > threshold, row(v*) as a bitmap
// of n bits (262 KB at 2^21 rows).  Every entry is one bitmap word, where a
// warp per row ran a merge path or binary searches against the whole of row(v*).
// A warp takes 32 descriptors at once; rows of at most `threshold` entries
// cannot qualify and are not read; uint rows up to kSimilarShort entries take 8
// lanes and 16-byte loads each, the others the whole warp, which stops once the
// threshold is passed.  Bound by the scattered bitmap words (L1, L2).  R-MAT scale 21, uint,
// threshold 10: 1.60 ms before.
constexpr uint32_t kSimilarShort = 256;
__global__ void __launch_bounds__(256) k_similar(uint32_t n, const RowDesc* __restrict__ desc,
                                                 const uint4* __restrict__ arena, uint32_t vstar,
                                                 const unsigned long long* __restrict__ bits, uint32_t threshold,
                                                 unsigned long long* out) {
  const uint32_t lane = threadIdx.x & 31, sl = lane & 7, grp = lane >> 3;
  const uint32_t* bits32 = reinterpret_cast<const uint32_t*>(bits);
  const auto in = [&](uint32_t y) -> uint32_t {  // kUintPad >= n
    return y < n ? (__ldg(bits32 + (y >> 5)) >> (y & 31)) & 1u : 0u;
  };
  const auto in4 = [&](uint4 v) { return in(v.x) + in(v.y) + in(v.z) + in(v.w); };
  unsigned long long acc = 0;
  const uint64_t nw = (uint64_t)gridDim.x * (blockDim.x / 32);
  // Pairs of rows (one sector of descriptors) are dealt round-robin, so that
  // the hubs at the front of a degree-ordered graph spread over the grid.
  const uint64_t w = (uint64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  for (uint64_t base = 2 * w; base < n; base += nw * 32) {
    const uint64_t r = base + (lane & 1) + (lane >> 1) * 2 * nw;
    const uint4 d = r < n ? __ldg(reinterpret_cast<const uint4*>(desc) + r) : make_uint4(0u, 0u, 0u, 0u);
    const bool candidate = d.y > threshold, brief = candidate && (d.w >> 30) == TY_UINT && d.y <= kSimilarShort;
    for (uint32_t m = __ballot_sync(FULL, brief); m;) {
      uint32_t own = m;  // group g takes the g-th row left
      for (uint32_t u = 0; u < 4; u++) {
        if (u < grp) own &= own - 1;
        m &= m - 1;
      }
      const uint32_t src = own ? __ffs(own) - 1 : 0u;
      const uint32_t off = __shfl_sync(FULL, d.x, src), card = __shfl_sync(FULL, d.y, src);
      const uint32_t n4 = own ? (card + 3) >> 2 : 0u;
      uint32_t c = 0;
      for (uint32_t q = sl; q < n4; q += 16) {
        const uint4 v0 = __ldg(arena + off + q);
        const uint4 v1 = q + 8 < n4 ? __ldg(arena + off + q + 8) : make_uint4(kUintPad, kUintPad, kUintPad, kUintPad);
        c += in4(v0) + in4(v1);
      }
      c += __shfl_xor_sync(FULL, c, 1);
      c += __shfl_xor_sync(FULL, c, 2);
      c += __shfl_xor_sync(FULL, c, 4);
      if (sl == 0 && c > threshold) acc++;
    }
    // A short pshort row is one lane's: its partition headers are a serial chain.
    const bool serial = candidate && (d.w >> 30) == TY_PSHORT && d.y <= kSimilarShort;
    if (serial) {
      const uint16_t* e = reinterpret_cast<const uint16_t*>(arena + d.x);
      const uint32_t len = d.w & 0x3fffffffu;
      uint32_t c = 0;
      for (uint32_t i = 0; i < len && c <= threshold;) {
        const uint32_t hb = (uint32_t)e[i] << 16, cnt = (uint32_t)e[i + 1] + 1;
        for (uint32_t k = 0; k < cnt; k++) c += in(hb | e[i + 2 + k]);
        i += cnt + 2;
      }
      acc += c > threshold;
    }
    __syncwarp();
    for (uint32_t m = __ballot_sync(FULL, candidate && !brief && !serial); m; m &= m - 1) {
      const uint32_t src = __ffs(m) - 1;
      RowView B;
      B.p = arena + __shfl_sync(FULL, d.x, src);
      B.card = __shfl_sync(FULL, d.y, src);
      B.aux = __shfl_sync(FULL, d.z, src);
      const uint32_t ty_len = __shfl_sync(FULL, d.w, src);
      B.type = ty_len >> 30;
      B.len = ty_len & 0x3fffffffu;
      // What the reference's pshort u16 counts would drop is not counted.
      uint64_t need = threshold;
      if (B.type == TY_PSHORT && B.card >= 65536u) need += pshort_pair_drop(load_view(desc, arena, vstar), B, ~0ull);
      uint32_t c = 0;  // uniform over the warp
      if (B.type == TY_UINT) {
        const uint4* p4 = static_cast<const uint4*>(B.p);
        const uint32_t n4 = (B.card + 3) >> 2;
        for (uint32_t q0 = 0; q0 < n4 && c <= need; q0 += 64) {
          const uint4 pad = make_uint4(kUintPad, kUintPad, kUintPad, kUintPad);
          const uint4 v0 = q0 + lane < n4 ? __ldg(p4 + q0 + lane) : pad;
          const uint4 v1 = q0 + lane + 32 < n4 ? __ldg(p4 + q0 + lane + 32) : pad;
          c += __reduce_add_sync(FULL, in4(v0) + in4(v1));
        }
      } else if (B.type == TY_BITSET) {
        const uint4* p4 = static_cast<const uint4*>(B.p);  // word pairs, zero-padded; bits has a spare word
        const uint32_t np = (B.len + 1) >> 1;
        for (uint32_t q0 = 0; q0 < np && c <= need; q0 += 64) {
          uint32_t h = 0;
#pragma unroll
          for (uint32_t u = 0; u < 64; u += 32) {
            const uint32_t q = q0 + u + lane;
            if (q < np) {
              const uint4 v = __ldg(p4 + q);
              h += __popcll(lo64(v) & __ldg(bits + B.aux + 2 * q)) + __popcll(hi64(v) & __ldg(bits + B.aux + 2 * q + 1));
            }
          }
          c += __reduce_add_sync(FULL, h);
        }
      } else {
        const uint16_t* e = static_cast<const uint16_t*>(B.p);
        for (uint32_t i = 0; i < B.len && c <= need;) {
          const uint32_t hb = (uint32_t)e[i] << 16, cnt = (uint32_t)e[i + 1] + 1;
          uint32_t h = 0;
          for (uint32_t k = lane; k < cnt; k += 32) h += in(hb | e[i + 2 + k]);
          c += __reduce_add_sync(FULL, h);
          i += cnt + 2;
        }
      }
      if (lane == 0 && c > need) acc++;
    }
  }
  acc = warp_sum_u64(acc);
  if (lane == 0 && acc) atomicAdd(out, acc);
}

// counts[p] = |row(a[p]) ∩ row(b[p])|, one warp per pair.  A pair naming a
// row >= n gets 0xffffffff.
__global__ void __launch_bounds__(256) k_intersect_rows(uint64_t n, const RowDesc* __restrict__ desc,
                                                        const uint4* __restrict__ arena,
                                                        const uint32_t* __restrict__ ra,
                                                        const uint32_t* __restrict__ rb, uint64_t np,
                                                        uint32_t* __restrict__ counts) {
  __shared__ PshortHdr s_hdr[8];
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t nw = (uint64_t)gridDim.x * (blockDim.x / 32);
  for (uint64_t p = (uint64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); p < np; p += nw) {
    if (ra[p] >= n || rb[p] >= n) {
      if (lane == 0) counts[p] = 0xffffffffu;
      continue;
    }
    const uint32_t c = warp_intersect_size(load_view(desc, arena, ra[p]), load_view(desc, arena, rb[p]), lane,
                                           &s_hdr[threadIdx.x >> 5]);
    if (lane == 0) counts[p] = c;
  }
}

}  // namespace

// Resident CTAs per SM that a shape may ask for (eh_matrix_set_shape).
constexpr int kMaxCtasPerSm = 8;

static int sm_count(int device) {
  static std::atomic<int> cache[64];
  if (device < 0 || device >= 64) return 152;
  int g = cache[device].load();
  if (g > 0) return g;
  cudaDeviceGetAttribute(&g, cudaDevAttrMultiProcessorCount, device);
  g = std::max(1, g);
  cache[device].store(g);
  return g;
}

int pivot_grid(int device) { return sm_count(device) * kMaxCtasPerSm; }

// Resident CTAs of a kernel with `bytes` of dynamic shared memory and at most
// `regs` CTAs per SM by registers (a larger grid would only queue).
static int resident_grid(int device, uint32_t bytes, int regs) {
  constexpr uint32_t kSmemPerSm = 228u << 10;
  return sm_count(device) * std::max(1, std::min<int>(regs, (int)(kSmemPerSm / (bytes + 2048))));
}

// Window bits of the tiers' membership bitmaps: the id range up to the tier's most.
static uint32_t window_bits(uint64_t n, uint32_t most) {
  uint32_t w = 4096;
  while (w < most && w < n) w *= 2;
  return w;
}

// Dynamic shared memory above 48 KB has to be allowed once per kernel and device.
static cudaError_t allow_smem(const void* kernel, uint32_t bytes, std::atomic<bool>* done, int device) {
  if (device < 0 || device >= 64) return cudaErrorInvalidDevice;
  if (done[device].load()) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) done[device].store(true);
  return e;
}

// Kernels that ask for different splits of L1 and shared memory do not run on an SM
// at the same time, and a short call is mostly the tails of its tiers: below
// kSplitRows rows, if there are several, all ask for the whole of it.  R-MAT, 14 edges a vertex, uint: 60 K
// vertices 46.9 -> 43.4 us, 130 K 80.5 -> 79.3 (hybrid 90.3 -> 86.7), 260 K even (the line
// lies halfway); above that L1 counts for more (520 K 247 -> 270, 1 M 544 -> 623).
constexpr uint64_t kSplitRows = 196608;

static uint32_t cap_of(uint32_t entries) { return std::max(32u, (entries + 31) & ~31u); }

// One launch of k_pivots_cta: n units, or order[pos0, pos0 + n) whole.
template <int NW, int MODE, bool LONG>
struct CtaLaunch {
  uint32_t n = 0, pos0 = 0, cap = 0, win = 0, bytes = 0;
  unsigned grid = 0;
  CtaLaunch(const PivotArgs& a, uint32_t n_, uint32_t pos0_, uint32_t largest, uint32_t window, int most, int device)
      : n(n_), pos0(pos0_) {
    if (!n) return;
    cap = cap_of(largest);
    win = window_bits(a.n, window);
    bytes = slice_bytes<NW, MODE>(cap, win);
    const int regs = (MODE == kSym ? 24 : 32) / NW;
    const int per = std::max(1, std::min(regs, most / sm_count(device) * (NWARPS / NW)));
    grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(n, resident_grid(device, bytes, per)));
  }
  cudaError_t run(const PivotArgs& a, const uint2* units, uint32_t* next, int device, cudaStream_t st,
                  unsigned split, bool& overlap) const {
    if (!n) return cudaSuccess;
    static std::atomic<bool> done[64];
    cudaError_t e = allow_smem((const void*)k_pivots_cta<NW, MODE, LONG>, slice_bytes<NW, MODE>(kCtaListCap, kCtaWindow),
                               done, device);
    if (e != cudaSuccess) return e;
    e = launch_overlapped(k_pivots_cta<NW, MODE, LONG>, grid, NW * 32, bytes, st, overlap, split, a, units, n, pos0, next,
                          cap, win);
    overlap = true;
    return e;
  }
};

template <int MODE, bool LONG>
static cudaError_t launch_pivots_as(PivotArgs a, const uint2* units, uint32_t n_units, int most, cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  int device = 0;
  if ((e = cudaGetDevice(&device)) != cudaSuccess) return e;
  if (a.graph_rows && (e = cudaMemsetAsync(a.out, 0, sizeof(unsigned long long) * a.num_graphs, st)) != cudaSuccess)
    return e;
  // Largest pivots first; the kernels overlap, their CTAs counted for the last one to finish.
  const bool giants = MODE != kSym && n_units && a.n_giant;
  const unsigned g_heavy =
      giants ? (unsigned)std::max(1, std::min(most, resident_grid(device, (uint32_t)sizeof(HeavySmem), 6))) : 0u;
  const uint32_t n_large = !units ? a.n_large : a.n_large > a.n_giant ? n_units : 0u;  // no list: whole pivots
  const CtaLaunch<kLargeWarps, MODE, LONG> large(a, n_large, 0, a.max_large, kCtaWindow, most, device);
  const CtaLaunch<kMidWarps, MODE, LONG> mid(a, a.n_heavy > a.n_large ? a.n_heavy - a.n_large : 0u, a.n_large, a.max_mid,
                                       kWarpWindow, most, device);
  const uint32_t cap = cap_of(a.max_warp), win = window_bits(a.n, kWarpWindow);
  const uint32_t bytes = NWARPS * slice_bytes<1, MODE>(cap, win);
  uint32_t mid1 = 0, mid_chunk = 1, tiny_grab = 1;
  int gw = 0;
  if (a.n_order > a.n_heavy) {
    mid1 = std::min(a.n_order, std::max(a.n_heavy, a.n_above_tiny));
    const uint32_t warp_pivots = mid1 - a.n_heavy, tiny = a.n_order - mid1;
    gw = std::max(1, std::min(most, resident_grid(device, bytes, MODE == kSym ? 3 : 4)));
    // Grabs small enough that every warp gets several; one pivot at least.
    const uint32_t warps = (uint32_t)gw * NWARPS;
    mid_chunk = std::max(1u, std::min(4u, warp_pivots / (16 * warps)));
    tiny_grab = std::max(1u, std::min(kTinyChunk, tiny / (4 * warps)));
    const uint64_t grabs = (uint64_t)warp_pivots / mid_chunk + tiny / tiny_grab + 1;
    gw = (int)std::min<uint64_t>(gw, (grabs + NWARPS - 1) / NWARPS);
  }
  a.ctas = g_heavy + large.grid + mid.grid + (unsigned)gw;
  if (a.ctas == 0)  // no row with a pair
    return a.graph_rows ? cudaSuccess : cudaMemsetAsync(a.out, 0, (a.report ? 2 : 1) * sizeof(unsigned long long), st);
  const unsigned split = a.n < kSplitRows && g_heavy + large.grid + mid.grid ? 100u : 0u;
  bool overlap = false;
  if (g_heavy) {
    e = launch_overlapped(k_pivots_heavy<MODE == kFull>, g_heavy, kCtaThreads, 0, st, false, split, a, units, n_units);
    overlap = true;
  }
  if (e == cudaSuccess) e = large.run(a, units, a.queue + 2, device, st, split, overlap);
  if (e == cudaSuccess) e = mid.run(a, nullptr, a.queue + 4, device, st, split, overlap);
  if (e == cudaSuccess && gw) {
    static std::atomic<bool> done[64];
    e = allow_smem((const void*)k_pivots_warp<MODE, LONG>, NWARPS * slice_bytes<1, MODE>(kLightMax, kWarpWindow), done,
                   device);
    if (e == cudaSuccess)
      e = launch_overlapped(k_pivots_warp<MODE, LONG>, (unsigned)gw, kCtaThreads, bytes, st, overlap, split, a, mid1,
                            mid_chunk, tiny_grab, cap, win);
  }
  // A launch that failed leaves the others short of the last CTA: clear the queue for the next call.
  if (e != cudaSuccess) cudaMemsetAsync(a.queue, 0, kPivotQueueWords * sizeof(uint32_t), st);
  return e;
}

// The kernels for matrices of bitset or pshort rows throughout (PivotArgs::long_rows) have
// the loops those rows want: long bitset rows four rounds in flight, pshort
// rows streamed.  Of their own, as they cost the others up to 2% (R-MAT scale 22,
// hybrid 5.37 against 5.49 ms); for them 23.8 against 18.2 ms (bitset) and 8.06 against 7.05
// (pshort).
template <int MODE>
static cudaError_t launch_pivots(const PivotArgs& a, const uint2* units, uint32_t n_units, int most, cudaStream_t st) {
  return a.long_rows ? launch_pivots_as<MODE, true>(a, units, n_units, most, st)
                     : launch_pivots_as<MODE, false>(a, units, n_units, most, st);
}

cudaError_t launch_pivot_units(const RowDesc* desc, const uint32_t* order, uint32_t n_heavy,
                               uint32_t unit_span, uint32_t* cnt, cudaStream_t st) {
  if (n_heavy == 0) return cudaSuccess;
  k_unit_counts<<<(n_heavy + 255) / 256, 256, 0, st>>>(desc, order, n_heavy, unit_span, cnt);
  return cudaGetLastError();
}
cudaError_t launch_pivot_unit_fill(const uint32_t* cnt, const uint32_t* start, uint32_t n_heavy,
                                   uint2* units, cudaStream_t st) {
  if (n_heavy == 0) return cudaSuccess;
  k_unit_fill<<<(n_heavy + 255) / 256, 256, 0, st>>>(cnt, start, n_heavy, units);
  return cudaGetLastError();
}

cudaError_t launch_triangles(PivotArgs a, const uint2* units, uint32_t n_units, int grid,
                             cudaStream_t st) {
  return launch_pivots<kTri>(a, units, n_units, grid, st);
}
cudaError_t launch_lollipops(PivotArgs a, const uint2* units, uint32_t n_units, int grid,
                             cudaStream_t st) {
  return a.lcard ? launch_pivots<kSym>(a, units, n_units, grid, st) : launch_pivots<kFull>(a, units, n_units, grid, st);
}

cudaError_t launch_core_build(const RowDesc* desc, const uint4* arena, uint32_t core_k, unsigned long long* core,
                              cudaStream_t st) {
  if (core_k == 0) return cudaSuccess;
  const uint32_t blocks = std::min<uint32_t>((core_k + 7) / 8, 152u * 16u);
  k_core_build<<<blocks, 256, 0, st>>>(desc, arena, core_k, core);
  return cudaGetLastError();
}

cudaError_t launch_row_bits(uint64_t n, const RowDesc* desc, const uint4* arena, uint32_t v, unsigned long long* bits,
                            cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(bits, 0, row_bits_words(n) * sizeof(unsigned long long), st);
  if (e != cudaSuccess || n == 0) return e;
  k_row_bits<<<152, 256, 0, st>>>(desc, arena, v, bits);
  return cudaGetLastError();
}

cudaError_t launch_similar(uint64_t n, const RowDesc* desc, const uint4* arena, uint32_t vstar,
                           const unsigned long long* bits, uint32_t threshold, unsigned long long* out,
                           cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(out, 0, sizeof(unsigned long long), st);
  if (e != cudaSuccess || n == 0) return e;
  const uint64_t g = std::min<uint64_t>((n + 255) / 256, 152 * 8);
  k_similar<<<(unsigned)g, 256, 0, st>>>((uint32_t)n, desc, arena, vstar, bits, threshold, out);
  return cudaGetLastError();
}

cudaError_t launch_intersect_rows(uint64_t n, const RowDesc* desc, const uint4* arena, const uint32_t* a,
                                  const uint32_t* b, uint64_t np, uint32_t* counts, cudaStream_t st) {
  if (np == 0) return cudaSuccess;
  uint64_t g = (np + 7) / 8;
  if (g > 152 * 32) g = 152 * 32;
  k_intersect_rows<<<(unsigned)g, 256, 0, st>>>(n, desc, arena, a, b, np, counts);
  return cudaGetLastError();
}

}  // namespace eh
