// The pairwise matcher's match list from its seeds, without replaying the
// reference's hash table seed by seed (included by match.cu).
//
// The reference (AddHashEntry, LM/MemHash.cpp:209-251) takes the unique seeds
// in mer order; a seed that lower_bound finds contained in an entry of its
// bucket is dropped, another one is extended (ExtendMatch) and inserted at
// its sorted place.  Replaying that is one chain per bucket, with an extension
// and an insert per match: 10.9 of 13.5 ms on a 12 Mbp pair of 221,000
// matches.  What the chain computes can be said without it:
//
//  * ExtendMatch walks along the seed's diagonal over matching windows at
//    most L apart, so its result is the connected component of the seed's
//    window: the same for every seed of the component.
//  * Seeds of one diagonal at most L apart are connected.  A segment is a
//    maximal chain of them; segments of one diagonal that follow each other
//    in their bucket may be connected through matching windows that are no
//    unique seeds, which a walk from one towards the other tells.
//  * Where the components of a bucket, in order of their starts in A, end
//    (with their last seed) before the next one starts, the entries before a
//    seed x's component start before x and are less, those after it start
//    behind x and are not less, and its own entry contains it: the comparator
//    is monotone for every x and every subset of the entries, lower_bound
//    finds x's entry iff it is there, and the bucket ends up with its
//    components in order of their starts, whatever the order of the seeds.
//  * Elsewhere (flagged buckets) only the seeds behind the start of a later
//    component can be missed by the bisection.  For each of these, in mer
//    order, the bisection is run as std::lower_bound runs it over the entries
//    there at its time (those whose component has a seed of smaller mer, and
//    copies inserted before).  A missed seed inserts a copy of its
//    component's entry right at the entry.
//
// So: a table of B positions by A position, segment ends by looking L
// positions to either side, one sort of the ends by bucket (not of the
// seeds), two walks per segment on eight lanes each, and a compaction.  The
// walks bound it: about 1,000 instructions for a group of eight lanes.
#pragma once
#include "match_common.cuh"

namespace mvg {

constexpr uint32_t kNoSeed = 0xffffffffu;  // no pair has B position 2^31 - 1
constexpr int kSegTile = 2048;

// A pair in the table: B position, bit 31 set for opposite strands.  Its
// diagonal: bit 32 the strand relation, low word y - x or y + x.
__device__ __forceinline__ uint64_t seed_diag(uint32_t v, uint32_t x) {
  const uint32_t y = v & 0x7fffffffu;
  return v >> 31 ? (1ull << 32) | (uint32_t)(y + x) : (uint64_t)(uint32_t)(y - x);
}

// The pair on diagonal d at A position x, as the table holds it.
__device__ __forceinline__ uint32_t diag_seed(uint64_t d, uint32_t x) {
  return d >> 32 ? 0x80000000u | ((uint32_t)d - x) : (uint32_t)d + x;
}

// CalculateOffset (LM/MatchHashEntry.cpp:141-162) of a diagonal.
__device__ __forceinline__ int64_t diag_offset(uint64_t d, int L) {
  return d >> 32 ? -(int64_t)(uint32_t)d - 2 - L : (int64_t)(int32_t)(uint32_t)d;
}
__device__ __forceinline__ uint32_t diag_bucket(uint64_t d, int L) {
  const int64_t t = kTableSize, off = diag_offset(d, L);
  return (uint32_t)(((off % t) + t) % t);
}

// The hash entry of windows [lo, hi] (A starts) on diagonal d.
__device__ __forceinline__ Mhe diag_entry(uint64_t d, uint32_t lo, uint32_t hi, int L) {
  Mhe m;
  m.s0 = (int64_t)lo + 1;
  m.len = (int64_t)(hi - lo) + L;
  m.s1 = d >> 32 ? -((int64_t)((uint32_t)d - hi) + 1) : (int64_t)((uint32_t)d + lo) + 1;
  m.off = diag_offset(d, L);
  return m;
}

// ------------------------------------------------------------ pair table

// From the joint sort (the bucketed join of pair_buckets.cu writes the table
// itself): runs of exactly one key per genome.
template <typename K>
__global__ void k_tab_runs(const K* __restrict__ keys, const uint32_t* __restrict__ pos, int64_t n,
                           uint32_t* __restrict__ tab) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || !pair_flag(keys, n, i)) return;
  const uint32_t k0 = (uint32_t)keys[i], k1 = (uint32_t)keys[i + 1];
  const uint32_t p0 = pos[i], p1 = pos[i + 1];
  const uint32_t rev = ((k0 ^ k1) >> 1) & 1u;
  tab[k0 & 1u ? p1 : p0] = (k0 & 1u ? p0 : p1) | rev << 31;
}

// -------------------------------------------------------------- segments

// Segment heads (no pair of the diagonal in the L positions before) and
// tails as bit masks over A's positions; per tile their counts (heads of all
// tiles, then tails), and the number of pairs.
__global__ void __launch_bounds__(256) k_seg_bits(const uint32_t* __restrict__ tab, int64_t n, int L,
                                                  uint32_t* __restrict__ headw, uint32_t* __restrict__ tailw,
                                                  uint32_t* __restrict__ tcount, int64_t ntiles,
                                                  uint32_t* __restrict__ npairs) {
  __shared__ uint32_t s[kSegTile + 64];
  __shared__ uint32_t sum[3];
  const int64_t base = (int64_t)blockIdx.x * kSegTile;
  if (threadIdx.x < 3) sum[threadIdx.x] = 0;
  for (int i = threadIdx.x; i < kSegTile + 64; i += 256) {
    const int64_t x = base - 32 + i;
    s[i] = x >= 0 && x < n ? tab[x] : kNoSeed;
  }
  __syncthreads();
  uint32_t nh = 0, nt = 0, nv = 0;
#pragma unroll 2
  for (int q = 0; q < kSegTile / 256; ++q) {
    const int i = 32 + q * 256 + (int)threadIdx.x;
    const uint32_t v = s[i];
    bool head = v != kNoSeed, tail = head;
    if (head) {
      // along the diagonal B moves with A or against it; a value that wraps
      // is no pair's, but can be the empty table's (B position -1)
      const uint32_t back = v >> 31 ? 1u : 0xffffffffu;
      for (int t = 1; t <= L && head; ++t) {
        const uint32_t want = v + back * (uint32_t)t;
        head = s[i - t] != want || want == kNoSeed;
      }
      for (int t = 1; t <= L && tail; ++t) tail = s[i + t] != v - back * (uint32_t)t;
    }
    const uint32_t hb = __ballot_sync(0xffffffffu, head), tb = __ballot_sync(0xffffffffu, tail);
    nv += __popc(__ballot_sync(0xffffffffu, v != kNoSeed));
    nh += __popc(hb);
    nt += __popc(tb);
    if ((threadIdx.x & 31) == 0) {
      const int64_t w = (base + q * 256 + threadIdx.x) >> 5;
      headw[w] = hb;
      tailw[w] = tb;
    }
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&sum[0], nh);
    atomicAdd(&sum[1], nt);
    atomicAdd(&sum[2], nv);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    tcount[blockIdx.x] = sum[0];
    tcount[ntiles + blockIdx.x] = sum[1];
    if (sum[2]) atomicAdd(npairs, sum[2]);
  }
}

// The ends in order of their A positions, heads then tails: key = bucket
// (tails behind all heads), value = position.  toff: the scanned counts.
__global__ void __launch_bounds__(128) k_seg_emit(const uint32_t* __restrict__ tab, int L,
                                                  const uint32_t* __restrict__ headw, const uint32_t* __restrict__ tailw,
                                                  const uint32_t* __restrict__ toff, int64_t ntiles,
                                                  uint32_t* __restrict__ key, uint32_t* __restrict__ val) {
  constexpr int kWords = kSegTile / 32;
  static_assert(kWords == 64, "two warps of head words, two of tail words");
  __shared__ uint32_t wsum[4];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const bool tails = wid >= 2;
  const int64_t w = (int64_t)blockIdx.x * kWords + (tid & (kWords - 1));
  uint32_t bits = (tails ? tailw : headw)[w];
  const uint32_t incl = warp_incl_scan(__popc(bits));
  if (lane == 31) wsum[wid] = incl;
  __syncthreads();
  uint32_t at = toff[(tails ? ntiles : 0) + blockIdx.x] + incl - __popc(bits) + (wid & 1 ? wsum[wid - 1] : 0u);
  while (bits) {
    const uint32_t x = (uint32_t)(w * 32) + (uint32_t)(__ffs(bits) - 1);
    bits &= bits - 1;
    key[at] = diag_bucket(seed_diag(tab[x], x), L) + (tails ? kTableSize : 0);
    val[at++] = x;
  }
}

// Sorted by bucket, a bucket's heads and tails have the same indices.  The
// tail of head k is the first one at or behind it on its diagonal: index k
// unless segments of the bucket interleave.
__global__ void k_seg_pair(const uint32_t* __restrict__ tab, const uint32_t* __restrict__ head,
                           const uint32_t* __restrict__ tkey, const uint32_t* __restrict__ tail, int64_t n,
                           uint32_t* __restrict__ last) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const uint32_t x = head[k], b = tkey[k];
  const uint64_t d = seed_diag(tab[x], x);
  int64_t j = k;
  while (j > 0 && tkey[j - 1] == b && tail[j - 1] >= x) --j;
  while (j < n - 1 && !(tail[j] >= x && seed_diag(tab[tail[j]], tail[j]) == d)) ++j;
  last[k] = tail[j];
}

// ----------------------------------------------------------------- walks

// One side of ExtendMatch from a segment end on eight lanes: tasks [0, n)
// from the tails to higher A positions, [n, 2n) from the heads down.  A walk
// towards a neighbouring segment of the same bucket and diagonal stops when
// it gets there.  Out: moved[task], and for the first n joined[k] (segment k
// is connected to segment k + 1).
__global__ void __launch_bounds__(256) k_seg_walk(MatchCtx c, const uint32_t* __restrict__ tab,
                                                  const uint32_t* __restrict__ key, const uint32_t* __restrict__ head,
                                                  const uint32_t* __restrict__ last, int64_t n,
                                                  uint32_t* __restrict__ moved, uint8_t* __restrict__ joined) {
  const int64_t task = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  if (task >= 2 * n) return;
  const int lane = threadIdx.x & 31, j = lane & 7, L = c.s.L;
  const unsigned group = 0xffu << (lane & 24);
  const bool up = task < n;
  const int64_t k = up ? task : task - n;
  const uint32_t x = up ? last[k] : head[k];
  const uint32_t v = tab[x];
  const uint64_t d = seed_diag(v, x);
  int64_t limit = INT64_MAX;  // distance to the neighbour
  if (up && k + 1 < n && key[k + 1] == key[k] && seed_diag(tab[head[k + 1]], head[k + 1]) == d)
    limit = (int64_t)head[k + 1] - x;
  if (!up && k > 0 && key[k - 1] == key[k] && seed_diag(tab[last[k - 1]], last[k - 1]) == d)
    limit = (int64_t)x - last[k - 1];
  const int64_t e1 = (int64_t)(v & 0x7fffffffu) + 1;
  const int64_t s0 = up ? -((int64_t)x + 1) : (int64_t)x + 1;
  const int64_t s1 = (v >> 31 != 0) != up ? -e1 : e1;
  const uint64_t pmask = pattern_mask64(c.s);
  uint32_t carry = 0;
  for (int64_t it = 0;; ++it) {
    const uint32_t w = ext_word(c, s0, s1, L, (it * 8 + j) * 32, pmask);
    uint32_t prev = __shfl_up_sync(group, w, 1, 8);
    if (j == 0) prev = carry;
    const int64_t idx = it * 8 + j - 1;  // the word whose successor is w
    const uint32_t hit = idx >= 0 ? stop_in_word(prev, w, idx == 0, L) : 0u;
    const unsigned any = __ballot_sync(group, hit != 0);
    if (any) {
      const int f = __ffs(any) - 1;
      if (lane == f) {
        const int64_t q = 32 * idx + (__ffs(hit) - 1);
        moved[task] = (uint32_t)(q < limit ? q : 0);
        if (up) joined[k] = q >= limit;
      }
      return;
    }
    if (32 * (it * 8 + 7) >= limit) {
      if (j == 0) {
        moved[task] = 0;
        if (up) joined[k] = 1;
      }
      return;
    }
    carry = __shfl_sync(group, w, 7, 8);
  }
}

// ------------------------------------------------------------ components

struct Components {
  uint32_t* lo;      // first window (A start)
  uint32_t* hi;      // last window
  uint32_t* seed;    // last seed
  uint32_t* bucket;
  uint64_t* diag;
  uint32_t* copies;  // entries the bucket holds of it
  uint64_t* time;    // flagged buckets: the component's smallest mer
};

__global__ void __launch_bounds__(256) k_comp_count(const uint8_t* __restrict__ joined, int64_t n,
                                                    uint32_t* __restrict__ tcount) {
  const int64_t i0 = (int64_t)blockIdx.x * kSegTile + (int64_t)threadIdx.x * 8;
  uint32_t cnt = 0, total;
  for (int q = 0; q < 8; ++q) {
    const int64_t k = i0 + q;
    cnt += k < n && !(k > 0 && joined[k - 1]);
  }
  block_excl_scan256(cnt, nullptr);
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  __shared__ uint32_t ws[8];
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = cnt;
  __syncthreads();
  if (threadIdx.x == 0) {
    total = 0;
    for (int w = 0; w < 8; ++w) total += ws[w];
    tcount[blockIdx.x] = total;
  }
}

// Components from segments: the first one's head and downward walk, the last
// one's tail and upward walk.
__global__ void __launch_bounds__(256) k_comp_emit(const uint32_t* __restrict__ tab, const uint32_t* __restrict__ key,
                                                   const uint32_t* __restrict__ head, const uint32_t* __restrict__ last,
                                                   const uint32_t* __restrict__ moved, const uint8_t* __restrict__ joined,
                                                   int64_t n, const uint32_t* __restrict__ toff, Components C) {
  const int64_t i0 = (int64_t)blockIdx.x * kSegTile + (int64_t)threadIdx.x * 8;
  uint32_t flags = 0;
  for (int q = 0; q < 8; ++q) {
    const int64_t k = i0 + q;
    flags |= (uint32_t)(k < n && !(k > 0 && joined[k - 1])) << q;
  }
  uint32_t id = toff[blockIdx.x] + block_excl_scan256(__popc(flags), nullptr);  // components before this thread's
  for (int q = 0; q < 8; ++q) {
    const int64_t k = i0 + q;
    if (k >= n) break;
    if (flags >> q & 1u) {
      const uint32_t x = head[k];
      C.lo[id] = x - moved[n + k];
      C.diag[id] = seed_diag(tab[x], x);
      C.bucket[id] = key[k];
      C.copies[id] = 1;
      ++id;
    }
    if (!joined[k]) {
      C.hi[id - 1] = last[k] + moved[k];
      C.seed[id - 1] = last[k];
    }
  }
}

__device__ __forceinline__ void comp_row(const Components& C, uint32_t e, int L, int64_t* __restrict__ out, uint64_t at,
                                         uint64_t cap) {
  if (at >= cap) return;
  const Mhe m = diag_entry(C.diag[e], C.lo[e], C.hi[e], L);
  out[3 * at + 0] = m.s0;
  out[3 * at + 1] = m.s1;
  out[3 * at + 2] = m.len;
}

// The match list when no bucket is flagged (GetMatchList order: buckets, then
// their entries, LM/MemHash.h:182-203), and the list of flagged buckets.
__global__ void k_comp_out(Components C, const uint32_t* __restrict__ ncomp, int L, int64_t* __restrict__ out,
                           uint64_t cap, uint32_t* __restrict__ bflag, uint32_t* __restrict__ flagged,
                           uint32_t* __restrict__ nflagged) {
  const uint32_t n = *ncomp;
  for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    comp_row(C, e, L, out, e, cap);
    if (e + 1 < n && C.bucket[e] == C.bucket[e + 1] && C.lo[e + 1] <= C.seed[e] &&
        atomicExch(&bflag[C.bucket[e]], 1u) == 0u)
      flagged[atomicAdd(nflagged, 1u)] = C.bucket[e];
  }
}

// --------------------------------------------------------- flagged buckets

__device__ __forceinline__ void comp_range(const Components& C, uint32_t n, uint32_t b, uint32_t& first, uint32_t& end) {
  uint32_t at[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    uint32_t lo = 0, len = n;
    while (len > 0) {
      const uint32_t half = len >> 1;
      if (C.bucket[lo + half] < b + q) {
        lo += half + 1;
        len -= half + 1;
      } else {
        len = half;
      }
    }
    at[q] = lo;
  }
  first = at[0];
  end = at[1];
}

// One CTA per flagged bucket: its components in entry order (they nearly are:
// exchanges of neighbours until nothing moves), a component found from
// several of its segments kept once.
__global__ void __launch_bounds__(256) k_flag_sort(Components C, uint32_t n, int L, const uint32_t* __restrict__ flagged) {
  __shared__ uint32_t range[2];
  if (threadIdx.x == 0) comp_range(C, n, flagged[blockIdx.x], range[0], range[1]);
  __syncthreads();
  const uint32_t first = range[0], end = range[1];
  for (bool again = true; again;) {
    bool moved = false;
    for (uint32_t parity = 0; parity < 2; ++parity) {
      for (uint32_t e = first + parity + 2 * threadIdx.x; e + 1 < end; e += 512) {
        const Mhe a = diag_entry(C.diag[e], C.lo[e], C.hi[e], L), b = diag_entry(C.diag[e + 1], C.lo[e + 1], C.hi[e + 1], L);
        if (!mhe_strict_lt(b, a, L)) continue;
        moved = true;
        const uint32_t lo = C.lo[e], hi = C.hi[e], seed = C.seed[e];
        const uint64_t diag = C.diag[e];
        C.lo[e] = C.lo[e + 1];
        C.hi[e] = C.hi[e + 1];
        C.seed[e] = C.seed[e + 1];
        C.diag[e] = C.diag[e + 1];
        C.lo[e + 1] = lo;
        C.hi[e + 1] = hi;
        C.seed[e + 1] = seed;
        C.diag[e + 1] = diag;
      }
      __syncthreads();
    }
    again = __syncthreads_or(moved);
  }
  // the last of a component's copies stays, with the last seed of all
  for (uint32_t e = first + threadIdx.x; e < end; e += 256) {
    C.time[e] = ~0ull;
    const bool more = e + 1 < end && C.diag[e] == C.diag[e + 1] && C.lo[e] == C.lo[e + 1];
    if (more) {
      C.copies[e] = 0;
      continue;
    }
    uint32_t seed = C.seed[e];
    for (uint32_t f = e; f > first && C.diag[f - 1] == C.diag[e] && C.lo[f - 1] == C.lo[e]; --f) seed = max(seed, C.seed[f - 1]);
    C.seed[e] = seed;
  }
}

// Mer of A's window at x as the reference orders seeds.
__device__ __forceinline__ uint64_t seed_time(const MatchCtx& c, uint32_t x) {
  return (canonical_mer(c.g[0], x, c.s) & c.s.seed_mask) >> (64 - 2 * c.s.w);
}

// Work on the seeds of flagged buckets' components in pieces of kFlagPiece
// positions: (component, first position).
constexpr uint32_t kFlagPiece = 1024;
struct FlagWork {
  uint32_t* count;  // [0] pieces of whole components, [1] pieces of their seeds behind the next component's start
  uint2* whole;     // null: count only
  uint2* behind;
};

__global__ void k_flag_plan(Components C, uint32_t n, const uint32_t* __restrict__ bflag, FlagWork W) {
  for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    if (!bflag[C.bucket[e]] || !C.copies[e]) continue;
    uint32_t f = e + 1;
    while (f < n && C.bucket[f] == C.bucket[e] && !C.copies[f]) ++f;
    const bool over = f < n && C.bucket[f] == C.bucket[e] && C.lo[f] <= C.seed[e];
    for (int list = 0; list < (over ? 2 : 1); ++list) {
      const uint32_t x0 = list ? max(C.lo[f], C.lo[e]) : C.lo[e];
      const uint32_t pieces = (C.seed[e] - x0) / kFlagPiece + 1;
      const uint32_t at = atomicAdd(&W.count[list], pieces);
      uint2* out = list ? W.behind : W.whole;
      for (uint32_t q = 0; out && q < pieces; ++q) out[at + q] = make_uint2(e, x0 + q * kFlagPiece);
    }
  }
}

// Every component's smallest mer (a warp per piece).
__global__ void k_flag_time(MatchCtx c, const uint32_t* __restrict__ tab, Components C, const uint2* __restrict__ work,
                            uint32_t pieces) {
  const int lane = threadIdx.x & 31;
  const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= pieces) return;
  const uint32_t e = work[w].x, x0 = work[w].y, x1 = min(C.seed[e], x0 + kFlagPiece - 1);
  const uint64_t d = C.diag[e];
  unsigned long long t = ~0ull;
  for (uint32_t x = x0 + lane; x <= x1; x += 32)
    if (tab[x] == diag_seed(d, x)) t = min(t, (unsigned long long)seed_time(c, x));
  for (int s = 16; s > 0; s >>= 1) t = min(t, __shfl_xor_sync(0xffffffffu, t, s));
  if (lane == 0 && t != ~0ull) atomicMin((unsigned long long*)&C.time[e], t);
}

// The seeds behind the start of a component after their own: mer, position
// and component, in any order (a warp per piece).
struct FlagSeeds {
  uint64_t* time;
  uint32_t *x, *e;
  uint32_t* id;     // 0, 1, ...
  uint32_t* count;
};
__global__ void k_flag_collect(MatchCtx c, const uint32_t* __restrict__ tab, Components C, const uint2* __restrict__ work,
                               uint32_t pieces, FlagSeeds S) {
  const int lane = threadIdx.x & 31;
  const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= pieces) return;
  const uint32_t e = work[w].x, x0 = work[w].y, x1 = min(C.seed[e], x0 + kFlagPiece - 1);
  const uint64_t d = C.diag[e], t0 = C.time[e];
  for (uint32_t xb = x0; xb <= x1; xb += 32) {
    const uint32_t x = xb + lane;
    bool in = x <= x1 && tab[x] == diag_seed(d, x);
    uint64_t t = 0;
    if (in) {
      t = seed_time(c, x);
      in = t != t0;  // the component's first seed finds no entry
    }
    const unsigned all = __ballot_sync(0xffffffffu, in);
    uint32_t base = 0;
    if (lane == 0 && all) base = atomicAdd(S.count, (uint32_t)__popc(all));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (in) {
      const uint32_t at = base + __popc(all & ((1u << lane) - 1u));
      S.time[at] = t;
      S.x[at] = x;
      S.e[at] = e;
      S.id[at] = at;
    }
  }
}

// The seeds' flagged-bucket numbers, in the order of ids (sorted by mer).
__global__ void k_flag_bucket(Components C, const uint32_t* __restrict__ e, const uint32_t* __restrict__ id, uint32_t n,
                              const uint32_t* __restrict__ bnumber, uint32_t* __restrict__ number) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) number[i] = bnumber[C.bucket[e[id[i]]]];
}

// The flagged buckets' numbers in the list.
__global__ void k_flag_numbers(const uint32_t* __restrict__ flagged, uint32_t n, uint32_t* __restrict__ bnumber) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) bnumber[flagged[i]] = i;
}

// One CTA per flagged bucket tests its seeds in mer order, 1024 at a time
// against the entries as they are; the first missed one inserts a copy of its
// component's entry and the tests go on behind it.  For a seed of component e
// the entries there at its time are, in order: p that are less, the c copies
// of e, which contain it, b that start between e's start and the seed's and
// are less, and the rest, which are not.  So lower_bound's bisection needs
// only p, c, b and the number of all.
__global__ void __launch_bounds__(1024) k_flag_test(Components C, uint32_t n, int L, const uint32_t* __restrict__ flagged,
                                                    const uint32_t* __restrict__ number, const uint32_t* __restrict__ id,
                                                    uint32_t nseeds, FlagSeeds S) {
  __shared__ uint32_t range[4];
  __shared__ uint32_t wmin[32];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (tid == 0) comp_range(C, n, flagged[blockIdx.x], range[0], range[1]);
  if (tid < 2) {
    uint32_t lo = 0, len = nseeds;
    while (len > 0) {
      const uint32_t half = len >> 1;
      if (number[lo + half] < blockIdx.x + tid) {
        lo += half + 1;
        len -= half + 1;
      } else {
        len = half;
      }
    }
    range[2 + tid] = lo;
  }
  __syncthreads();
  const uint32_t first = range[0], end = range[1], send = range[3];
  for (uint32_t pos = range[2]; pos < send;) {
    bool missed = false;
    if (pos + tid < send) {
      const uint32_t s = id[pos + tid], x = S.x[s], e = S.e[s];
      const uint64_t t = S.time[s];
      const Mhe seed = diag_entry(C.diag[e], x, x, L);
      uint32_t b = 0;
      for (uint32_t i = e + 1; i < end && C.lo[i] <= x; ++i)
        if (C.time[i] < t && mhe_strict_lt(diag_entry(C.diag[i], C.lo[i], C.hi[i], L), seed, L)) b += C.copies[i];
      if (b) {
        uint32_t p = 0, all = 0;
        for (uint32_t i = first; i < end; ++i) {
          const uint32_t v = C.time[i] < t ? C.copies[i] : 0u;
          all += v;
          p += i < e ? v : 0u;
        }
        const uint32_t c = C.copies[e];
        uint32_t f = 0, len = all;
        while (len > 0) {
          const uint32_t half = len >> 1, mid = f + half;
          if (mid < p || (mid >= p + c && mid < p + c + b)) {
            f = mid + 1;
            len -= half + 1;
          } else {
            len = half;
          }
        }
        missed = f < p || f >= p + c;
      }
    }
    uint32_t at = __reduce_min_sync(0xffffffffu, missed ? (uint32_t)tid : 1024u);
    if (lane == 0) wmin[wid] = at;
    __syncthreads();
    at = __reduce_min_sync(0xffffffffu, wmin[lane]);
    if (tid == 0 && at < 1024u) C.copies[S.e[id[pos + at]]] += 1;
    pos += at < 1024u ? at + 1 : 1024u;
    __syncthreads();
  }
}

// The match list with copies: at = exclusive sums of copies.
__global__ void k_comp_out_copies(Components C, uint32_t n, const uint32_t* __restrict__ at, int L,
                                  int64_t* __restrict__ out, uint64_t cap) {
  for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x)
    for (uint32_t q = 0; q < C.copies[e]; ++q) comp_row(C, e, L, out, (uint64_t)at[e] + q, cap);
}

}  // namespace mvg
