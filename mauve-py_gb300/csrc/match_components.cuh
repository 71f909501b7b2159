// The pairwise matcher's match list from its seeds, without replaying the
// reference's hash table seed by seed (included by match.cu and
// gapsearch.cu).
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
//    behind x and are not less, and its own entry contains it (MheCompare,
//    LM/MatchHashEntry.h:121-143, over Contains, LM/MatchHashEntry.cpp:164-200,
//    where neither is less): the comparator
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
// seeds), two walks per segment, and a compaction.
#pragma once
#include <algorithm>

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
  return m;
}

// What the kernels below ask of a matching problem P, by A position x (and
// the table's value v there):
//   seed_len(x)   the seed's length
//   key(v, x)     sort key: the hash bucket (below the gap's number)
//   view(x, a, b) packed sequences, lengths and seed, and the positions at
//                 which they start among A's and B's
//   row(...)      writes the entry of windows [lo, hi] on diagonal d as row at
//   mer_bits()    width of the widest mer (host)
// One genome pair: positions are the genomes'.
struct OnePair {
  MatchCtx c;
  int64_t* out;
  uint64_t cap;
  int mer_bits() const { return 2 * c.s.w; }
  __device__ __forceinline__ int seed_len(uint32_t) const { return c.s.L; }
  __device__ __forceinline__ uint32_t key(uint32_t v, uint32_t x) const { return diag_bucket(seed_diag(v, x), c.s.L); }
  __device__ __forceinline__ MatchView view(uint32_t, uint32_t& a, uint32_t& b) const {
    a = b = 0;
    return MatchView{{c.g[0], c.g[1]}, {c.n[0], c.n[1]}, c.s};
  }
  __device__ __forceinline__ void row(uint64_t d, uint32_t lo, uint32_t hi, uint64_t at) const {
    if (at >= cap) return;
    const Mhe m = diag_entry(d, lo, hi, c.s.L);
    out[3 * at + 0] = m.s0;
    out[3 * at + 1] = m.s1;
    out[3 * at + 2] = m.len;
  }
};

// The pair table from a joint sort of both genomes' keys (the bucketed join of
// pair_buckets.cu writes it itself): runs of exactly one key per genome.
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
// tiles, then tails), and the number of pairs; what the join left (left) beside
// them.  Most pairs have their
// diagonal's neighbour right beside them; the others' searches go through a
// list, so that a warp's lanes all have one to do.  (Searched where they lie,
// one lane in a warp kept it for L steps: bits, counts and lists of the ends of
// 5,003 gaps, 23 million positions of A, took 0.31 ms, now 0.235.)
template <class P>
__global__ void __launch_bounds__(256) k_seg_bits(P prob, const uint32_t* __restrict__ tab, int64_t n,
                                                  uint32_t* __restrict__ headw, uint32_t* __restrict__ tailw,
                                                  uint32_t* __restrict__ tcount, int64_t ntiles,
                                                  uint32_t* __restrict__ npairs, const uint32_t* __restrict__ left,
                                                  uint32_t* __restrict__ left_out) {
  __shared__ uint32_t s[kSegTile + 64];
  __shared__ uint16_t list[2 * kSegTile];  // entries of s to search from, 2 i + 1 for a tail
  __shared__ uint32_t bits[2][kSegTile / 32];
  __shared__ uint32_t sum[3], listed;
  const int64_t base = (int64_t)blockIdx.x * kSegTile;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 3) sum[threadIdx.x] = 0;
  if (threadIdx.x == 0) listed = 0;
  if (threadIdx.x < 2 * (kSegTile / 32)) bits[threadIdx.x & 1][threadIdx.x >> 1] = 0;
  for (int i = threadIdx.x; i < kSegTile + 64; i += 256) {
    const int64_t x = base - 32 + i;
    s[i] = x >= 0 && x < n ? tab[x] : kNoSeed;
  }
  __syncthreads();
  // along the diagonal B moves with A or against it; a value that wraps is no
  // pair's, but can be the empty table's (B position -1)
  auto same = [&](int at, uint32_t want) { return s[at] == want && want != kNoSeed; };
  uint32_t nv = 0;
#pragma unroll 2
  for (int q = 0; q < kSegTile / 256; ++q) {
    const int i = 32 + q * 256 + (int)threadIdx.x;
    const uint32_t v = s[i], back = v >> 31 ? 1u : 0xffffffffu;
    const bool in = v != kNoSeed, head = in && !same(i - 1, v + back), tail = in && !same(i + 1, v - back);
    nv += __popc(__ballot_sync(0xffffffffu, in));
    const uint32_t hb = __ballot_sync(0xffffffffu, head), tb = __ballot_sync(0xffffffffu, tail);
    const uint32_t nh = __popc(hb), nl = nh + __popc(tb), lt = (1u << lane) - 1u;
    uint32_t at = 0;
    if (lane == 0 && nl) at = atomicAdd(&listed, nl);
    at = __shfl_sync(0xffffffffu, at, 0);
    if (head) list[at + __popc(hb & lt)] = (uint16_t)(2 * i);
    if (tail) list[at + nh + __popc(tb & lt)] = (uint16_t)(2 * i + 1);
  }
  if (lane == 0) atomicAdd(&sum[2], nv);
  __syncthreads();
  for (uint32_t k = threadIdx.x; k < listed; k += 256) {
    const int i = list[k] >> 1, tail = list[k] & 1, step = tail ? 1 : -1;
    const uint32_t v = s[i], move = (v >> 31 ? 1u : 0xffffffffu) * (tail ? 0xffffffffu : 1u);
    const int L = prob.seed_len((uint32_t)(base + i - 32));
    int t = 2;
    uint32_t want = v + 2 * move;
    while (t <= L && !same(i + t * step, want)) {
      ++t;
      want += move;
    }
    if (t > L) atomicOr(&bits[tail][(i - 32) >> 5], 1u << (i & 31));
  }
  __syncthreads();
  if (threadIdx.x < 2 * (kSegTile / 32)) {
    const int tail = threadIdx.x / (kSegTile / 32), w = threadIdx.x % (kSegTile / 32);
    const uint32_t b = bits[tail][w];
    (tail ? tailw : headw)[(base >> 5) + w] = b;
    const uint32_t c = __reduce_add_sync(0xffffffffu, __popc(b));
    if (lane == 0) atomicAdd(&sum[tail], c);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    tcount[blockIdx.x] = sum[0];
    tcount[ntiles + blockIdx.x] = sum[1];
    if (sum[2]) atomicAdd(npairs, sum[2]);
    if (left && blockIdx.x == 0) *left_out = *left;
  }
}

// The ends in order of their A positions, heads then tails: key = bucket
// (tails behind all heads), value = position.  toff: the scanned counts.
template <class P>
__global__ void __launch_bounds__(128) k_seg_emit(P prob, const uint32_t* __restrict__ tab,
                                                  const uint32_t* __restrict__ headw, const uint32_t* __restrict__ tailw,
                                                  const uint32_t* __restrict__ toff, int64_t ntiles,
                                                  int tail_bit, uint32_t* __restrict__ key,
                                                  uint32_t* __restrict__ val) {
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
    key[at] = prob.key(tab[x], x) | (tails ? 1u << tail_bit : 0u);
    val[at++] = x;
  }
}

// Sorted by bucket, a bucket's heads and tails have the same indices.  The
// tail of head k is the first one at or behind it on its diagonal: index k
// unless segments of the bucket interleave.
static __global__ void k_seg_pair(const uint32_t* __restrict__ tab, const uint32_t* __restrict__ head,
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

// One side of ExtendMatch from a segment end: tasks [0, n) from the tails to
// higher A positions, [n, 2n) from the heads down.  A walk towards a
// neighbouring segment of the same bucket and diagonal stops when it gets
// there.
template <class P>
struct SegTask {
  const bool up;
  const int64_t k;
  const uint32_t x;  // the seed it starts from
  uint32_t a0, b0;   // where its sequences begin
  const MatchView c;
  int64_t limit;     // distance to the neighbour
  int64_t s0, s1;

  __device__ __forceinline__ SegTask(const P& prob, const uint32_t* tab, const uint32_t* key, const uint32_t* head,
                                     const uint32_t* last, int64_t n, int64_t task)
      : up(task < n), k(up ? task : task - n), x(up ? last[k] : head[k]), c(prob.view(x, a0, b0)) {
    const uint32_t v = tab[x];
    const uint64_t d = seed_diag(v, x);
    limit = INT64_MAX;
    if (up && k + 1 < n && key[k + 1] == key[k] && seed_diag(tab[head[k + 1]], head[k + 1]) == d)
      limit = (int64_t)head[k + 1] - x;
    if (!up && k > 0 && key[k - 1] == key[k] && seed_diag(tab[last[k - 1]], last[k - 1]) == d)
      limit = (int64_t)x - last[k - 1];
    const int64_t e0 = (int64_t)(x - a0) + 1, e1 = (int64_t)((v & 0x7fffffffu) - b0) + 1;
    s0 = up ? -e0 : e0;
    s1 = (v >> 31 != 0) != up ? -e1 : e1;
  }

  // Words of 32 displacements from word `start` on, LANES (this lane is the
  // j-th of `group`) at a time, `rounds` times: the displacement of the stop,
  // the limit or beyond when it gets there, -1 when neither is reached.
  // Word start - 1 and those before have been looked at.
  template <int LANES>
  __device__ __forceinline__ int64_t walk(int64_t start, int64_t rounds, unsigned group, int j) const {
    const int L = c.s.L;
    uint32_t carry = 0;
    for (int64_t it = 0; it < rounds; ++it) {
      const int64_t at = start + it * LANES;
      const uint32_t w = ext_word(c, s0, s1, L, (at + j) * 32);
      uint32_t prev = __shfl_up_sync(group, w, 1, LANES);
      if (j == 0) prev = carry;
      const int64_t idx = at + j - 1;  // the word whose successor is w
      const uint32_t hit = idx >= start ? stop_in_word(prev, w, idx == 0, L) : 0u;
      const unsigned any = __ballot_sync(group, hit != 0);
      if (any) {
        const int f = __ffs(any) - 1;  // a lane of this group
        return __shfl_sync(group, 32 * idx + (__ffs(hit) - 1), f % LANES, LANES);
      }
      if (32 * (at + LANES - 1) >= limit) return limit;
      carry = __shfl_sync(group, w, LANES - 1, LANES);
    }
    return -1;
  }

  // moved: what the walk covered; joined[k]: segment k is connected to k + 1.
  __device__ __forceinline__ void done(int64_t q, int64_t task, uint32_t* moved, uint8_t* joined) const {
    moved[task] = (uint32_t)(q < limit ? q : 0);
    if (up) joined[k] = q >= limit;
  }
};

// Two lanes per task look at the first words, as far as most walks go; the
// warp's other tasks go on in fours, eight lanes each, and what is left then
// one by one with the whole warp.  The instructions of making and searching
// words bound short walks, latency the few long ones: eight lanes per task
// throughout took 1.06 ms for the walks of 5,003 gaps and 0.045 ms for the 4.6
// Mbp recoded pair's, this 0.42 and 0.037 (two lanes throughout: 0.44 and
// 0.125).
template <class P>
__global__ void __launch_bounds__(256) k_seg_walk(P prob, const uint32_t* __restrict__ tab,
                                                  const uint32_t* __restrict__ key, const uint32_t* __restrict__ head,
                                                  const uint32_t* __restrict__ last, int64_t n,
                                                  uint32_t* __restrict__ moved, uint8_t* __restrict__ joined) {
  constexpr int kEight = 1;  // rounds of eight lanes
  constexpr int kFrom8 = 2 - 1, kFrom32 = kFrom8 + 8 * kEight - 1;  // a walk's last word has no successor yet
  const int lane = threadIdx.x & 31;
  const int64_t first = ((int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31)) / 2;  // the warp's first task
  const int64_t task = first + lane / 2;
  bool open = false;
  if (task < 2 * n) {
    const SegTask<P> t(prob, tab, key, head, last, n, task);
    const int64_t q = t.template walk<2>(0, 1, 3u << (lane & 30), lane & 1);
    open = q < 0;
    if (!open && (lane & 1) == 0) t.done(q, task, moved, joined);
  }
  const unsigned left = __ballot_sync(0xffffffffu, open) & 0x55555555u;
  const int more = __popc(left);
  unsigned rest = 0;
  for (int r = lane >> 3; r < more; r += 4) {
    const int at = (int)__fns(left, 0, r + 1);
    const SegTask<P> t(prob, tab, key, head, last, n, first + at / 2);
    const int64_t q = t.template walk<8>(kFrom8, kEight, 0xffu << (lane & 24), lane & 7);
    if (q < 0) rest |= 1u << at;
    else if ((lane & 7) == 0) t.done(q, first + at / 2, moved, joined);
  }
  for (rest = __reduce_or_sync(0xffffffffu, rest); rest; rest &= rest - 1) {
    const int64_t mine = first + (__ffs(rest) - 1) / 2;
    const SegTask<P> t(prob, tab, key, head, last, n, mine);
    const int64_t q = t.template walk<32>(kFrom32, INT64_MAX, 0xffffffffu, lane);
    if (lane == 0) t.done(q, mine, moved, joined);
  }
}

// ------------------------------------------------------------ components

struct Components {
  uint32_t* lo;      // first window (A start)
  uint32_t* hi;      // last window
  uint32_t* seed;    // last seed
  uint32_t* key;     // its bucket's sort key
  uint64_t* diag;
  uint32_t* copies;  // entries the bucket holds of it
  uint64_t* time;    // flagged buckets: the component's smallest mer
};

static __global__ void __launch_bounds__(256) k_comp_count(const uint8_t* __restrict__ joined, int64_t n,
                                                    uint32_t* __restrict__ tcount) {
  const int64_t i0 = (int64_t)blockIdx.x * kSegTile + (int64_t)threadIdx.x * 8;
  uint32_t cnt = 0;
  for (int q = 0; q < 8; ++q) {
    const int64_t k = i0 + q;
    cnt += k < n && !(k > 0 && joined[k - 1]);
  }
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  __shared__ uint32_t ws[8];
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = cnt;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t total = 0;
    for (int w = 0; w < 8; ++w) total += ws[w];
    tcount[blockIdx.x] = total;
  }
}

// Components from segments: the first one's head and downward walk, the last
// one's tail and upward walk.
static __global__ void __launch_bounds__(256) k_comp_emit(const uint32_t* __restrict__ tab, const uint32_t* __restrict__ key,
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
      C.key[id] = key[k];
      C.copies[id] = 1;
      ++id;
    }
    if (!joined[k]) {
      C.hi[id - 1] = last[k] + moved[k];
      C.seed[id - 1] = last[k];
    }
  }
}

// The match list when no bucket is flagged (GetMatchList order: buckets, then
// their entries, LM/MemHash.h:182-203), and the list of flagged buckets.
template <class P>
__global__ void k_comp_out(P prob, Components C, const uint32_t* __restrict__ ncomp, uint32_t* __restrict__ bflag,
                           uint32_t* __restrict__ flagged, uint32_t* __restrict__ nflagged) {
  const uint32_t n = *ncomp;
  for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    prob.row(C.diag[e], C.lo[e], C.hi[e], e);
    if (e + 1 < n && C.key[e] == C.key[e + 1] && C.lo[e + 1] <= C.seed[e]) {
      // the bucket's flag is the word of its first component
      uint32_t lo = 0, len = e;
      while (len > 0) {
        const uint32_t half = len >> 1;
        if (C.key[lo + half] < C.key[e]) {
          lo += half + 1;
          len -= half + 1;
        } else {
          len = half;
        }
      }
      if (atomicExch(&bflag[lo], 1u) == 0u) flagged[atomicAdd(nflagged, 1u)] = C.key[e];
    }
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
      if (C.key[lo + half] < b + q) {
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
template <class P>
__global__ void __launch_bounds__(256) k_flag_sort(P prob, Components C, uint32_t n, const uint32_t* __restrict__ flagged) {
  __shared__ uint32_t range[2];
  if (threadIdx.x == 0) comp_range(C, n, flagged[blockIdx.x], range[0], range[1]);
  __syncthreads();
  const uint32_t first = range[0], end = range[1];
  const int L = prob.seed_len(C.lo[first]);
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
template <class P>
__device__ __forceinline__ uint64_t seed_time(const P& prob, uint32_t x) {
  uint32_t a0, b0;
  const MatchView c = prob.view(x, a0, b0);
  return (canonical_mer(c.g[0], x - a0, c.s) & c.s.seed_mask) >> (64 - 2 * c.s.w);
}

// Work on the seeds of flagged buckets' components in pieces of kFlagPiece
// positions: component, first position, the bucket's number in the list.
constexpr uint32_t kFlagPiece = 1024;
struct FlagWork {
  uint32_t* count;  // [0] pieces of whole components, [1] pieces of their seeds behind the next component's start
  uint4* whole;     // null: count only
  uint4* behind;
};

// One CTA per flagged bucket.
static __global__ void __launch_bounds__(256) k_flag_plan(Components C, uint32_t n, const uint32_t* __restrict__ flagged,
                                                   FlagWork W) {
  __shared__ uint32_t range[2];
  if (threadIdx.x == 0) comp_range(C, n, flagged[blockIdx.x], range[0], range[1]);
  __syncthreads();
  for (uint32_t e = range[0] + threadIdx.x; e < range[1]; e += 256) {
    if (!C.copies[e]) continue;
    uint32_t f = e + 1;
    while (f < range[1] && !C.copies[f]) ++f;
    const bool over = f < range[1] && C.lo[f] <= C.seed[e];
    for (int list = 0; list < (over ? 2 : 1); ++list) {
      const uint32_t x0 = list ? max(C.lo[f], C.lo[e]) : C.lo[e];
      const uint32_t pieces = (C.seed[e] - x0) / kFlagPiece + 1;
      const uint32_t at = atomicAdd(&W.count[list], pieces);
      uint4* out = list ? W.behind : W.whole;
      for (uint32_t q = 0; out && q < pieces; ++q) out[at + q] = make_uint4(e, x0 + q * kFlagPiece, blockIdx.x, 0u);
    }
  }
}

// Every component's smallest mer (a warp per piece).
template <class P>
__global__ void k_flag_time(P prob, const uint32_t* __restrict__ tab, Components C, const uint4* __restrict__ work,
                            uint32_t pieces) {
  const int lane = threadIdx.x & 31;
  const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= pieces) return;
  const uint32_t e = work[w].x, x0 = work[w].y, x1 = min(C.seed[e], x0 + kFlagPiece - 1);
  const uint64_t d = C.diag[e];
  unsigned long long t = ~0ull;
  for (uint32_t x = x0 + lane; x <= x1; x += 32)
    if (tab[x] == diag_seed(d, x)) t = min(t, (unsigned long long)seed_time(prob, x));
  for (int s = 16; s > 0; s >>= 1) t = min(t, __shfl_xor_sync(0xffffffffu, t, s));
  if (lane == 0 && t != ~0ull) atomicMin((unsigned long long*)&C.time[e], t);
}

// The seeds behind the start of a component after their own: mer, position,
// component and bucket, in any order (a warp per piece).
struct FlagSeeds {
  uint64_t* time;
  uint32_t *x, *e, *number;
  uint32_t* id;     // 0, 1, ...
  uint32_t* count;
};
template <class P>
__global__ void k_flag_collect(P prob, const uint32_t* __restrict__ tab, Components C, const uint4* __restrict__ work,
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
      t = seed_time(prob, x);
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
      S.number[at] = work[w].z;
      S.id[at] = at;
    }
  }
}

// The seeds' bucket numbers in the order of ids (sorted by mer).
static __global__ void k_flag_number(FlagSeeds S, const uint32_t* __restrict__ id, uint32_t n, uint32_t* __restrict__ number) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) number[i] = S.number[id[i]];
}

// One CTA per flagged bucket tests its seeds in mer order, 1024 at a time
// against the entries as they are; the first missed one inserts a copy of its
// component's entry and the tests go on behind it.  For a seed of component e
// the entries there at its time are, in order: p that are less, the c copies
// of e, which contain it, b that start between e's start and the seed's and
// are less, and the rest, which are not.  So lower_bound's bisection needs
// only p, c, b and the number of all.
template <class P>
__global__ void __launch_bounds__(1024) k_flag_test(P prob, Components C, uint32_t n, const uint32_t* __restrict__ flagged,
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
  const int L = prob.seed_len(C.lo[first]);
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
template <class P>
__global__ void k_comp_out_copies(P prob, Components C, uint32_t n, const uint32_t* __restrict__ at) {
  for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x)
    for (uint32_t q = 0; q < C.copies[e]; ++q) prob.row(C.diag[e], C.lo[e], C.hi[e], (uint64_t)at[e] + q);
}

// ------------------------------------------------------------------ host

// Exclusive scan of n counts and their sum: one launch where it fits.
static void scan_counts(const uint32_t* in, int64_t n, uint32_t* out, uint32_t* scratch, uint32_t* total,
                        cudaStream_t st, uint64_t* launches) {
  if (n <= 16384) {
    pair_scan_small(in, (int)n, out, total, st);
    *launches += 1;
  } else {
    exclusive_scan(in, out, n, scratch, total, st, launches);
  }
}

struct ComponentResult {
  Components C;
  uint32_t ncomp = 0;
  uint64_t pairs = 0, rows = 0;
  const uint32_t* at = nullptr;  // rows before each component (null: its index)
};

// The buckets k_comp_out flagged, exactly, and the rows again.
template <class P, class F>
int flagged_components(Ctx* c, P& prob, const uint32_t* tab, const uint32_t* flagged, uint32_t nflagged, F room_for,
                       ComponentResult* out) {
  const Components& C = out->C;
  const uint32_t ncomp = out->ncomp;
  Workspace& ws = c->ws;
  // work and seed counts, sums, all components' first rows, scan scratch
  uint32_t* w = (uint32_t*)ws.get(c, 37, ((size_t)ncomp + scan_scratch_words(ncomp) + 16) * 4);
  if (!w) return report_error(MVG_ERR_NOMEM, "workspace allocation failed");
  uint32_t *count = w, *cat = w + 16, *scratch = cat + ncomp;
  MVG_CUDA_TRY(cudaMemsetAsync(count, 0, 64, c->stream));
  k_flag_sort<<<nflagged, 256, 0, c->stream>>>(prob, C, ncomp, flagged);
  FlagWork W{count, nullptr, nullptr};
  k_flag_plan<<<nflagged, 256, 0, c->stream>>>(C, ncomp, flagged, W);
  c->launches += 2;
  MVG_CUDA_TRY(cudaMemcpyAsync(c->h_scalars, count, 8, cudaMemcpyDeviceToHost, c->stream));
  MVG_CUDA_TRY(cudaStreamSynchronize(c->stream));
  const uint32_t whole = ((const uint32_t*)c->h_scalars)[0], behind = ((const uint32_t*)c->h_scalars)[1];
  // the pieces, and room for every position of the seeds' pieces
  const size_t room = (size_t)behind * kFlagPiece;
  W.whole = (uint4*)ws.get(c, 39, ((size_t)whole + behind) * 16 + 16);
  uint64_t* t0 = (uint64_t*)ws.get(c, 40, room * 8 + 16);
  uint64_t* t1 = (uint64_t*)ws.get(c, 41, room * 8 + 16);
  uint32_t* u = (uint32_t*)ws.get(c, 42, room * 4 * 5 + 16);
  uint32_t* sscr = (uint32_t*)ws.get(c, 43, sort_scratch_words((int64_t)room, 64) * 4);
  if (!W.whole || !t0 || !t1 || !u || !sscr) return report_error(MVG_ERR_NOMEM, "workspace allocation failed");
  W.behind = W.whole + whole;
  W.count = count + 2;
  FlagSeeds S{t0, u, u + room, u + 2 * room, u + 3 * room, count + 4};
  k_flag_plan<<<nflagged, 256, 0, c->stream>>>(C, ncomp, flagged, W);
  k_flag_time<<<div_up((int64_t)whole * 32, 256), 256, 0, c->stream>>>(prob, tab, C, W.whole, whole);
  c->launches += 2;
  if (behind) {
    k_flag_collect<<<div_up((int64_t)behind * 32, 256), 256, 0, c->stream>>>(prob, tab, C, W.behind, behind, S);
    c->launches++;
  }
  MVG_CUDA_TRY(cudaMemcpyAsync(c->h_scalars, count + 4, 4, cudaMemcpyDeviceToHost, c->stream));
  MVG_CUDA_TRY(cudaStreamSynchronize(c->stream));
  const uint32_t nseeds = ((const uint32_t*)c->h_scalars)[0];
  if (nseeds) {
    // by mer, then stably by bucket; the mers stay where they are for the tests
    uint64_t* keys = (uint64_t*)ws.get(c, 48, (size_t)nseeds * 8);
    if (!keys) return report_error(MVG_ERR_NOMEM, "workspace allocation failed");
    MVG_CUDA_TRY(cudaMemcpyAsync(keys, t0, (size_t)nseeds * 8, cudaMemcpyDeviceToDevice, c->stream));
    uint32_t *id = S.id, *id_alt = u + 4 * room;
    if (sort_pairs<uint64_t>(keys, id, t1, id_alt, nseeds, prob.mer_bits(), sscr, c->stream, &c->launches, c->d_err))
      std::swap(id, id_alt);
    uint32_t *number = (uint32_t*)keys, *number_alt = (uint32_t*)t1;
    k_flag_number<<<div_up(nseeds, 256), 256, 0, c->stream>>>(S, id, nseeds, number);
    int bits = 1;
    while ((1u << bits) < nflagged) ++bits;
    if (sort_pairs<uint32_t>(number, id, number_alt, id_alt, nseeds, bits, sscr, c->stream, &c->launches, c->d_err)) {
      std::swap(number, number_alt);
      std::swap(id, id_alt);
    }
    k_flag_test<<<nflagged, 1024, 0, c->stream>>>(prob, C, ncomp, flagged, number, id, nseeds, S);
    c->launches += 2;
  }
  exclusive_scan(C.copies, cat, ncomp, scratch, count + 5, c->stream, &c->launches);
  MVG_CUDA_TRY(cudaMemcpyAsync(c->h_scalars, count + 5, 4, cudaMemcpyDeviceToHost, c->stream));
  MVG_CUDA_TRY(cudaStreamSynchronize(c->stream));
  out->rows = ((const uint32_t*)c->h_scalars)[0];
  out->at = cat;
  if (int rc = room_for(out->rows)) return rc;
  k_comp_out_copies<<<grid_for(ncomp, 256), 256, 0, c->stream>>>(prob, C, ncomp, cat);
  c->launches++;
  MVG_CUDA_TRY(cudaGetLastError());
  return 0;
}

// The match list of the pairs in tab (n A positions): rows through prob.row,
// in order of buckets and of the entries in them.  key_bits: width of
// prob.key; room_for(rows) is called before rows are written.  join: the join
// that made the table, whose buckets of repeated mers may be to do (or null).
// Waits for the stream twice (once more for such buckets, three times more with
// flagged ones); the rows' kernel may still be running on return.
template <class P, class F>
int match_components(Ctx* c, P& prob, uint32_t* tab, const PairBucketBufs* join, int64_t n, int key_bits, F room_for,
                     ComponentResult* out) {
  Workspace& ws = c->ws;
  const int64_t ntiles = div_up(n, kSegTile);
  uint32_t* masks = (uint32_t*)ws.get(c, 39, (size_t)ntiles * (kSegTile / 32) * 2 * 4);
  // head and tail counts per tile, their offsets, scan scratch
  uint32_t* tcount = (uint32_t*)ws.get(c, 44, ((size_t)ntiles * 4 + scan_scratch_words(2 * ntiles) + 16) * 4);
  uint32_t* scal = (uint32_t*)ws.get(c, 34, 64);  // segment ends, pairs, what the join left; components, flagged buckets
  if (!masks || !tcount || !scal) return report_error(MVG_ERR_NOMEM, "workspace allocation failed");
  uint32_t *headw = masks, *tailw = masks + ntiles * (kSegTile / 32);
  uint32_t *toff = tcount + 2 * ntiles, *tscr = toff + 2 * ntiles;
  const uint32_t* left = join ? join->pieces.count : nullptr;
  for (;;) {
    MVG_CUDA_TRY(cudaMemsetAsync(scal, 0, 64, c->stream));
    stage_mark(c, "segments");
    k_seg_bits<<<(unsigned)ntiles, 256, 0, c->stream>>>(prob, tab, n, headw, tailw, tcount, ntiles, scal + 1, left,
                                                        scal + 2);
    c->launches++;
    scan_counts(tcount, 2 * ntiles, toff, tscr, scal, c->stream, &c->launches);
    MVG_CUDA_TRY(cudaMemcpyAsync(c->h_scalars, scal, 12, cudaMemcpyDeviceToHost, c->stream));
    if (int rc = check_device_error(c)) return rc;
    if (((const uint32_t*)c->h_scalars)[2] == 0) break;
    // few inputs have any: asked for here, where the host waits anyway (a
    // launch that looks for them took 8 of 231 us of a 1 Mbp pair)
    left = nullptr;
    stage_mark(c, "repeats");
    pair_bucket_repeats(c, *join, tab);
  }
  const int64_t ends = ((const uint32_t*)c->h_scalars)[0], nseg = ends / 2;
  out->pairs = ((const uint32_t*)c->h_scalars)[1];
  if (out->pairs == 0) return 0;

  uint32_t* k0 = (uint32_t*)ws.get(c, 40, ends * 4);
  uint32_t* v0 = (uint32_t*)ws.get(c, 41, ends * 4);
  uint32_t* k1 = (uint32_t*)ws.get(c, 42, ends * 4);
  uint32_t* v1 = (uint32_t*)ws.get(c, 48, ends * 4);
  uint32_t* sscr = (uint32_t*)ws.get(c, 43, sort_scratch_words(ends, key_bits + 1) * 4);
  // per segment: last position, two walks, the join with the next one; its
  // tiles' component counts and offsets; per component (at most one per
  // segment) its fields, its bucket's flag and the list of flagged buckets
  const int64_t ctiles = div_up(nseg, kSegTile);
  uint64_t* blk = (uint64_t*)ws.get(
      c, 45, (size_t)nseg * (8 * 2 + 4 * 7 + 4 * 3 + 1) + (2 * ctiles + scan_scratch_words(ctiles)) * 4 + 256);
  if (!k0 || !v0 || !k1 || !v1 || !sscr || !blk) return report_error(MVG_ERR_NOMEM, "workspace allocation failed");
  Components& C = out->C;
  C.diag = blk;
  C.time = blk + nseg;
  uint32_t* w = (uint32_t*)(blk + 2 * nseg);
  auto take = [&](int64_t k) {
    uint32_t* p = w;
    w += k;
    return p;
  };
  C.lo = take(nseg);
  C.hi = take(nseg);
  C.seed = take(nseg);
  C.key = take(nseg);
  C.copies = take(nseg);
  uint32_t *bflag = take(nseg), *flagged = take(nseg);
  uint32_t *last = take(nseg), *moved = take(2 * nseg);
  uint32_t *ccount = take(ctiles), *coff = take(ctiles), *cscr = take(scan_scratch_words(ctiles));
  uint8_t* joined = (uint8_t*)w;
  if (int rc = room_for((uint64_t)nseg)) return rc;
  k_seg_emit<<<(unsigned)ntiles, 128, 0, c->stream>>>(prob, tab, headw, tailw, toff, ntiles, key_bits, k0, v0);
  stage_mark(c, "segment_sort");
  const bool alt = sort_pairs<uint32_t>(k0, v0, k1, v1, ends, key_bits + 1, sscr, c->stream, &c->launches, c->d_err) != 0;
  const uint32_t *key = alt ? k1 : k0, *head = alt ? v1 : v0, *tail = head + nseg;
  stage_mark(c, "walks");
  k_seg_pair<<<div_up(nseg, 256), 256, 0, c->stream>>>(tab, head, key, tail, nseg, last);
  k_seg_walk<<<div_up(2 * nseg * 2, 256), 256, 0, c->stream>>>(prob, tab, key, head, last, nseg, moved, joined);
  stage_mark(c, "components");
  MVG_CUDA_TRY(cudaMemsetAsync(bflag, 0, (size_t)nseg * 4, c->stream));
  k_comp_count<<<(unsigned)ctiles, 256, 0, c->stream>>>(joined, nseg, ccount);
  scan_counts(ccount, ctiles, coff, cscr, scal + 3, c->stream, &c->launches);
  k_comp_emit<<<(unsigned)ctiles, 256, 0, c->stream>>>(tab, key, head, last, moved, joined, nseg, coff, C);
  k_comp_out<<<grid_for(nseg, 256), 256, 0, c->stream>>>(prob, C, scal + 3, bflag, flagged, scal + 4);
  c->launches += 6;
  stage_mark(c, "flagged");
  MVG_CUDA_TRY(cudaMemcpyAsync(c->h_scalars, scal + 3, 8, cudaMemcpyDeviceToHost, c->stream));
  if (int rc = check_device_error(c)) return rc;
  out->ncomp = ((const uint32_t*)c->h_scalars)[0];
  out->rows = out->ncomp;
  const uint32_t nflagged = ((const uint32_t*)c->h_scalars)[1];
  return nflagged ? flagged_components(c, prob, tab, flagged, nflagged, room_for, out) : 0;
}

}  // namespace mvg
