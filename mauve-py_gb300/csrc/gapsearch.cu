// Batched gap anchor search: ProgressiveAligner::pairwiseAnchorSearch
// (LM/ProgressiveAligner.cpp:590-679) for every inter-anchor gap of a
// recursion round in one pass over the GPU.
//
// Per gap the reference cuts the two gap sequences out of the genomes, picks
// the seed weight getDefaultSeedWeight of their mean length (no search below
// MIN_DNA_SEED_WEIGHT = 5, LM/SeedMasks.h:375), builds a DNAMemorySML of each
// with the rank-0 spaced seed, runs MemHash::FindMatches (seeds unique in both
// gap sequences, hashed by diagonal offset into 40,000 buckets, extended to
// maximal matches), then EliminateOverlaps_v2 (LM/ProgressiveAligner.h:302-392)
// and LengthFilter(MIN_ANCHOR_LENGTH + 3) (LM/MatchList.h:680-692), and shifts
// the anchors to genome coordinates.  Gaps never interact, so here all gaps
// are one segmented problem:
//
//   k_gs_pack        each gap's sequences 2-bit packed into their own word
//                    range (zero padded like translate32's buffer)
//   k_gs_keys,       the seed join of pair_buckets.cu over all gaps' positions
//   k_gs_scatter     at once, with keys (gap, canonical rank-0 seed mer of the
//                    gap's own seed): the seeds unique in each gap, by A slot
//   match_components the genome matcher's match list (match_components.cuh)
//                    over all gaps, its buckets (gap, bucket): GetMatchList
//                    order per gap
//   k_gs_filter      EliminateOverlaps_v2 and LengthFilter per gap, where no
//                    two matches have equal left ends (any sort gives the
//                    reference's order then)
//   host             the same with std::sort for the other gaps (the order of
//                    equal left ends is the library sort's, as in the
//                    reference) and for gaps of more matches than shared
//                    memory takes
//
// A gap's positions take slots from a multiple of 32 on, with at least 31
// empty ones after them, so that chains of seeds never cross into the next
// gap and a warp's 32 slots are one gap's.  (A joint 64-bit radix sort of all
// keys and a warp's replay per (gap, bucket) took 6.6 ms of device time for
// 5,003 gaps of 200-20,000 bp, 43 Mbp; the device passes
// here take 2.8 ms.)
#include <string.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <thread>
#include <vector>

#include "match_components.cuh"

namespace mvg {

constexpr int kGsMinWeight = 5;      // MIN_DNA_SEED_WEIGHT, LM/SeedMasks.h:375
constexpr int64_t kGsMinAnchor = 12;  // MIN_ANCHOR_LENGTH + 3, LM/Aligner.h:266
constexpr int kGsSlot = 80;           // workspace slots 80..95

// translate32's table (LM/SortedMerList.cpp:29-47) for this module; bit 7
// flags '-'.  Rank-0 seeds by weight (LM/SeedMasks.h:298-321).
__constant__ uint8_t c_gs_base[256];
__constant__ SeedDesc c_gs_seed[32];

struct GapDev {
  uint64_t src[2];   // first base of the gap in genome A / B
  uint64_t word[2];  // first packed word of the gap's A / B sequence
  uint32_t slot[2];  // first slot of the gap's A / B positions
  uint32_t cnt[2];   // seed positions
  uint32_t len[2];   // gap lengths
  int32_t w;         // seed weight
  int32_t pad;
};

// Index of the last gap whose packed words start at or before x.
__device__ __forceinline__ int gap_of(const GapDev* __restrict__ g, int n, int side, uint64_t x) {
  int lo = 0, len = n;
  while (len > 0) {
    const int half = len >> 1;
    if (g[lo + half].word[side] <= x) {
      lo += half + 1;
      len -= half + 1;
    } else {
      len = half;
    }
  }
  return lo - 1;
}

// One thread per packed word of all gaps' sequences (A words, then B words).
__global__ void k_gs_pack(const uint8_t* __restrict__ ga, const uint8_t* __restrict__ gb,
                          const GapDev* __restrict__ gaps, int ngaps, uint64_t words_a, uint64_t words_b,
                          uint32_t* __restrict__ pa, uint32_t* __restrict__ pb, uint32_t* err) {
  const uint64_t total = words_a + words_b, stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += stride) {
    const int side = t < words_a ? 0 : 1;
    const uint64_t w = side ? t - words_a : t;
    const int g = gap_of(gaps, ngaps, side, w);
    const GapDev& d = gaps[g];
    const uint8_t* s = (side ? gb : ga) + d.src[side];
    const uint64_t b0 = (w - d.word[side]) * 16;
    uint32_t word = 0, bad = 0;
#pragma unroll 4
    for (int k = 0; k < 16; ++k) {
      const uint64_t i = b0 + k;
      if (i < d.len[side]) {
        const uint32_t v = c_gs_base[s[i]];
        bad |= v;
        word |= (v & 3u) << (30 - 2 * k);
      }
    }
    if (bad & 0x80u) set_error(err, kDevGapChar);
    (side ? pb : pa)[w] = word;
  }
}

// The gap of every 32 slots (a CTA per gap).
__global__ void k_gs_slots(const GapDev* __restrict__ gaps, uint32_t* __restrict__ ga, uint32_t* __restrict__ gb) {
  const GapDev& d = gaps[blockIdx.x];
#pragma unroll
  for (int side = 0; side < 2; ++side) {
    const uint32_t w0 = d.slot[side] >> 5, n = d.cnt[side] ? (d.cnt[side] + 62) >> 5 : 0;
    for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) (side ? gb : ga)[w0 + k] = blockIdx.x;
  }
}

// All gaps as one matching problem over their slots.
struct GapSet {
  const uint32_t *pa, *pb;
  const GapDev* gaps;
  const uint32_t *ga, *gb;  // the gap of every 32 A / B slots
  uint32_t slots[2];
  int mbits;     // mer bits: the widest seed's
  int32_t* out;  // rows (start A, start B, length) in gap coordinates
  int mer_bits() const { return mbits; }
  __device__ __forceinline__ int seed_len(uint32_t x) const { return c_gs_seed[gaps[ga[x >> 5]].w].L; }
  __device__ __forceinline__ uint32_t key(uint32_t v, uint32_t x) const {
    const uint32_t g = ga[x >> 5];
    const GapDev& d = gaps[g];
    return g << 16 | diag_bucket(seed_diag(v - d.slot[1], x - d.slot[0]), c_gs_seed[d.w].L);
  }
  __device__ __forceinline__ MatchView view(uint32_t x, uint32_t& a, uint32_t& b) const {
    const GapDev& d = gaps[ga[x >> 5]];
    a = d.slot[0];
    b = d.slot[1];
    return MatchView{{pa + d.word[0], pb + d.word[1]}, {d.len[0], d.len[1]}, c_gs_seed[d.w]};
  }
  __device__ __forceinline__ void row(uint64_t diag, uint32_t lo, uint32_t hi, uint64_t at) const {
    const GapDev& d = gaps[ga[lo >> 5]];
    const Mhe m = diag_entry(diag, lo, hi, c_gs_seed[d.w].L);
    out[3 * at + 0] = (int32_t)(m.s0 - d.slot[0]);
    out[3 * at + 1] = (int32_t)(m.s1 > 0 ? m.s1 - d.slot[1] : m.s1 + d.slot[1]);
    out[3 * at + 2] = (int32_t)m.len;
  }
};

// The gather tables (gather_mer) of the weights in `weights` (bit w; the
// default weights are odd, 5 to 15), 6 window bytes each: seeds of up to 23
// bases.  (Gathering run by run, some 190 instructions per position, took 0.48
// ms for the keys of 43 Mbp and 0.58 for their scatter, with the tables 0.32 and
// 0.53.)
constexpr int kGsTables = 6, kGsTableBytes = 6;
constexpr int kGsLutBytes = kGsTables * kGsTableBytes * 256 * 4;
using GsLut = uint32_t (*)[kGsTableBytes][256];
__device__ __forceinline__ void gs_lut(uint32_t weights, GsLut lut) {
  for (int t = 0; t < kGsTables; ++t)
    if (weights >> (kGsMinWeight + 2 * t) & 1) seed_lut_build32(c_gs_seed[kGsMinWeight + 2 * t], lut[t]);
}

// Calls f(mixed keys, strands, in B, first slot, valid) for groups of four
// slots of this block's tile (A's, then B's), of which those with a bit in
// `valid` hold a seed position; a warp's slots, and so a group's, are aligned
// pieces of gaps.  A group's seeds lie in one 32-base window.
template <class F>
__device__ __forceinline__ void gs_tile(const GapSet& P, GsLut lut, int bits, int64_t tile, F f) {
  const uint64_t n = (uint64_t)P.slots[0] + P.slots[1], base = (uint64_t)blockIdx.x * (uint64_t)tile;
  for (int64_t o = 4 * threadIdx.x; o < tile; o += 4 * blockDim.x) {
    const uint64_t p = base + (uint64_t)o;
    if (p >= n) break;
    const int side = p >= P.slots[0];
    const uint32_t q = (uint32_t)(side ? p - P.slots[0] : p);
    const uint32_t g = (side ? P.gb : P.ga)[q >> 5];
    const GapDev& d = P.gaps[g];
    const uint32_t x = q - d.slot[side];
    if (x >= d.cnt[side]) continue;
    const SeedDesc& s = c_gs_seed[d.w];
    const uint32_t(*const table)[256] = lut[(d.w - kGsMinWeight) >> 1];
    const int nb = seed_bytes(s), w = s.w;
    const uint64_t win = window64((side ? P.pb : P.pa) + d.word[side], x);
    uint64_t key[4];
    uint32_t strand[4], valid = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      uint32_t fw = 0;
#pragma unroll
      for (int c = 0; c < kGsTableBytes; ++c)
        if (c < nb) fw |= table[c][(uint32_t)(win >> (56 - 8 * c - 2 * u)) & 255u];
      const uint32_t r = revcomp_mer32(fw, w), m = fw < r ? fw : r;
      key[u] = mix_mer<uint64_t>((uint64_t)g << P.mbits | m >> (32 - 2 * w), bits);
      strand[u] = m & 1u;
      valid |= (x + u < d.cnt[side] ? 1u : 0u) << u;
    }
    f(key, strand, side, q, valid);
  }
}

__global__ void __launch_bounds__(1024) k_gs_keys(GapSet P, uint32_t weights, int bits, int bbits, int64_t tile,
                                                  uint32_t* __restrict__ counts) {
  extern __shared__ uint32_t h[];  // nbuckets counts, the gather tables
  const int nbk = 1 << bbits, bsh = bits - bbits;
  GsLut lut = reinterpret_cast<GsLut>(h + nbk);
  gs_lut(weights, lut);
  for (int d = threadIdx.x; d < nbk; d += blockDim.x) h[d] = 0;
  __syncthreads();
  gs_tile(P, lut, bits, tile, [&](const uint64_t(&k)[4], const uint32_t(&)[4], int, uint32_t, uint32_t valid) {
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (valid >> u & 1) atomicAdd(&h[(uint32_t)(k[u] >> bsh)], 1u);
  });
  __syncthreads();
  for (int d = threadIdx.x; d < nbk; d += blockDim.x) counts[(int64_t)blockIdx.x * nbk + d] = h[d];
}

__global__ void __launch_bounds__(1024) k_gs_scatter(GapSet P, uint32_t weights, int bits, int bbits, int64_t tile,
                                                     const uint32_t* __restrict__ offsets, uint2* __restrict__ out) {
  extern __shared__ uint32_t cur[];  // next free slot per bucket, the gather tables
  const int nbk = 1 << bbits, bsh = bits - bbits;
  GsLut lut = reinterpret_cast<GsLut>(cur + nbk);
  gs_lut(weights, lut);
  const uint32_t rest = (uint32_t)(((uint64_t)1 << bsh) - 1);
  for (int d = threadIdx.x; d < nbk; d += blockDim.x) cur[d] = offsets[(int64_t)blockIdx.x * nbk + d];
  __syncthreads();
  gs_tile(P, lut, bits, tile, [&](const uint64_t(&k)[4], const uint32_t(&strand)[4], int side, uint32_t q, uint32_t valid) {
    uint32_t slot[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (valid >> u & 1) slot[u] = atomicAdd(&cur[(uint32_t)(k[u] >> bsh)], 1u);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (valid >> u & 1) out[slot[u]] = make_uint2(((uint32_t)k[u] & rest) << 2 | strand[u] << 1 | (uint32_t)side, q + u);
  });
}

// First row of every gap, and their number.
__global__ void k_gs_gap_rows(const uint32_t* __restrict__ key, uint32_t ncomp, const uint32_t* __restrict__ at,
                              uint32_t rows, uint32_t ngaps, uint32_t* __restrict__ out) {
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g > ngaps) return;
  uint32_t lo = 0, len = g < ngaps ? ncomp : 0;
  while (len > 0) {
    const uint32_t half = len >> 1;
    if (key[lo + half] < g << 16) {
      lo += half + 1;
      len -= half + 1;
    } else {
      len = half;
    }
  }
  out[g] = g == ngaps || lo == ncomp ? rows : at ? at[lo] : lo;
}

struct Anchor {  // in gap coordinates
  int32_t s[2];
  int32_t len;
};
__host__ __device__ __forceinline__ int32_t left_end(const Anchor& m, int q) { return m.s[q] < 0 ? -m.s[q] : m.s[q]; }
// CropStart / CropEnd (LM/UngappedLocalAlignment.h:137-152 over
// LM/HybridAbstractMatch.h:271-290): a forward start follows the first
// column, a reverse start the last.
__host__ __device__ __forceinline__ void crop_start(Anchor& m, int32_t k) {
  m.len -= k;
  for (int q = 0; q < 2; ++q)
    if (m.s[q] > 0) m.s[q] += k;
}
__host__ __device__ __forceinline__ void crop_end(Anchor& m, int32_t k) {
  m.len -= k;
  for (int q = 0; q < 2; ++q)
    if (m.s[q] < 0) m.s[q] -= k;
}

// EliminateOverlaps_v2's walk over one sequence's overlaps
// (LM/ProgressiveAligner.h:302-392, eliminate_both = false): item k's match
// is a[at[k * STEP]], in order of left ends; a match that overlaps a longer one is
// cropped (CropRight / CropLeft in the sequence's orientation) or, when
// nothing is left of it, deleted (at = -1); the cropped-off pieces are
// single-sequence matches, which processNewMatch drops.
template <int STEP>
__host__ __device__ __forceinline__ void walk_overlaps(Anchor* a, int32_t* at, int64_t m, int q) {
  for (int64_t i = 0; i < m; ++i) {
    if (at[i * STEP] < 0) continue;
    Anchor& A = a[at[i * STEP]];
    for (int64_t j = i + 1; j < m; ++j) {
      if (at[j * STEP] < 0) continue;
      Anchor& B = a[at[j * STEP]];
      const int32_t len_i = A.len;
      const int32_t over = len_i - (left_end(B, q) - left_end(A, q));
      if (over <= 0) break;
      if (B.len > len_i) {  // i is the shorter: crop its right end or delete it
        if (over >= len_i) {
          at[i * STEP] = -1;
          break;  // the reference steps back to i, finds it deleted and moves on
        }
        if (A.s[q] > 0) crop_end(A, over);
        else crop_start(A, over);
      } else {  // j is: crop its left end or delete it
        if (over >= B.len)
          at[j * STEP] = -1;
        else if (B.s[q] > 0)
          crop_start(B, over);
        else
          crop_end(B, over);
      }
    }
  }
}

// Overlap elimination and length filter of one gap per CTA: its matches sorted
// in shared memory by their left ends in A and walked, the rest by their left
// ends in B and walked, and the kept ones written over the gap's rows.  A
// match whose left end no earlier match reaches starts a run that shares
// nothing with the matches before it (walking only shortens them), so threads
// walk runs.  What the host has to do is left in todo[g]: 0 nothing; 1 all of
// it, the rows as they were (more than kGsFilterRows matches, or two equal
// left ends in A); m > 1 the B half of the gap's first m rows, which the A half
// left in order (two equal left ends in B).  Latency of the sorts and the
// longest run's walk bound it.  (On 16 host threads, all of it: 1.9 ms per
// 180,000 matches; a walk by one thread per gap: 0.46 ms; with 128 threads
// 0.124 ms, with 256 0.102.)
constexpr int kGsFilterRows = 1536;
constexpr int kGsFilterThreads = 256;
__global__ void __launch_bounds__(kGsFilterThreads)
    k_gs_filter(Anchor* __restrict__ rows, const uint32_t* __restrict__ gap_row, uint32_t* __restrict__ kept,
                uint32_t* __restrict__ todo) {
  constexpr int T = kGsFilterThreads;
  __shared__ uint64_t key[kGsFilterRows];  // the sort's keys; then the runs' heads and the warps' counts
  __shared__ Anchor a[kGsFilterRows];
  __shared__ int32_t order[kGsFilterRows];
  __shared__ int32_t reach[T / 32];
  uint8_t* const head = reinterpret_cast<uint8_t*>(key);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = blockIdx.x;
  const uint32_t r0 = gap_row[g];
  const int n = (int)(gap_row[g + 1] - r0);
  if (n == 0 || n > kGsFilterRows) {
    if (tid == 0) {
      kept[g] = 0;
      todo[g] = n > 0;
    }
    return;
  }
  for (int i = tid; i < n; i += T) {
    a[i] = rows[r0 + i];
    order[i] = i;
  }
  int m = n;  // matches left, in order
  for (int q = 0; q < 2; ++q) {
    int size = 2;  // the sort's; keys from m on count as larger than all others
    while (size < m) size <<= 1;
    __syncthreads();
    for (int i = tid; i < m; i += T) key[i] = (uint64_t)(uint32_t)left_end(a[order[i]], q) << 32 | (uint32_t)order[i];
    __syncthreads();
    for (int len = 2; len <= size; len <<= 1)
      for (int step = len >> 1; step > 0; step >>= 1) {
        const bool first = step == len >> 1;  // mirrored pairs: every pair ascends
        for (int i = tid; i < size / 2; i += T) {
          const int blk = i & ~(step - 1), in = i & (step - 1);
          const int lo = 2 * blk + in, hi = first ? 2 * blk + len - 1 - in : lo + step;
          if (hi >= m) continue;
          const uint64_t x = key[lo], y = key[hi];
          if (x > y) {
            key[lo] = y;
            key[hi] = x;
          }
        }
        __syncthreads();
      }
    bool tie = false;
    for (int i = tid + 1; i < m; i += T) tie |= key[i] >> 32 == key[i - 1] >> 32;
    if (__syncthreads_or(tie)) {
      if (q == 1)
        for (int i = tid; i < m; i += T) rows[r0 + i] = a[order[i]];
      if (tid == 0) {
        kept[g] = 0;
        todo[g] = q == 0 ? 1u : (uint32_t)m;
      }
      return;
    }
    // the farthest end before each thread's matches, which are consecutive
    const int per = (m + T - 1) / T, lo = min(tid * per, m), hi = min(lo + per, m);
    int32_t far = 0;
    for (int i = lo; i < hi; ++i) {
      const int x = (int)(uint32_t)key[i];
      order[i] = x;
      far = max(far, (int32_t)(key[i] >> 32) + a[x].len);
    }
    int32_t scan = far;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int32_t v = __shfl_up_sync(0xffffffffu, scan, d);
      if (lane >= d) scan = max(scan, v);
    }
    if (lane == 31) reach[warp] = scan;
    scan = __shfl_up_sync(0xffffffffu, scan, 1);
    if (lane == 0) scan = 0;
    __syncthreads();
    for (int w = 0; w < warp; ++w) scan = max(scan, reach[w]);
    for (int i = lo; i < hi; ++i) {
      const Anchor& x = a[order[i]];
      const int32_t l = left_end(x, q);
      head[i] = l >= scan;
      scan = max(scan, l + x.len);
    }
    __syncthreads();
    for (int i = tid; i < m; i += T)
      if (head[i]) {
        int e = i + 1;
        while (e < m && !head[e]) ++e;
        if (e > i + 1) walk_overlaps<1>(a, order + i, e - i, q);
      }
    __syncthreads();
    if (tid < 32) {  // the matches left, in order
      int w = 0;
      for (int base = 0; base < m; base += 32) {
        const int x = base + lane < m ? order[base + lane] : -1;
        const unsigned b = __ballot_sync(0xffffffffu, x >= 0);
        __syncwarp();
        if (x >= 0) order[w + __popc(b & ((1u << lane) - 1u))] = x;
        w += __popc(b);
      }
      if (lane == 0) reach[0] = w;
    }
    __syncthreads();
    m = reach[0];
  }
  if (tid < 32) {
    int w = 0;
    for (int base = 0; base < m; base += 32) {
      const int i = base + lane;
      const bool in = i < m && a[order[i < m ? i : 0]].len >= kGsMinAnchor;
      const unsigned b = __ballot_sync(0xffffffffu, in);
      if (in) rows[r0 + w + __popc(b & ((1u << lane) - 1u))] = a[order[i]];
      w += __popc(b);
    }
    if (lane == 0) {
      kept[g] = (uint32_t)w;
      todo[g] = 0;
    }
  }
}

// The kept rows of every gap in genome coordinates, at its first output row.
__global__ void k_gs_out(const Anchor* __restrict__ rows, const uint32_t* __restrict__ gap_row,
                         const uint32_t* __restrict__ kept, const uint32_t* __restrict__ at,
                         const GapDev* __restrict__ gaps, int64_t* __restrict__ out) {
  const int g = blockIdx.x;
  const GapDev& d = gaps[g];
  for (uint32_t u = threadIdx.x; u < kept[g]; u += blockDim.x) {
    const Anchor x = rows[gap_row[g] + u];
    int64_t* o = out + 3 * ((uint64_t)at[g] + u);
#pragma unroll
    for (int q = 0; q < 2; ++q) o[q] = x.s[q] > 0 ? x.s[q] + (int64_t)d.src[q] : x.s[q] - (int64_t)d.src[q];
    o[2] = x.len;
  }
}

// ------------------------------------------------------------------ host

static std::mutex g_gs_mu;
static int g_gs_ready_dev = -1;

static int gs_upload_tables(int device) {
  std::lock_guard<std::mutex> lk(g_gs_mu);
  if (g_gs_ready_dev == device) return 0;
  uint8_t t[256] = {};
  for (const char* p = "cCbByY"; *p; ++p) t[(uint8_t)*p] = 1;
  for (const char* p = "gGsSkK"; *p; ++p) t[(uint8_t)*p] = 2;
  t[(uint8_t)'t'] = t[(uint8_t)'T'] = 3;
  t[(uint8_t)'-'] = 0x80;
  MVG_CUDA_TRY(cudaMemcpyToSymbol(c_gs_base, t, 256));
  SeedDesc sd[32];
  for (int w = 0; w < 32; ++w) sd[w] = make_seed_desc(w >= kGsMinWeight ? mvg_get_seed(w, 0) : 0);
  MVG_CUDA_TRY(cudaMemcpyToSymbol(c_gs_seed, sd, sizeof(sd)));
  g_gs_ready_dev = device;
  return 0;
}

namespace {
// One gap's overlap elimination and length filter with the sort the reference
// uses: std::sort's result on equal left ends follows from the sequence of
// comparisons alone, so (left end, index) pairs are sorted.  from: the first
// sequence (1: A's half is done).  Returns the number kept, at a[0 ..).
struct FilterScratch {
  struct Item {
    int32_t left;
    int32_t at;  // -1: deleted
  };
  std::vector<Item> ml;
  std::vector<Anchor> kept;
};
int64_t filter_gap(Anchor* a, int64_t n, int from, FilterScratch& F) {
  auto& ml = F.ml;
  ml.resize(n);
  for (int64_t k = 0; k < n; ++k) ml[k].at = (int32_t)k;
  if (n >= 2) {
    for (int q = from; q < 2; ++q) {
      for (auto& x : ml) x.left = left_end(a[x.at], q);
      std::sort(ml.begin(), ml.end(),
                [](const FilterScratch::Item& x, const FilterScratch::Item& y) { return x.left < y.left; });
      walk_overlaps<2>(a, &ml[0].at, (int64_t)ml.size(), q);
      ml.erase(std::remove_if(ml.begin(), ml.end(), [](const FilterScratch::Item& x) { return x.at < 0; }), ml.end());
    }
  }
  auto& kept = F.kept;
  kept.clear();
  for (const auto& x : ml)
    if (a[x.at].len >= kGsMinAnchor) kept.push_back(a[x.at]);
  std::copy(kept.begin(), kept.end(), a);
  return (int64_t)kept.size();
}

// One chunk of a call's gaps: the searched gaps' device descriptors and
// caller indices, and the device pass's results in pinned memory: the kept
// rows in genome coordinates and the matches of the gaps left to the host (in
// GetMatchList order).
struct GsChunk {
  std::vector<GapDev> gd;
  std::vector<uint32_t> gid;  // caller's gap index of each searched gap
  uint64_t words[2] = {0, 0};
  uint32_t slots[2] = {0, 0};
  uint64_t keys[2] = {0, 0};
  const int64_t* out = nullptr;  // rows of the gaps filtered on the device, gap by gap
  std::vector<uint32_t> nkept;   // rows per gap
  std::vector<uint32_t> todo;    // gaps left to the host, ascending
  std::vector<uint32_t> todo_at, todo_n;  // their matches: rows[todo_at ..]
  std::vector<uint8_t> todo_q;            // the sequence to begin with
  Anchor* rows = nullptr;
};

// Runs fn(i) for i in [0, n) on up to nthreads host threads that claim runs
// of 16 indices from a counter.
template <class F>
void run_claimed(int n, int nthreads, F&& fn) {
  std::atomic<int> next{0};
  auto worker = [&]() {
    for (;;) {
      const int i0 = next.fetch_add(16);
      if (i0 >= n) break;
      for (int i = i0; i < std::min(n, i0 + 16); ++i) fn(i);
    }
  };
  if (nthreads > 1) {
    std::vector<std::thread> pool;
    for (int t = 0; t < nthreads; ++t) pool.emplace_back(worker);
    for (std::thread& th : pool) th.join();
  } else {
    worker();
  }
}

int host_threads_for(size_t items) {
  const unsigned hw = std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
  return (int)std::min<uint64_t>(hw, std::max<uint64_t>(1, items / 10000));
}
}  // namespace

// Slots of a chunk of gaps, and its most gaps: the seed join's buckets hold
// 2,048 keys each up to 2^25 keys, and its keys 44 bits, 30 of them the
// widest mer's.  Below that a chunk is as
// large as this because the host pass of one chunk runs beside the device
// pass of the next (43 Mbp in gaps: 5.9 ms with 2^23 slots, 5.2 with 2^24, 5.8
// with 2^25, 5.6 in one chunk).
constexpr uint64_t kGsSlots = 1ull << 24;
constexpr size_t kGsGaps = 1u << (kPairMaxBits - 30);

// Host plan (gaps already validated): seed weights, word and slot ranges of
// the gaps that are searched, in chunks.
static int gs_plan(const int64_t* gaps, uint64_t ngaps, uint64_t total_slots, std::vector<GsChunk>& chunks) {
  const uint64_t parts = std::max<uint64_t>(1, (total_slots + kGsSlots - 1) / kGsSlots);
  const uint64_t share = total_slots / parts + 1;
  chunks.emplace_back();
  for (uint64_t g = 0; g < ngaps; ++g) {
    const int64_t* q = gaps + 4 * g;
    const unsigned w = mvg_default_seed_weight((uint64_t)(q[1] + q[3]) / 2);
    if (w < (unsigned)kGsMinWeight) continue;  // the reference returns without searching
    if (w > 15)
      return report_error(MVG_ERR_ARG, "gap of mean length above 5.9 Mbp (seed weight above 15): search it with "
                                       "mvg_pairwise_matches and the rank-0 seed");
    if (chunks.back().gd.size() >= kGsGaps || (uint64_t)chunks.back().slots[0] + chunks.back().slots[1] >= share)
      chunks.emplace_back();
    GsChunk& ch = chunks.back();
    const int L = mvg_seed_length(mvg_get_seed((int)w, 0));
    GapDev d{};
    d.w = (int32_t)w;
    for (int s = 0; s < 2; ++s) {
      const uint64_t len = (uint64_t)q[1 + 2 * s];
      d.src[s] = (uint64_t)q[2 * s];
      d.len[s] = (uint32_t)len;
      d.word[s] = ch.words[s];
      d.slot[s] = ch.slots[s];
      d.cnt[s] = len >= (uint64_t)L ? (uint32_t)(len - L + 1) : 0;
      ch.words[s] += packed_words(len);  // translate32's layout: two zero words after each gap
      ch.keys[s] += d.cnt[s];
      if (d.cnt[s]) ch.slots[s] += (d.cnt[s] + 62) & ~31u;
    }
    ch.gd.push_back(d);
    ch.gid.push_back((uint32_t)g);
  }
  return 0;
}

// Device pass of one chunk, from packing to the kept rows, which are copied to
// the pinned buffer `buf` with the matches of the gaps left to the host.
// Synchronous.
static int gs_device(Ctx* c, const uint8_t* d_a, const uint8_t* d_b, GsChunk& ch, int buf) {
  const int ng = (int)ch.gd.size();
  if (ng == 0) return 0;
  ch.nkept.assign(ng, 0);
  Workspace& ws = c->ws;
  const uint64_t* words = ch.words;
  const uint32_t wa = ch.slots[0] >> 5, wb = ch.slots[1] >> 5;
  GapDev* d_gaps = (GapDev*)ws.get(c, kGsSlot + 0, ng * sizeof(GapDev));
  uint32_t* pa = (uint32_t*)ws.get(c, kGsSlot + 1, words[0] * 4 + 64);
  uint32_t* pb = (uint32_t*)ws.get(c, kGsSlot + 2, words[1] * 4 + 64);
  uint32_t* gmap = (uint32_t*)ws.get(c, kGsSlot + 3, ((size_t)wa + wb) * 4 + 64);
  uint32_t* tab = (uint32_t*)ws.get(c, 38, (size_t)ch.slots[0] * 4 + 64);
  if (!d_gaps || !pa || !pb || !gmap || !tab) return report_error(MVG_ERR_NOMEM, "workspace allocation failed");
  MVG_CUDA_TRY(cudaMemsetAsync(c->d_err, 0, 4, c->stream));
  stage_mark(c, "gs_pack");
  MVG_CUDA_TRY(cudaMemcpyAsync(d_gaps, ch.gd.data(), ng * sizeof(GapDev), cudaMemcpyHostToDevice, c->stream));
  k_gs_pack<<<grid_for(words[0] + words[1], 256), 256, 0, c->stream>>>(d_a, d_b, d_gaps, ng, words[0], words[1],
                                                                        pa, pb, c->d_err);
  c->launches++;
  if (ch.keys[0] == 0 || ch.keys[1] == 0) {  // no seed in one genome's gaps: no match anywhere
    MVG_CUDA_TRY(cudaStreamSynchronize(c->stream));
    return check_device_error(c);
  }
  MVG_CUDA_TRY(cudaMemsetAsync(tab, 0xff, (size_t)ch.slots[0] * 4, c->stream));
  stage_mark(c, "gs_keys");
  int gbits = 1;
  while ((1ll << gbits) < ng) ++gbits;
  // a seed's bits are its pattern's selected positions, which for some table
  // entries exceed the nominal weight (weight 11's rank-0 seed selects 12)
  int wmax = 0;
  uint32_t weights = 0;
  for (const GapDev& d : ch.gd) weights |= 1u << d.w;
  for (int w = kGsMinWeight; w < 32; ++w)
    if (weights >> w & 1) wmax = std::max(wmax, __builtin_popcountll(mvg_get_seed(w, 0)));
  GapSet P{pa, pb, d_gaps, gmap, gmap + wa, {ch.slots[0], ch.slots[1]}, 2 * wmax, nullptr};
  const int bits = 2 * wmax + gbits;
  if (bits > kPairMaxBits) return report_error(MVG_ERR_DEVICE, "gap search keys wider than the join's");
  PairBucketBufs b;
  int rc = pair_bucket_bufs(c, (uint64_t)ch.slots[0] + ch.slots[1], bits, &b);
  if (rc) return rc;
  if (!c->search_ready) {  // more than 48 KB of dynamic shared memory
    MVG_CUDA_TRY(cudaFuncSetAttribute(k_gs_keys, cudaFuncAttributeMaxDynamicSharedMemorySize, 16384 * 4 + kGsLutBytes));
    MVG_CUDA_TRY(cudaFuncSetAttribute(k_gs_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, kOneCta));
    c->search_ready = true;
  }
  const size_t hsm = (size_t)b.g.nbuckets * 4 + kGsLutBytes;
  static_assert(16384 * 4 + kGsLutBytes <= kOneCta, "the scatter's shared memory");
  k_gs_slots<<<ng, 128, 0, c->stream>>>(d_gaps, gmap, gmap + wa);
  k_gs_keys<<<(unsigned)b.g.ntiles, 1024, hsm, c->stream>>>(P, weights, bits, b.g.bbits, b.g.tile, b.counts);
  pair_bucket_offsets(c, b);
  stage_mark(c, "gs_scatter");
  k_gs_scatter<<<(unsigned)b.g.ntiles, 1024, kOneCta, c->stream>>>(P, weights, bits, b.g.bbits, b.g.tile, b.offs, b.buf);
  c->launches += 3;
  stage_mark(c, "gs_join");
  pair_bucket_join(c, b, tab);
  MVG_CUDA_TRY(cudaGetLastError());
  ComponentResult r;
  auto room_for = [&](uint64_t rows) {
    P.out = (int32_t*)ws.get(c, kGsSlot + 5, rows * 12 + 16);
    return P.out ? 0 : report_error(MVG_ERR_NOMEM, "workspace allocation failed");
  };
  if ((rc = match_components(c, P, tab, &b, (int64_t)ch.slots[0], 16 + gbits, room_for, &r))) return rc;
  if (r.rows == 0) return 0;
  stage_mark(c, "gs_filter");
  // per gap: first match, rows kept, left to the host, first output row; their sum (k_gs_filter's todo)
  uint32_t* d_tab = (uint32_t*)ws.get(c, kGsSlot + 4, ((size_t)ng * 4 + 2) * 4);
  int64_t* d_out = (int64_t*)ws.get(c, kGsSlot + 6, r.rows * 24);
  if (!d_tab || !d_out) return report_error(MVG_ERR_NOMEM, "workspace allocation failed");
  uint32_t *gap_row = d_tab, *kept = d_tab + ng + 1, *todo = kept + ng, *at = todo + ng, *sum = at + ng;
  Anchor* d_rows = (Anchor*)P.out;
  k_gs_gap_rows<<<div_up(ng + 1, 256), 256, 0, c->stream>>>(r.C.key, r.ncomp, r.at, (uint32_t)r.rows, (uint32_t)ng,
                                                            gap_row);
  k_gs_filter<<<ng, kGsFilterThreads, 0, c->stream>>>(d_rows, gap_row, kept, todo);
  pair_scan_small(kept, ng, at, sum, c->stream);
  k_gs_out<<<ng, 64, 0, c->stream>>>(d_rows, gap_row, kept, at, d_gaps, d_out);
  c->launches += 4;
  MVG_CUDA_TRY(cudaGetLastError());
  stage_mark(c, "gs_copy");
  const size_t tab_bytes = ((size_t)ng * 4 + 2) * 4;
  uint32_t* h = (uint32_t*)pinned_buf(c, buf, std::max(tab_bytes, (size_t)r.rows * 24 + 256));
  if (!h) return report_error(MVG_ERR_NOMEM, "pinned allocation failed");
  MVG_CUDA_TRY(cudaMemcpyAsync(h, d_tab, tab_bytes, cudaMemcpyDeviceToHost, c->stream));
  MVG_CUDA_TRY(cudaStreamSynchronize(c->stream));
  std::vector<uint32_t> first(h, h + ng + 1);
  ch.nkept.assign(h + ng + 1, h + 2 * ng + 1);
  const uint64_t nout = h[4 * ng + 1];
  uint64_t nrows = 0;
  for (int g = 0; g < ng; ++g)
    if (const uint32_t t = h[2 * ng + 1 + g]) {
      ch.todo.push_back((uint32_t)g);
      ch.todo_q.push_back(t > 1);
      ch.todo_n.push_back(t > 1 ? t : first[g + 1] - first[g]);
      ch.todo_at.push_back((uint32_t)nrows);
      nrows += ch.todo_n.back();
    }
  const bool all = ch.todo.size() > 32;  // one copy of every row instead of a copy per gap
  if (all) {
    nrows = r.rows;
    for (size_t k = 0; k < ch.todo.size(); ++k) ch.todo_at[k] = first[ch.todo[k]];
  }
  const size_t rows_at = (nout * 24 + 255) & ~(size_t)255;
  uint8_t* base = pinned_buf(c, buf, rows_at + nrows * sizeof(Anchor));
  if (!base) return report_error(MVG_ERR_NOMEM, "pinned allocation failed");
  ch.out = (const int64_t*)base;
  ch.rows = (Anchor*)(base + rows_at);
  if (nout) MVG_CUDA_TRY(cudaMemcpyAsync(base, d_out, nout * 24, cudaMemcpyDeviceToHost, c->stream));
  if (all) MVG_CUDA_TRY(cudaMemcpyAsync(ch.rows, d_rows, nrows * sizeof(Anchor), cudaMemcpyDeviceToHost, c->stream));
  for (size_t k = 0; k < ch.todo.size() && !all; ++k)
    MVG_CUDA_TRY(cudaMemcpyAsync(ch.rows + ch.todo_at[k], d_rows + first[ch.todo[k]], ch.todo_n[k] * sizeof(Anchor),
                                 cudaMemcpyDeviceToHost, c->stream));
  MVG_CUDA_TRY(cudaStreamSynchronize(c->stream));
  return 0;
}

// Host pass of one chunk: the gaps the device left (their sizes differ by
// orders of magnitude, so host threads claim them), and all rows to the
// caller's output from row `base` on.  Returns the row after the chunk's last.
static uint64_t gs_finish(GsChunk& ch, int64_t* out, uint64_t cap, uint64_t base) {
  const size_t nt = ch.todo.size();
  uint64_t nrows = 0;
  for (uint32_t n : ch.todo_n) nrows += n;
  run_claimed((int)nt, host_threads_for(nrows), [&](int k) {
    FilterScratch scratch;
    ch.nkept[ch.todo[k]] = (uint32_t)filter_gap(ch.rows + ch.todo_at[k], ch.todo_n[k], ch.todo_q[k], scratch);
  });
  const int64_t* src = ch.out;
  size_t g = 0;
  auto copy = [&](size_t to) {  // the device's rows of gaps [g, to), none of them in todo
    uint64_t n = 0;
    for (; g < to; ++g) n += ch.nkept[g];
    const uint64_t fit = base < cap ? std::min(n, cap - base) : 0;
    if (fit) memcpy(out + 3 * base, src, fit * 24);
    src += 3 * n;
    base += n;
  };
  for (size_t k = 0; k < nt; ++k) {
    copy(ch.todo[k]);
    const GapDev& d = ch.gd[g];
    for (uint32_t u = 0; u < ch.nkept[g]; ++u, ++base) {
      if (base >= cap) continue;
      const Anchor& x = ch.rows[ch.todo_at[k] + u];
      int64_t* o = out + 3 * base;
      for (int q = 0; q < 2; ++q) o[q] = x.s[q] > 0 ? x.s[q] + (int64_t)d.src[q] : x.s[q] - (int64_t)d.src[q];
      o[2] = x.len;
    }
    ++g;
  }
  copy(ch.nkept.size());
  return base;
}

// Gaps are searched in chunks: the host pass of one chunk runs on host
// threads while the device pass of the next runs on the GPU.
int gap_anchor_search_dev(Ctx* c, const uint8_t* d_a, uint64_t na, const uint8_t* d_b, uint64_t nb,
                          const int64_t* gaps, uint64_t ngaps, int64_t* out, uint64_t cap, uint64_t* gap_off,
                          uint64_t* count) {
  *count = 0;
  stage_begin_call(c);
  if (ngaps >= (1ull << 31)) return report_error(MVG_ERR_ARG, "too many gaps");
  int rc = gs_upload_tables(c->device);
  if (rc) return rc;
  uint64_t total_slots = 0;
  for (uint64_t g = 0; g < ngaps; ++g) {
    const int64_t* q = gaps + 4 * g;
    if (q[0] < 0 || q[1] < 0 || q[2] < 0 || q[3] < 0 || (uint64_t)(q[0] + q[1]) > na ||
        (uint64_t)(q[2] + q[3]) > nb)
      return report_error(MVG_ERR_RANGE, "gap outside its genome");
    if (q[1] >= (1ll << 31) || q[3] >= (1ll << 31)) return report_error(MVG_ERR_ARG, "gap longer than 2^31-1");
    total_slots += (uint64_t)(q[1] + q[3]) + 62;
  }
  std::vector<GsChunk> chunks;
  if ((rc = gs_plan(gaps, ngaps, total_slots, chunks))) return rc;
  uint64_t total = 0;  // rows of the chunks filtered so far
  std::thread filt;    // the host pass of the previous chunk
  struct Joiner {
    std::thread& t;
    ~Joiner() {
      if (t.joinable()) t.join();
    }
  } joiner{filt};
  for (size_t k = 0; k < chunks.size(); ++k) {
    if ((rc = gs_device(c, d_a, d_b, chunks[k], (int)(k & 1)))) return rc;
    HostSpan wait(c, "gs_filter_wait");
    if (filt.joinable()) filt.join();
    GsChunk& ch = chunks[k];
    if (k + 1 < chunks.size())
      filt = std::thread([&ch, &total, out, cap] { total = gs_finish(ch, out, cap, total); });
    else
      total = gs_finish(ch, out, cap, total);
  }
  stage_end(c);
  if (gap_off) {
    std::vector<uint64_t> per_gap(ngaps, 0);
    for (const GsChunk& ch : chunks)
      for (size_t gi = 0; gi < ch.gd.size(); ++gi) per_gap[ch.gid[gi]] = ch.nkept[gi];
    gap_off[0] = 0;
    for (uint64_t g = 0; g < ngaps; ++g) gap_off[g + 1] = gap_off[g] + per_gap[g];
  }
  *count = total;
  if (total > cap) return report_error(MVG_ERR_CAPACITY, "anchor output buffer too small");
  return 0;
}

}  // namespace mvg

using namespace mvg;

static Ctx* gs_ctx(mvg_handle h) { return reinterpret_cast<Ctx*>(h); }

extern "C" int mvg_gap_anchor_search_dev(mvg_handle h, const uint8_t* d_seq_a, uint64_t na, const uint8_t* d_seq_b,
                                         uint64_t nb, const int64_t* gaps, uint64_t ngaps, int64_t* out,
                                         uint64_t cap, uint64_t* gap_off, uint64_t* count) {
  if (!h || !count || (!gaps && ngaps) || (!out && cap) || (!d_seq_a && na) || (!d_seq_b && nb))
    return report_error(MVG_ERR_ARG, "null argument");
  Ctx* c = gs_ctx(h);
  MVG_CUDA_TRY(cudaSetDevice(c->device));
  return gap_anchor_search_dev(c, d_seq_a, na, d_seq_b, nb, gaps, ngaps, out, cap, gap_off, count);
}

extern "C" int mvg_gap_anchor_search(mvg_handle h, const uint8_t* seq_a, uint64_t na, const uint8_t* seq_b,
                                     uint64_t nb, const int64_t* gaps, uint64_t ngaps, int64_t* out, uint64_t cap,
                                     uint64_t* gap_off, uint64_t* count) {
  if (!h || !count || (!gaps && ngaps) || (!out && cap) || (!seq_a && na) || (!seq_b && nb))
    return report_error(MVG_ERR_ARG, "null argument");
  Ctx* c = gs_ctx(h);
  MVG_CUDA_TRY(cudaSetDevice(c->device));
  uint8_t* da = (uint8_t*)c->ws.get(c, 46, na + 16);
  uint8_t* db = (uint8_t*)c->ws.get(c, 47, nb + 16);
  if (!da || !db) return report_error(MVG_ERR_NOMEM, "workspace allocation failed");
  if (na) MVG_CUDA_TRY(cudaMemcpyAsync(da, seq_a, na, cudaMemcpyHostToDevice, c->stream));
  if (nb) MVG_CUDA_TRY(cudaMemcpyAsync(db, seq_b, nb, cudaMemcpyHostToDevice, c->stream));
  return gap_anchor_search_dev(c, da, na, db, nb, gaps, ngaps, out, cap, gap_off, count);
}
