// Device primitives shared by the seed and match kernels: an exclusive scan
// over uint32 and a stable LSD radix sort of (key, uint32 value) pairs.
//
// Radix sort, one 8-bit digit per pass:
//   k_digit_hist   per-tile digit counts           (reads keys once)
//   scan           exclusive scan of the digit-major count table
//   k_digit_scatter stages the tile in shared memory in stable digit order,
//                   then writes each digit's run contiguously (coalesced).
// Stability inside a tile comes from ranking 256-element chunks in order with
// __match_any_sync peer masks and per-warp counts, so equal digits keep their
// input order and the whole sort is stable.
#pragma once
#include <atomic>

#include "mvg_common.cuh"

namespace mvg {

constexpr int kScanTile = 4096;  // elements per scan block (256 threads x 16)
constexpr int kSortThreads = 256;
constexpr int kSortTile = 2048;  // elements per sort block (8 chunks of 256)

// ------------------------------------------------------------------ scan

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    uint32_t t = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= d) v += t;
  }
  return v;
}

// Block-wide exclusive scan of one value per thread (blockDim.x == 256).
// Returns the exclusive prefix; *total gets the block sum.
__device__ __forceinline__ uint32_t block_excl_scan256(uint32_t v, uint32_t* total) {
  __shared__ uint32_t wsum[8];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t inc = warp_incl_scan(v);
  if (lane == 31) wsum[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    uint32_t x = lane < 8 ? wsum[lane] : 0;
    uint32_t y = warp_incl_scan(x);
    if (lane < 8) wsum[lane] = y - x;
    if (lane == 7 && total) *total = y;
  }
  __syncthreads();
  uint32_t r = wsum[wid] + inc - v;
  __syncthreads();
  return r;
}

// Pass 1: per-block sums of tiles of kScanTile elements.
__global__ void k_scan_reduce(const uint32_t* __restrict__ in, int64_t n, uint32_t* __restrict__ bsum);
// Pass 2: exclusive scan of the block sums (one block, loops over chunks).
__global__ void k_scan_bsums(uint32_t* __restrict__ bsum, int64_t nb, uint32_t* __restrict__ total);
// Pass 3: exclusive scan of each tile plus its block prefix.
__global__ void k_scan_down(const uint32_t* in, int64_t n, const uint32_t* __restrict__ bsum, uint32_t* out);

// Host side: exclusive scan of n uint32 into out (may alias in); *d_total
// (device) gets the sum.  scratch needs scan_scratch_words(n) words.
inline int64_t scan_scratch_words(int64_t n) { return (n + kScanTile - 1) / kScanTile + 1; }
void exclusive_scan(const uint32_t* in, uint32_t* out, int64_t n, uint32_t* scratch, uint32_t* d_total,
                    cudaStream_t st, uint64_t* launches);

// ------------------------------------------------------------ radix sort

template <typename K>
__global__ void k_digit_hist(const K* __restrict__ keys, int64_t n, int shift, uint32_t* __restrict__ counts,
                             int nblocks) {
  __shared__ uint32_t h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kSortTile;
  const int64_t end = min(base + kSortTile, n);
  for (int64_t i = base + threadIdx.x; i < end; i += kSortThreads) {
    uint32_t d = (uint32_t)(keys[i] >> shift) & 255u;
    atomicAdd(&h[d], 1u);
  }
  __syncthreads();
  counts[(int64_t)threadIdx.x * nblocks + blockIdx.x] = h[threadIdx.x];
}

template <typename K>
__global__ void __launch_bounds__(kSortThreads) k_digit_scatter(const K* __restrict__ kin, const uint32_t* __restrict__ vin,
                                                                K* __restrict__ kout, uint32_t* __restrict__ vout, int64_t n,
                                                                int shift, const uint32_t* __restrict__ counts,
                                                                const uint32_t* __restrict__ offsets, int nblocks) {
  __shared__ K skey[kSortTile];
  __shared__ uint32_t sval[kSortTile];
  __shared__ uint32_t wcnt[8][256];
  __shared__ uint32_t run[256];
  __shared__ uint32_t lstart[256];
  __shared__ uint32_t gbase[256];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int64_t base = (int64_t)blockIdx.x * kSortTile;
  const int tile_n = (int)min((int64_t)kSortTile, n - base);

  uint32_t mycount = counts[(int64_t)tid * nblocks + blockIdx.x];
  gbase[tid] = offsets[(int64_t)tid * nblocks + blockIdx.x];
  uint32_t ls = block_excl_scan256(mycount, nullptr);
  lstart[tid] = ls;
  run[tid] = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) wcnt[w][tid] = 0;
  __syncthreads();

  const uint32_t lt_mask = (1u << lane) - 1u;
  for (int c = 0; c < kSortTile; c += kSortThreads) {
    const int li = c + tid;
    const bool valid = li < tile_n;
    K key = 0;
    uint32_t val = 0, d = 256u + (uint32_t)lane;  // invalid lanes get private digits
    if (valid) {
      key = kin[base + li];
      val = vin[base + li];
      d = (uint32_t)(key >> shift) & 255u;
    }
    uint32_t peers = __match_any_sync(0xffffffffu, d);
    uint32_t lrank = __popc(peers & lt_mask);
    if (valid && lrank == 0) wcnt[wid][d] = __popc(peers);
    __syncthreads();
    if (valid) {
      uint32_t r = run[d] + lrank;
      for (int w = 0; w < wid; ++w) r += wcnt[w][d];
      const uint32_t lp = lstart[d] + r;
      skey[lp] = key;
      sval[lp] = val;
    }
    __syncthreads();
    {
      uint32_t s = 0;
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        s += wcnt[w][tid];
        wcnt[w][tid] = 0;
      }
      run[tid] += s;
    }
    __syncthreads();
    if (c + kSortThreads >= tile_n) break;
  }
  for (int i = tid; i < tile_n; i += kSortThreads) {
    K key = skey[i];
    uint32_t d = (uint32_t)(key >> shift) & 255u;
    int64_t o = (int64_t)gbase[d] + (i - (int)lstart[d]);
    kout[o] = key;
    vout[o] = sval[i];
  }
}

// Stable LSD radix sort of (keys, vals) on bits [0, nbits).  Ping-pongs
// between the input arrays and the alternates; returns which buffer holds
// the result (0 = keys/vals, 1 = alt).  scratch: radix_scratch_words(n).
inline int64_t radix_scratch_words(int64_t n) {
  int64_t nb = (n + kSortTile - 1) / kSortTile;
  return 2 * 256 * nb + scan_scratch_words(256 * nb) + 2;
}

template <typename K>
int radix_sort_pairs(K* keys, uint32_t* vals, K* keys_alt, uint32_t* vals_alt, int64_t n, int nbits,
                     uint32_t* scratch, cudaStream_t st, uint64_t* launches) {
  if (n <= 0) return 0;
  const int nb = (int)((n + kSortTile - 1) / kSortTile);
  uint32_t* counts = scratch;
  uint32_t* offsets = scratch + (int64_t)256 * nb;
  uint32_t* sscr = offsets + (int64_t)256 * nb;
  uint32_t* total = sscr + scan_scratch_words((int64_t)256 * nb);
  K* ka = keys;
  K* kb = keys_alt;
  uint32_t* va = vals;
  uint32_t* vb = vals_alt;
  int which = 0;
  for (int shift = 0; shift < nbits; shift += 8) {
    k_digit_hist<K><<<nb, kSortThreads, 0, st>>>(ka, n, shift, counts, nb);
    exclusive_scan(counts, offsets, (int64_t)256 * nb, sscr, total, st, launches);
    k_digit_scatter<K><<<nb, kSortThreads, 0, st>>>(ka, va, kb, vb, n, shift, counts, offsets, nb);
    if (launches) *launches += 2;
    K* tk = ka;
    ka = kb;
    kb = tk;
    uint32_t* tv = va;
    va = vb;
    vb = tv;
    which ^= 1;
  }
  return which;
}

// ------------------------------------- reduce-then-scan radix sort
//
// Stable LSD sort by 8-bit digits, three kernels per pass and no waits
// between tiles:
//   k_rts_count    per tile of keys: its 256 digit counts, stored
//                  tile-major (one coalesced 1 KB row per tile), and added
//                  into the counts of the tile's chunk (ctiles tiles)
//   k_rts_offsets  one block per chunk: every digit's global start (from
//                  all chunks' sums) plus the chunks before this one, then
//                  the chunk's tiles' rows turned into output offsets in
//                  place
//   k_rts_scatter  per tile: keys ranked stably in shared memory and
//                  written out digit run by digit run
// Rows are read and written whole, so every count access is coalesced; the
// chunk sums make the offsets kernel a two-level scan with no serial walk
// over thousands of tiles.
namespace os {
constexpr int kThreads = 256;
constexpr int kItems = 8;
constexpr int kTile = kThreads * kItems;
}  // namespace os

struct RtsGeom {
  int64_t ntiles, ctiles, nchunks;
  int npass;
};

// Chunks of at least 64 tiles and at most about 128 chunks.
inline RtsGeom rts_geom(int64_t n, int nbits) {
  RtsGeom g;
  g.npass = (nbits + 7) / 8;
  g.ntiles = (n + os::kTile - 1) / os::kTile;
  int64_t ct = (g.ntiles + 127) / 128;
  ct = (ct + 3) & ~3ll;
  g.ctiles = ct < 64 ? 64 : ct;
  g.nchunks = (g.ntiles + g.ctiles - 1) / g.ctiles;
  return g;
}

// Scratch layout: the tile count rows (ntiles x 256 words, reused by every
// pass), then each pass's chunk sums (nchunks x 256 words per pass, zeroed
// before the sort).  nchunks <= min(ntiles, 128), so sizing by that bound
// makes a scratch sized for n and nbits fit every smaller sort.
inline int64_t rts_scratch_words(int64_t n, int nbits) {
  const RtsGeom g = rts_geom(n, nbits);
  const int64_t cap = g.ntiles < 128 ? g.ntiles : 128;
  return g.ntiles * 256 + (int64_t)g.npass * cap * 256 + 16;
}
inline uint32_t* rts_counts(uint32_t* scratch) { return scratch; }
inline uint32_t* rts_csum(uint32_t* scratch, const RtsGeom& g) { return scratch + g.ntiles * 256; }

// Where a pass reads (key, value) i from and writes it to.
template <typename K>
struct SplitIn {  // two arrays
  const K* keys;
  const uint32_t* vals;
  __device__ __forceinline__ K key(int64_t i) const { return keys[i]; }
  __device__ __forceinline__ void load(int64_t i, K& k, uint32_t& v) const {
    k = keys[i];
    v = vals[i];
  }
};
template <typename K>
struct SplitOut {
  K* keys;
  uint32_t* vals;
  __device__ __forceinline__ void store(int64_t o, K k, uint32_t v) const {
    keys[o] = k;
    vals[o] = v;
  }
};
struct PairIn {  // one array of 8-byte pairs
  const uint2* kv;
  __device__ __forceinline__ uint32_t key(int64_t i) const { return kv[i].x; }
  __device__ __forceinline__ void load(int64_t i, uint32_t& k, uint32_t& v) const {
    const uint2 x = kv[i];
    k = x.x;
    v = x.y;
  }
};
struct PairOut {
  uint2* kv;
  __device__ __forceinline__ void store(int64_t o, uint32_t k, uint32_t v) const { kv[o] = make_uint2(k, v); }
};
template <typename K>
struct IndexIn {  // a key's value is its index
  const K* keys;
  __device__ __forceinline__ K key(int64_t i) const { return keys[i]; }
  __device__ __forceinline__ void load(int64_t i, K& k, uint32_t& v) const {
    k = keys[i];
    v = (uint32_t)i;
  }
};
// An SML's mers (the seed's bases left-aligned, the strand in bit 0) and
// positions, where wanted.
template <typename K>
struct MersOut {
  uint64_t* mer;
  uint32_t* pos;
  int w;
  __device__ __forceinline__ void store(int64_t o, K k, uint32_t v) const {
    if (mer) mer[o] = ((uint64_t)k >> 1) << (64 - 2 * w) | ((uint64_t)k & 1);
    if (pos) pos[o] = v;
  }
};

template <typename In>
__global__ void __launch_bounds__(os::kThreads) k_rts_count(const In in, int64_t n, int shift,
                                                            uint32_t* __restrict__ counts, uint32_t* __restrict__ csum,
                                                            int64_t ctiles) {
  __shared__ uint32_t h[8][256];
  const int tid = threadIdx.x, wid = tid >> 5;
#pragma unroll
  for (int w = 0; w < 8; ++w) h[w][tid] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * os::kTile;
  uint32_t d[os::kItems];
#pragma unroll
  for (int k = 0; k < os::kItems; ++k) {
    const int64_t i = base + k * os::kThreads + tid;
    d[k] = i < n ? ((uint32_t)(in.key(i) >> shift) & 255u) : 256u;
  }
#pragma unroll
  for (int k = 0; k < os::kItems; ++k)
    if (d[k] < 256u) atomicAdd(&h[wid][d[k]], 1u);
  __syncthreads();
  uint32_t s = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) s += h[w][tid];
  counts[(int64_t)blockIdx.x * 256 + tid] = s;
  if (s) atomicAdd(&csum[((int64_t)blockIdx.x / ctiles) * 256 + tid], s);
}

// Block c, 1024 threads: thread (q, d) handles digit d for a quarter q of
// the chunk sums and a quarter of chunk c's tiles.
__global__ void k_rts_offsets(uint32_t* __restrict__ counts, int64_t ntiles, const uint32_t* __restrict__ csum,
                              int64_t ctiles, int64_t nchunks);

template <typename K, typename In, typename Out>
__global__ void __launch_bounds__(os::kThreads, sizeof(K) == 4 ? 4 : 3)
    k_rts_scatter(const In in, const Out out, int64_t n, int shift, const uint32_t* __restrict__ offsets) {
  using namespace os;
  constexpr bool kPacked = sizeof(K) == 4;  // (key, value) as one 8-byte word in shared memory
  __shared__ __align__(16) uint32_t sbuf[kPacked ? 2 * kTile : kTile * (sizeof(K) / 4 + 1)];
  __shared__ uint32_t wofs[8][256];  // per-warp digit counts, then each warp's first slot per digit
  __shared__ uint32_t gofs[256];     // output index of the tile's slot 0 for each digit
  uint2* skv = reinterpret_cast<uint2*>(sbuf);
  K* skey = reinterpret_cast<K*>(sbuf);
  uint32_t* sval = sbuf + kTile * (sizeof(K) / 4);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
#pragma unroll
  for (int w = 0; w < 8; ++w) wofs[w][tid] = 0;
  const uint32_t gbase = offsets[(int64_t)blockIdx.x * 256 + tid];
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kTile;
  const int tile_n = (int)min((int64_t)kTile, n - base);
  // warp w owns tile items [256 w, 256 w + 256): item 256 w + 32 k + lane
  K key[kItems];
  uint32_t val[kItems], rank[kItems];
  const int first = wid * 256 + lane;
  const uint32_t lt_mask = (1u << lane) - 1u;
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    const int li = first + 32 * k;
    key[k] = 0;
    val[k] = 0;
    if (li < tile_n) in.load(base + li, key[k], val[k]);
  }
  // stable rank inside the warp: earlier rounds, then lower lanes
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    const bool live = first + 32 * k < tile_n;
    const uint32_t d = (uint32_t)(key[k] >> shift) & 255u;
    uint32_t peers = __ballot_sync(0xffffffffu, live);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const uint32_t m = __ballot_sync(0xffffffffu, d >> b & 1u);
      peers &= d >> b & 1u ? m : ~m;
    }
    const uint32_t before = wofs[wid][d];
    rank[k] = before + __popc(peers & lt_mask);
    __syncwarp();
    if (live && (peers & lt_mask) == 0) wofs[wid][d] = before + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  uint32_t wpre[8], mine = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    wpre[w] = mine;
    mine += wofs[w][tid];
  }
  const uint32_t lstart = block_excl_scan256(mine, nullptr);
#pragma unroll
  for (int w = 0; w < 8; ++w) wofs[w][tid] = lstart + wpre[w];
  gofs[tid] = gbase - lstart;  // gbase >= lstart: earlier digits of this tile precede it
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    if (first + 32 * k < tile_n) {
      const uint32_t d = (uint32_t)(key[k] >> shift) & 255u;
      const uint32_t lp = wofs[wid][d] + rank[k];
      if constexpr (kPacked) {
        skv[lp] = make_uint2((uint32_t)key[k], val[k]);
      } else {
        skey[lp] = key[k];
        sval[lp] = val[k];
      }
    }
  }
  __syncthreads();
  for (int i = tid; i < tile_n; i += kThreads) {
    K k;
    uint32_t v;
    if constexpr (kPacked) {
      const uint2 kv = skv[i];
      k = (K)kv.x;
      v = kv.y;
    } else {
      k = skey[i];
      v = sval[i];
    }
    const uint32_t d = (uint32_t)(k >> shift) & 255u;
    out.store((int64_t)gofs[d] + i, k, v);
  }
}

// One pass over digit p; counted: its tile count rows and chunk sums are there.
template <typename K, typename In, typename Out>
void rts_pass(const In& in, const Out& out, int64_t n, int p, const RtsGeom& g, uint32_t* scratch, bool counted,
              cudaStream_t st, uint64_t* launches) {
  uint32_t* counts = rts_counts(scratch);
  uint32_t* cs = rts_csum(scratch, g) + (int64_t)p * g.nchunks * 256;
  if (!counted) k_rts_count<In><<<(unsigned)g.ntiles, os::kThreads, 0, st>>>(in, n, 8 * p, counts, cs, g.ctiles);
  k_rts_offsets<<<(unsigned)g.nchunks, 1024, 0, st>>>(counts, g.ntiles, cs, g.ctiles, g.nchunks);
  k_rts_scatter<K, In, Out><<<(unsigned)g.ntiles, os::kThreads, 0, st>>>(in, out, n, 8 * p, counts);
  if (launches) *launches += counted ? 2 : 3;
}

// counted: the producer of the keys already wrote the first pass's tile
// count rows and chunk sums (rts_counts, rts_csum) for tiles of os::kTile,
// and zeroed the other passes' chunk sums.
template <typename K>
int rts_sort_pairs(K* keys, uint32_t* vals, K* keys_alt, uint32_t* vals_alt, int64_t n, int nbits,
                   uint32_t* scratch, cudaStream_t st, uint64_t* launches, bool counted = false) {
  if (n <= 0) return 0;
  const RtsGeom g = rts_geom(n, nbits);
  if (!counted) cudaMemsetAsync(rts_csum(scratch, g), 0, (size_t)g.npass * g.nchunks * 256 * 4, st);
  K* k[2] = {keys, keys_alt};
  uint32_t* v[2] = {vals, vals_alt};
  for (int p = 0; p < g.npass; ++p) {
    const int a = p & 1, b = a ^ 1;
    rts_pass<K>(SplitIn<K>{k[a], v[a]}, SplitOut<K>{k[b], v[b]}, n, p, g, scratch, counted && p == 0, st, launches);
  }
  return g.npass & 1;
}

// An SML: counted keys, whose values are their indexes, to mers and
// positions.  Between passes 32-bit keys travel with their values in 8-byte
// pairs: a tile's run of a digit is 8 keys on average, which as pairs fills
// two whole sectors with one store each instead of parts of four with two.
// (3.98 million 31-bit keys, a scatter pass: 34 us in two arrays with
// ranks by __match_any_sync, 24 as pairs with ranks by eight ballots; tiles
// half as large again or twice as large are no faster.)
// keys[0] holds the keys; buf[0], buf[1]: n pairs each, or for 64-bit keys n
// values, with keys[1].
template <typename K>
void rts_sort_mers(K* const (&keys)[2], void* const (&buf)[2], int64_t n, int nbits, const MersOut<K>& out,
                   uint32_t* scratch, cudaStream_t st, uint64_t* launches) {
  const RtsGeom g = rts_geom(n, nbits);
  for (int p = 0; p < g.npass; ++p) {
    const int b = p & 1, a = b ^ 1;
    auto pass = [&](const auto& in, const auto& to) {
      rts_pass<K>(in, to, n, p, g, scratch, p == 0, st, launches);
    };
    auto from = [&](const auto& to) {
      if (p == 0)
        pass(IndexIn<K>{keys[0]}, to);
      else if constexpr (sizeof(K) == 4)
        pass(PairIn{(const uint2*)buf[a]}, to);
      else
        pass(SplitIn<K>{keys[a ^ 1], (const uint32_t*)buf[a]}, to);
    };
    if (p + 1 == g.npass)
      from(out);
    else if constexpr (sizeof(K) == 4)
      from(PairOut{(uint2*)buf[b]});
    else
      from(SplitOut<K>{keys[b ^ 1], (uint32_t*)buf[b]});
  }
}

// --------------------------------------------------- one CTA's radix sort
//
// Up to 8,192 pairs in one launch: a thread holds eight in registers, warp w
// the 256 from 256 w on; a pass ranks them as k_rts_scatter does and exchanges
// them through shared memory.  In place.  (Three launches per pass, each
// waiting for the one before, took 45 us for the 20-bit keys of a few thousand
// segments; this 12.)
constexpr int kSmallSort = 8192;
template <typename K>
constexpr size_t small_sort_smem(int warps) {
  return (size_t)warps * 256 * (sizeof(K) + 4) + (size_t)warps * 256 * 4;
}

template <typename K>
__global__ void __launch_bounds__(1024) k_small_sort(K* __restrict__ keys, uint32_t* __restrict__ vals, int n,
                                                     int npass, int dbits) {
  extern __shared__ __align__(16) uint8_t ss_smem[];
  __shared__ uint32_t wsum[8];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, warps = blockDim.x >> 5;
  K* const skey = reinterpret_cast<K*>(ss_smem);
  uint32_t* const sval = reinterpret_cast<uint32_t*>(skey + warps * 256);
  uint32_t* const wofs = sval + warps * 256;  // [warp][digit]: counts, then first slots
  const int first = wid * 256 + lane, ndig = 1 << dbits;
  const uint32_t lt_mask = (1u << lane) - 1u;
  K key[8];
  uint32_t val[8], rank[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int i = first + 32 * k;
    key[k] = i < n ? keys[i] : (K)0;
    val[k] = i < n ? vals[i] : 0u;
  }
  for (int p = 0; p < npass; ++p) {
    const int shift = p * dbits;
    for (int d = lane; d < ndig; d += 32) wofs[wid * ndig + d] = 0;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const bool live = first + 32 * k < n;
      const uint32_t d = (uint32_t)(key[k] >> shift) & (ndig - 1);
      uint32_t peers = __ballot_sync(0xffffffffu, live);
      for (int b = 0; b < dbits; ++b) {
        const uint32_t m = __ballot_sync(0xffffffffu, d >> b & 1u);
        peers &= d >> b & 1u ? m : ~m;
      }
      const uint32_t before = wofs[wid * ndig + d];
      rank[k] = before + __popc(peers & lt_mask);
      __syncwarp();
      if (live && (peers & lt_mask) == 0) wofs[wid * ndig + d] = before + __popc(peers);
      __syncwarp();
    }
    __syncthreads();
    // threads 0 .. 255: digit tid's count in every warp, then its first slots
    uint32_t total = 0, inc = 0;
    if (tid < 256) {
      if (tid < ndig)
        for (int w = 0; w < warps; ++w) total += wofs[w * ndig + tid];
      inc = warp_incl_scan(total);
      if (lane == 31) wsum[wid] = inc;
    }
    __syncthreads();
    if (tid < ndig) {
      uint32_t run = inc - total;
      for (int w = 0; w < wid; ++w) run += wsum[w];
      for (int w = 0; w < warps; ++w) {
        const uint32_t c = wofs[w * ndig + tid];
        wofs[w * ndig + tid] = run;
        run += c;
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (first + 32 * k < n) {
        const uint32_t at = wofs[wid * ndig + ((uint32_t)(key[k] >> shift) & (ndig - 1))] + rank[k];
        skey[at] = key[k];
        sval[at] = val[k];
      }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int i = first + 32 * k;
      if (i < n) {
        key[k] = skey[i];
        val[k] = sval[i];
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int i = first + 32 * k;
    if (i < n) {
      keys[i] = key[k];
      vals[i] = val[k];
    }
  }
}

// false when the device does not give it the shared memory.  Static, as its
// caller: the flags below are this file's kernels', and the local statics of a
// function with external linkage are one per process, shared with every other
// copy of the library in it.
template <typename K>
static bool small_sort_pairs(K* keys, uint32_t* vals, int n, int nbits, cudaStream_t st, uint64_t* launches) {
  static std::atomic<bool> ready[64];  // per device: the opt-in for more than 48 KB
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return false;
  if (!ready[dev]) {
    if (cudaFuncSetAttribute(k_small_sort<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)small_sort_smem<K>(32)) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    ready[dev] = true;
  }
  const int warps = n <= 2048 ? 8 : (n + 255) / 256;
  const int npass = (nbits + 7) / 8, dbits = (nbits + npass - 1) / npass;
  k_small_sort<K><<<1, 32 * warps, small_sort_smem<K>(warps), st>>>(keys, vals, n, npass, dbits);
  if (launches) *launches += 1;
  return true;
}

// The sort the workspace paths use: one CTA's for a few thousand elements,
// reduce-then-scan passes below 2^31, the older three-kernel passes above.  scratch:
// sort_scratch_words(n, nbits) words.
inline int64_t sort_scratch_words(int64_t n, int nbits) {
  const int64_t a = radix_scratch_words(n), b = rts_scratch_words(n, nbits);
  return a > b ? a : b;
}

template <typename K>
static int sort_pairs(K* keys, uint32_t* vals, K* keys_alt, uint32_t* vals_alt, int64_t n, int nbits, uint32_t* scratch,
               cudaStream_t st, uint64_t* launches, uint32_t* err) {
  (void)err;
  if (n <= 0) return 0;
  if (n <= kSmallSort && nbits > 0 && small_sort_pairs<K>(keys, vals, (int)n, nbits, st, launches)) return 0;
  if (n < (1ll << 31)) return rts_sort_pairs<K>(keys, vals, keys_alt, vals_alt, n, nbits, scratch, st, launches);
  return radix_sort_pairs<K>(keys, vals, keys_alt, vals_alt, n, nbits, scratch, st, launches);
}

}  // namespace mvg
