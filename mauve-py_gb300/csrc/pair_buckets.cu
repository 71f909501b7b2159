// The pairwise matcher's seed join by buckets: the seeds unique in each of
// the two genomes, without sorting the keys.
//
// The SearchRange merge of the two sorted mer lists (LM/MatchFinder.cpp:
// 172-340, driven by LM/PairwiseMatchFinder.cpp:37-71) hashes every mer that
// occurs exactly once in each genome.  The matcher needs the set of these
// pairs, by their position in A (match_components.cuh), not their mer order,
// so mers are dealt to buckets by a bijective mix of their bits: buckets come
// out even whatever the genomes' composition (by the mer's own top bits the
// buckets of a genome at GC 0.38 differ ten times in size).
//
//   k_pb_keys     each position's bucket (the mixed mer's top BB bits),
//                 counted: one row of counts per tile
//   k_pb_csum     per-chunk sums of the count rows
//   k_pb_scan     every bucket's start and size; chunk starts
//   k_pb_offsets  count rows -> each tile's first slot in each bucket
//   k_pb_scatter  the mers computed again (a few instructions a base; storing
//                 and reading them back moved 16 bytes a base) and (rest of
//                 the mixed mer, strand, genome; position) put into their
//                 buckets; the order inside a bucket is arbitrary
//                 (shared-memory atomics)
//   k_pb_local    one block per bucket: grouped by the next 9 bits in shared
//                 memory, then a thread per key looks for its mer in its
//                 group.  A mer with one position in each genome goes to the
//                 table: position in B, the strand relation in bit 31, at the
//                 position in A.
//   k_pb_repeats  (where there are any; match_components asks) larger buckets,
//                 which repeated mers (runs of N, tandem repeats) make, by way of a hash table of their mers; those
//                 above 8,192 keys piece by piece, each piece leaving what may
//                 be unique.  A bucket of more mers than the table holds is
//                 sorted in chunks through global memory and its runs taken.
//
// With in-bucket keys of 32 bits this takes seeds of weight up to 22 (24 M
// seeds of weight 17 in 1.06 ms, against 1.38 ms of a 64-bit radix sort
// and its runs; 9.2 M of weight 15 in 0.27 ms against 0.39 ms with stored
// keys, buckets in mer order and pairs staged in that order).  Positions are
// below 2^25 on this path (the host takes the full sort beyond that).
#include <algorithm>

#include "mvg_internal.h"
#include "prim.cuh"

namespace mvg {

namespace pb {
constexpr int kKeyThreads = 1024;
constexpr int kLocThreads = 256;
constexpr int kLocWarps = kLocThreads / 32;
constexpr int kCap = 3072;      // bucket elements sorted in shared memory
constexpr int kLocItems = kCap / kLocThreads;
constexpr int kMaxDigit = 64;   // chunked in-bucket passes: digits of at most 6 bits
constexpr int kGroups = 512;    // groups of a bucket: its top 9 in-bucket bits
constexpr int kGroupMax = 1024;  // larger groups: the bucket goes through the hash table
constexpr int kPiece = 8192;    // larger buckets: keys of a piece
constexpr int kRepeatCtas = 608;
constexpr int kProbes = 512;    // table entries looked at for a mer before the bucket is sorted instead
constexpr int kChunkTiles = 32;
constexpr uint64_t kInL2 = 96ull << 20;  // of 129 MB
}  // namespace pb

// Keys of a tile.  A tile writes its keys of a bucket as a run at the bucket's
// next slots, at random times, so the open sectors are those of all the tiles
// in flight: one CTA per SM (kOneCta), and once the keys outgrow L2, tiles of
// two keys per bucket, 38 MB of 24 million keys in flight.  Smaller tiles cost
// more count rows, larger ones leave L2 with partial sectors (24 million keys,
// 16,384 buckets: keys and scatter 0.52 ms with one key per bucket and tile,
// 0.49 with two, 0.53 with four, 0.73 with eight, 0.75 with four and two CTAs
// per SM).  Below that, eight (9.2 million: 0.15 ms, 0.18 with two).
// Tiles fill whole waves of the CTAs.
PairBucketGeom pair_bucket_geom(uint64_t n, int bits, int sms) {
  PairBucketGeom g;
  int bb = 4;
  while (bb < 14 && ((uint64_t)2048 << bb) < n) ++bb;  // about 2048 keys per bucket at most
  if (bb < bits - kPairRestBits) bb = bits - kPairRestBits;
  if (bb > bits) bb = bits;
  g.bbits = bb;
  g.nbuckets = 1 << bb;
  const uint64_t per = n * 8 <= pb::kInL2 ? 8 : 2;
  const uint64_t wave = (uint64_t)sms * std::max<uint64_t>(16384, per * g.nbuckets);
  const uint64_t waves = std::max<uint64_t>(1, (n + wave / 2) / wave);
  g.tile = (int64_t)((n / (waves * sms) + 1 + 4095) & ~4095ull);
  g.ntiles = (int64_t)((n + g.tile - 1) / g.tile);
  g.nchunks = (g.ntiles + pb::kChunkTiles - 1) / pb::kChunkTiles;
  // in-bucket key: the rest of the mixed mer, then the genome bit; an odd
  // number of passes leaves a sort's result in the scratch copy
  const int lbits = bits - bb + 1;
  int np = (lbits + 5) / 6;
  if ((np & 1) == 0) ++np;
  g.npass = np;
  g.dbits = (lbits + np - 1) / np;
  g.lbits = lbits;
  return g;
}

// ------------------------------------------------------------------ keys

// The reverse complement of a mer left-aligned in K, its strand bit set.
__device__ __forceinline__ uint32_t revcomp_in(uint32_t m, int w) { return revcomp_mer32(m, w); }
__device__ __forceinline__ uint64_t revcomp_in(uint64_t m, int w) { return revcomp_mer(m, w); }

// Calls f(mixed mers, strands, in B, first position, how many) for groups of
// up to four consecutive positions of this block's tile, made from one
// 32-base window where they fit.  K = uint32_t: w <= 15.  (A position per
// thread and call left one window load in flight per thread: the keys of 24
// million seeds of weight 17 took 0.21 ms, in groups 0.15.)
template <typename K, class F>
__device__ __forceinline__ void pb_tile(const uint32_t* __restrict__ ga, uint64_t ca, const uint32_t* __restrict__ gb,
                                        uint64_t cb, const SeedDesc& s, const K (*lut)[256], int64_t tile, F f) {
  const int nb = seed_bytes(s);
  const uint64_t n = ca + cb;
  const uint64_t base = (uint64_t)blockIdx.x * (uint64_t)tile;
  const bool quad = nb <= 7;
  const int sh = 8 * (int)sizeof(K) - 2 * s.w;
  for (int64_t o = 4 * threadIdx.x; o < tile; o += 4 * pb::kKeyThreads) {
    const uint64_t p0 = base + (uint64_t)o;
    if (p0 >= n) break;
    K m[4];
    uint32_t strand[4];
    auto take = [&](int k, K fw) {
      const K r = revcomp_in(fw, s.w), c = fw < r ? fw : r;
      m[k] = mix_mer<K>(c >> sh, 2 * s.w);
      strand[k] = (uint32_t)c & 1u;
    };
    if (quad && p0 + 4 <= n && (p0 + 4 <= ca || p0 >= ca)) {
      const bool in_b = p0 >= ca;
      const uint64_t q0 = in_b ? p0 - ca : p0;
      const uint64_t win = window64(in_b ? gb : ga, q0);
#pragma unroll
      for (int u = 0; u < 4; ++u) take(u, gather_mer<K>(win, u, lut, nb));
      f(m, strand, in_b, (uint32_t)q0, 4);
    } else {
      for (uint64_t p = p0; p < p0 + 4 && p < n; ++p) {
        const bool in_b = p >= ca;
        const uint64_t q = in_b ? p - ca : p;
        take(0, gather_mer<K>(window64(in_b ? gb : ga, q), 0, lut, nb));
        f(m, strand, in_b, (uint32_t)q, 1);
      }
    }
  }
}

template <typename K>
__device__ __forceinline__ void pb_lut(const SeedDesc& s, K (*lut)[256]) {
  if constexpr (sizeof(K) == 4)
    seed_lut_build32(s, lut);
  else
    seed_lut_build(s, lut);
}

template <typename K>
__global__ void __launch_bounds__(pb::kKeyThreads) k_pb_keys(const uint32_t* __restrict__ ga, uint64_t ca,
                                                             const uint32_t* __restrict__ gb, uint64_t cb, SeedDesc s,
                                                             uint32_t* __restrict__ counts, int bbits, int64_t tile) {
  extern __shared__ uint32_t h[];  // nbuckets counts
  __shared__ K lut[8][256];
  const int nbk = 1 << bbits, bsh = 2 * s.w - bbits;
  pb_lut(s, lut);
  for (int d = threadIdx.x; d < nbk; d += pb::kKeyThreads) h[d] = 0;
  __syncthreads();
  pb_tile<K>(ga, ca, gb, cb, s, lut, tile,
             [&](const K(&m)[4], const uint32_t(&)[4], bool, uint32_t, int count) {
#pragma unroll
               for (int u = 0; u < 4; ++u)
                 if (u < count) atomicAdd(&h[(uint32_t)(m[u] >> bsh)], 1u);
             });
  __syncthreads();
  uint32_t* row = counts + (int64_t)blockIdx.x * nbk;
  for (int d = threadIdx.x; d < nbk; d += pb::kKeyThreads) row[d] = h[d];
}

// ------------------------------------------------------- bucket offsets

// Block (x, c): buckets 256x .. 256x+255 summed over chunk c's tiles.
__global__ void __launch_bounds__(256) k_pb_csum(const uint32_t* __restrict__ counts, int64_t ntiles, int nbk,
                                                 uint32_t* __restrict__ csum) {
  const int d = blockIdx.x * 256 + threadIdx.x;
  if (d >= nbk) return;
  const int64_t c = blockIdx.y;
  const int64_t t0 = c * pb::kChunkTiles, t1 = min(ntiles, t0 + pb::kChunkTiles);
  uint32_t s = 0;
#pragma unroll 8
  for (int64_t t = t0; t < t1; ++t) s += counts[t * nbk + d];
  csum[c * nbk + d] = s;
}

// One block of 1024 threads, 16 consecutive buckets per thread (nbk <=
// 16384): every bucket's total over the chunks and its start (exclusive
// scan over buckets), and the pieces of the large ones.
__global__ void __launch_bounds__(1024) k_pb_scan(const uint32_t* __restrict__ csum, int64_t nchunks, int nbk,
                                                  uint32_t* __restrict__ bstart, uint32_t* __restrict__ bsize,
                                                  PairPieces P) {
  constexpr int kPer = 16;
  __shared__ uint32_t wsum[32], npieces;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (tid == 0) npieces = 0;
  const int d0 = tid * kPer;
  uint32_t tot[kPer];
#pragma unroll
  for (int k = 0; k < kPer; ++k) tot[k] = 0;
  if (d0 < nbk) {
#pragma unroll 4
    for (int64_t c = 0; c < nchunks; ++c) {
      const uint4* q = reinterpret_cast<const uint4*>(csum + c * nbk + d0);
#pragma unroll
      for (int k = 0; k < kPer / 4; ++k) {
        const uint4 v = q[k];
        tot[4 * k] += v.x;
        tot[4 * k + 1] += v.y;
        tot[4 * k + 2] += v.z;
        tot[4 * k + 3] += v.w;
      }
    }
  }
  uint32_t mine = 0;
#pragma unroll
  for (int k = 0; k < kPer; ++k) mine += tot[k];
  const uint32_t inc = warp_incl_scan(mine);
  if (lane == 31) wsum[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    const uint32_t x = wsum[lane];
    const uint32_t y = warp_incl_scan(x);
    wsum[lane] = y - x;
  }
  __syncthreads();
  uint32_t start = wsum[wid] + inc - mine;
#pragma unroll
  for (int k = 0; k < kPer; k += 4) {  // 16 bytes at a time: nbk is a multiple of 4, both arrays aligned
    if (d0 + k >= nbk) break;
    const uint32_t s1 = start + tot[k], s2 = s1 + tot[k + 1], s3 = s2 + tot[k + 2];
    *reinterpret_cast<uint4*>(bstart + d0 + k) = make_uint4(start, s1, s2, s3);
    *reinterpret_cast<uint4*>(bsize + d0 + k) = make_uint4(tot[k], tot[k + 1], tot[k + 2], tot[k + 3]);
    start = s3 + tot[k + 3];
  }
#pragma unroll
  for (int k = 0; k < kPer; ++k)
    if (d0 + k < nbk && tot[k] > (uint32_t)pb::kPiece) {
      const uint32_t m = (tot[k] + pb::kPiece - 1) / pb::kPiece, at = atomicAdd(&npieces, m);
      for (uint32_t q = 0; q < m; ++q) P.piece[at + q] = make_uint4((uint32_t)(d0 + k), q, at, m);
      P.left[at] = make_uint2(0u, 0u);
    }
  __syncthreads();
  if (tid == 0) *P.count = npieces;
}

// Block (x, c): chunk c's tiles' first slots per bucket (offs): the
// bucket's start plus the earlier chunks' sums, then the chunk's count rows
// (all loads issued before any store).
__global__ void __launch_bounds__(256) k_pb_offsets(const uint32_t* __restrict__ counts, int64_t ntiles, int nbk,
                                                    const uint32_t* __restrict__ csum,
                                                    const uint32_t* __restrict__ bstart, uint32_t* __restrict__ offs) {
  const int d = blockIdx.x * 256 + threadIdx.x;
  if (d >= nbk) return;
  const int64_t c = blockIdx.y;
  const int64_t t0 = c * pb::kChunkTiles;
  const int nt = (int)min((int64_t)pb::kChunkTiles, ntiles - t0);
  uint32_t v[pb::kChunkTiles];
#pragma unroll
  for (int k = 0; k < pb::kChunkTiles; ++k) v[k] = k < nt ? counts[(t0 + k) * nbk + d] : 0u;
  uint32_t run = bstart[d];
  for (int64_t cc = 0; cc < c; ++cc) run += csum[cc * nbk + d];
#pragma unroll
  for (int k = 0; k < pb::kChunkTiles; ++k) {
    if (k < nt) offs[(t0 + k) * nbk + d] = run;
    run += v[k];
  }
}

// Exclusive scan of n <= 16384 counts by one block of 1024 threads (16
// consecutive counts each); *total gets the sum.
__global__ void __launch_bounds__(1024) k_pb_scan_small(const uint32_t* __restrict__ in, int n,
                                                        uint32_t* __restrict__ out, uint32_t* __restrict__ total) {
  constexpr int kPer = 16;
  __shared__ uint32_t wsum[32];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int i0 = tid * kPer;
  uint32_t v[kPer], mine = 0;
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    v[k] = i0 + k < n ? in[i0 + k] : 0u;
    mine += v[k];
  }
  const uint32_t inc = warp_incl_scan(mine);
  if (lane == 31) wsum[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    const uint32_t x = wsum[lane];
    const uint32_t y = warp_incl_scan(x);
    wsum[lane] = y - x;
    if (lane == 31 && total) *total = y;
  }
  __syncthreads();
  uint32_t r = wsum[wid] + inc - mine;
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    if (i0 + k < n) out[i0 + k] = r;
    r += v[k];
  }
}

void pair_scan_small(const uint32_t* in, int n, uint32_t* out, uint32_t* total, cudaStream_t st) {
  k_pb_scan_small<<<1, 1024, 0, st>>>(in, n, out, total);
}

// ------------------------------------------------------------- scatter

template <typename K>
__global__ void __launch_bounds__(pb::kKeyThreads) k_pb_scatter(const uint32_t* __restrict__ ga, uint64_t ca,
                                                                const uint32_t* __restrict__ gb, uint64_t cb, SeedDesc s,
                                                                const uint32_t* __restrict__ offsets, int bbits,
                                                                int64_t tile, uint2* __restrict__ out) {
  extern __shared__ uint32_t cur[];  // next free slot per bucket
  __shared__ K lut[8][256];
  const int nbk = 1 << bbits, bsh = 2 * s.w - bbits;
  const uint32_t rest = (uint32_t)(((uint64_t)1 << bsh) - 1);
  const uint32_t* row = offsets + (int64_t)blockIdx.x * nbk;
  pb_lut(s, lut);
  for (int d = threadIdx.x; d < nbk; d += pb::kKeyThreads) cur[d] = row[d];
  __syncthreads();
  pb_tile<K>(ga, ca, gb, cb, s, lut, tile,
             [&](const K(&m)[4], const uint32_t(&strand)[4], bool in_b, uint32_t q, int count) {
               uint32_t slot[4];
#pragma unroll
               for (int u = 0; u < 4; ++u)
                 if (u < count) slot[u] = atomicAdd(&cur[(uint32_t)(m[u] >> bsh)], 1u);
#pragma unroll
               for (int u = 0; u < 4; ++u)
                 if (u < count)
                   out[slot[u]] = make_uint2(((uint32_t)m[u] & rest) << 2 | strand[u] << 1 | (in_b ? 1u : 0u), q + u);
             });
}

// ------------------------------------------- buckets of repeated mers

// A mer of a bucket: x the mer, with its positions in A (0, 1, or 2 for more)
// in bits 31:30; y its position in B and strand (bit 31), kNone before one was
// seen, kMany after two.  Free entries have all bits set, as no x or y has:
// there is no count 3, and no position of 31 bits.
constexpr uint32_t kNone = 0xffffffffu, kMany = 0xfffffffeu;

__device__ __forceinline__ uint32_t table_at(uint32_t mer, uint32_t entries) {
  return __umulhi(mer * 0x9E3779B1u, entries);
}

// Counts a key; false: no room for its mer.  Entries only ever gain, and a mer
// seen too often is left alone, so a run of one mer costs two shared reads a
// key.
__device__ __forceinline__ bool table_add(uint2* T, uint32_t entries, uint2 key) {
  const uint32_t mer = key.x >> 2, one = key.x & 1u ? 0u : 1u << 30;
  uint32_t i = table_at(mer, entries);
  for (int probe = 0; probe < pb::kProbes; ++probe) {
    uint32_t x = *(volatile uint32_t*)&T[i].x;
    bool made = false;
    if (x == kNone) {
      x = atomicCAS(&T[i].x, kNone, mer | one);
      made = x == kNone;
    }
    if (made || (x & 0x3fffffffu) == mer) {
      if (one) {
        while (!made && x >> 31 == 0) {  // counted none or one so far
          const uint32_t was = atomicCAS(&T[i].x, x, x + one);
          made = was == x;
          x = was;
        }
      } else {
        uint32_t y = *(volatile uint32_t*)&T[i].y;
        if (y == kNone) y = atomicCAS(&T[i].y, kNone, key.y | (key.x >> 1 & 1u) << 31);
        if (y != kNone && y != kMany) *(volatile uint32_t*)&T[i].y = kMany;
      }
      return true;
    }
    if (++i == entries) i = 0;
  }
  return false;
}

// The entry of a mer that was counted.
__device__ __forceinline__ uint2 table_find(const uint2* T, uint32_t entries, uint32_t mer) {
  uint32_t i = table_at(mer, entries);
  while ((T[i].x & 0x3fffffffu) != mer) i = i + 1 == entries ? 0 : i + 1;
  return T[i];
}

// v[0, n) counted in an emptied table, by the block; false: too many mers.
__device__ bool table_fill(uint2* T, uint32_t entries, const uint2* v, int n) {
  constexpr int kAhead = 4;
  for (uint32_t i = threadIdx.x; i < entries; i += pb::kLocThreads) T[i] = make_uint2(kNone, kNone);
  __syncthreads();
  bool ok = true;
  for (int i0 = threadIdx.x; i0 < n && ok; i0 += kAhead * pb::kLocThreads) {
    uint2 key[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k)
      if (i0 + k * pb::kLocThreads < n) key[k] = v[i0 + k * pb::kLocThreads];
#pragma unroll
    for (int k = 0; k < kAhead; ++k)
      if (i0 + k * pb::kLocThreads < n) ok = table_add(T, entries, key[k]) && ok;
  }
  return !__syncthreads_or(!ok);
}

// The pairs of v[0, n) by way of the table; false: too many mers.
__device__ __noinline__ bool table_pairs(uint2* T, uint32_t entries, const uint2* v, int n, uint32_t* __restrict__ tab) {
  if (!table_fill(T, entries, v, n)) return false;
#pragma unroll 4
  for (int i = threadIdx.x; i < n; i += pb::kLocThreads) {
    const uint2 key = v[i];
    if (key.x & 1u) continue;  // a pair's position in A
    const uint2 e = table_find(T, entries, key.x >> 2);
    if (e.x >> 30 == 1u && e.y != kNone && e.y != kMany)
      tab[key.y] = (e.y & 0x7fffffffu) | ((key.x >> 1 & 1u) ^ e.y >> 31) << 31;
  }
  return true;
}

// What may be unique of the piece v[0, n), appended to the bucket's list: the
// keys of mers with one position at most in either genome, and two keys in A
// for every other mer, so that it stays out.  left: the list's length (bit 31:
// it is not the whole bucket) and the pieces done.
__device__ __noinline__ void table_thin(uint2* T, uint32_t entries, const uint2* v, int n, uint2* list, uint2* left) {
  const int lane = threadIdx.x & 31;
  if (!table_fill(T, entries, v, n)) {
    if (threadIdx.x == 0) atomicOr(&left->x, 1u << 31);
    return;
  }
  auto append = [&](bool in, uint2 key) {
    const unsigned all = __ballot_sync(0xffffffffu, in);
    uint32_t at = 0;
    if (lane == 0 && all) at = atomicAdd(&left->x, (uint32_t)__popc(all));
    at = (__shfl_sync(0xffffffffu, at, 0) & 0x7fffffffu) + __popc(all & ((1u << lane) - 1u));
    if (in) list[at] = key;
  };
  for (int i0 = threadIdx.x & ~31; i0 < n; i0 += pb::kLocThreads) {
    const int i = i0 + lane;
    uint2 key = make_uint2(0u, 0u);
    bool in = i < n;
    if (in) {
      key = v[i];
      const uint2 e = table_find(T, entries, key.x >> 2);
      in = e.x >> 31 == 0 && e.y != kMany;
    }
    append(in, key);
  }
  for (uint32_t i0 = threadIdx.x & ~31; i0 < entries; i0 += pb::kLocThreads) {
    const uint2 e = i0 + lane < entries ? T[i0 + lane] : make_uint2(kNone, kNone);
    const bool many = e.x != kNone && (e.x >> 31 || e.y == kMany);
    const uint2 key = make_uint2((e.x & 0x3fffffffu) << 2, 0u);
    append(many, key);
    append(many, key);
  }
}

// ---------------------------------------------------- in-bucket sort

struct LocalSmem {
  uint32_t whist[pb::kLocWarps][pb::kMaxDigit];   // per-warp digit counts, then each warp's first slot
  uint32_t run[pb::kMaxDigit];                    // chunked sort: slots used so far by each digit
  uint32_t dstart[pb::kMaxDigit];                 // chunked sort: each digit's first slot in the bucket
};

// In-bucket key: the rest of the mixed mer, then the genome bit.
__device__ __forceinline__ uint32_t pb_lkey(uint32_t key, int lbits) {
  return (((key >> 2) << 1) | (key & 1u)) & ((1u << lbits) - 1u);
}

// Stable rank of up to kLocItems * 32 items per warp: warp w takes items
// [w * rounds * 32, (w + 1) * rounds * 32) of src[0, n) in order, counting
// its digits in S.whist[w].  Items past n get private digits.
__device__ __forceinline__ void pb_rank(const uint2* src, int n, int rounds, int shift, uint32_t mask, int lbits,
                                        LocalSmem& S, uint2 (&item)[pb::kLocItems],
                                        uint32_t (&rank)[pb::kLocItems]) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t lt_mask = (1u << lane) - 1u;
  const int wbase = wid * rounds * 32;
#pragma unroll
  for (int k = 0; k < pb::kLocItems; ++k) {
    if (k < rounds) {
      const int li = wbase + k * 32 + lane;
      uint32_t d;
      if (li < n) {
        item[k] = src[li];
        d = (pb_lkey(item[k].x, lbits) >> shift) & mask;
      } else {
        item[k] = make_uint2(0u, 0u);
        d = 0x10000u + (uint32_t)lane;  // private digit: shares no rank
      }
      const uint32_t peers = __match_any_sync(0xffffffffu, d);
      const uint32_t before = d < 0x10000u ? S.whist[wid][d] : 0u;
      rank[k] = before + __popc(peers & lt_mask);
      __syncwarp();
      if (d < 0x10000u && (peers & lt_mask) == 0) S.whist[wid][d] = before + __popc(peers);
      __syncwarp();
    }
  }
}

// One stable LSD pass over a bucket too large for shared memory: src and
// dst in global memory, chunks of kCap elements in order, digits of up to 6
// bits.
__device__ void pb_pass_chunked(const uint2* src, uint2* dst, int n, int shift, uint32_t mask, int lbits,
                                LocalSmem& S) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int ndig = (int)mask + 1;
  if (tid < pb::kMaxDigit) {
    S.run[tid] = 0;
    S.dstart[tid] = 0;
  }
  __syncthreads();
  for (int i = tid; i < n; i += pb::kLocThreads) atomicAdd(&S.dstart[(pb_lkey(src[i].x, lbits) >> shift) & mask], 1u);
  __syncthreads();
  if (wid == 0) {  // exclusive scan of at most 64 counts by one warp
    const uint32_t a = lane < ndig ? S.dstart[lane] : 0u, b = lane + 32 < ndig ? S.dstart[lane + 32] : 0u;
    const uint32_t ia = warp_incl_scan(a), ib = warp_incl_scan(b);
    const uint32_t ta = __shfl_sync(0xffffffffu, ia, 31);
    if (lane < ndig) S.dstart[lane] = ia - a;
    if (lane + 32 < ndig) S.dstart[lane + 32] = ta + ib - b;
  }
  __syncthreads();
  for (int c0 = 0; c0 < n; c0 += pb::kCap) {
    const int cn = min(pb::kCap, n - c0);
    const int rounds = (cn + pb::kLocThreads - 1) / pb::kLocThreads;
    for (int d = lane; d < ndig; d += 32) S.whist[wid][d] = 0;
    __syncwarp();
    uint2 item[pb::kLocItems];
    uint32_t rank[pb::kLocItems];
    pb_rank(src + c0, cn, rounds, shift, mask, lbits, S, item, rank);
    __syncthreads();
    if (tid < ndig) {  // per digit: the warps' first slots in this chunk
      uint32_t r = S.dstart[tid] + S.run[tid];
#pragma unroll
      for (int w = 0; w < pb::kLocWarps; ++w) {
        const uint32_t x = S.whist[w][tid];
        S.whist[w][tid] = r;
        r += x;
      }
      S.run[tid] = r - S.dstart[tid];
    }
    __syncthreads();
    const int wbase = wid * rounds * 32;
#pragma unroll
    for (int k = 0; k < pb::kLocItems; ++k)
      if (k < rounds && wbase + k * 32 + lane < cn)
        dst[S.whist[wid][(pb_lkey(item[k].x, lbits) >> shift) & mask] + rank[k]] = item[k];
    __syncthreads();
  }
}

// Runs of the sorted bucket v[0, n): element i opens a pair when it and
// i + 1 hold the same mer from different genomes and neither i - 1 nor
// i + 2 holds that mer.
__device__ void pb_pairs(const uint2* v, int n, uint32_t* __restrict__ tab) {
  for (int i = threadIdx.x; i + 1 < n; i += pb::kLocThreads) {
    const uint32_t k0 = v[i].x, k1 = v[i + 1].x, m = k0 >> 2;  // key >> 2: the mer
    if ((k1 >> 2) != m || ((k0 ^ k1) & 1u) == 0) continue;
    if (i > 0 && (v[i - 1].x >> 2) == m) continue;
    if (i + 2 < n && (v[i + 2].x >> 2) == m) continue;
    const uint32_t p0 = v[i].y, p1 = v[i + 1].y;
    // SetDirection (LM/MemHash.cpp:189-207): B is reversed relative to A
    // when the two occurrences have different strand bits
    tab[k0 & 1u ? p1 : p0] = (k0 & 1u ? p0 : p1) | (((k0 ^ k1) >> 1) & 1u) << 31;
  }
}

// A bucket sorted in chunks between its region of `buf` (g) and the same region
// of `alt` (h) in an odd number of passes of up to 6 bits, which leaves it in
// `alt`, and its runs.
__device__ __noinline__ void pb_sort(uint2* g, uint2* h, int n, int lbits, int npass, int dbits, LocalSmem& S,
                                     uint32_t* __restrict__ tab) {
  const uint32_t mask = (1u << dbits) - 1u;
  const uint2* src = g;
  uint2* dst = h;
  for (int p = 0; p < npass; ++p) {
    pb_pass_chunked(src, dst, n, p * dbits, mask, lbits, S);
    uint2* t = (uint2*)src;
    src = dst;
    dst = t;
  }
  pb_pairs(src, n, tab);  // npass is odd: the sorted bucket is in alt
}

// Block b finds the unique pairs of bucket b.  A bucket of at most cap
// (<= kCap) keys is split in shared memory by its top in-bucket bits (up to
// 9) into at most 512 groups of a few keys each (atomics place a group's keys
// in any order).  Then one thread per key of A: a key whose mer occurs
// exactly twice in its group, once per genome, is a pair.  A repeated mer's keys
// have seen enough after its third, so a group may hold hundreds of one.  Other
// buckets, and one with a group of more than kGroupMax keys, are left to
// k_pb_repeats: that costs the call 40 us, which a bacterial genome should not
// pay for a mer of 260 positions.
// Loads and shared-memory round trips bound it: six CTAs per SM take 0.21 ms for
// 24 million keys and 0.081 for 9.2, three (80 registers) took 0.30 and 0.112.
__global__ void __launch_bounds__(pb::kLocThreads, 6) k_pb_local(const uint2* __restrict__ buf,
                                                              const uint32_t* __restrict__ bstart,
                                                              const uint32_t* __restrict__ bsize, int lbits, int cap,
                                                              PairPieces P, uint32_t* __restrict__ tab) {
  extern __shared__ __align__(16) uint2 sbuf[];  // kCap elements
  __shared__ uint32_t gcnt[pb::kGroups], gbeg[pb::kGroups], gcur[pb::kGroups];
  const int tid = threadIdx.x;
  const int b = blockIdx.x;
  const int n = (int)bsize[b];
  const uint2* g = buf + bstart[b];
  if (n > pb::kPiece) return;  // in pieces
  bool rest = n > cap;
  if (!rest) {
    // group bits: mer bits only (never the genome bit), at most 9
    const int hbits = lbits - 1 < 9 ? lbits - 1 : 9, lo = lbits - hbits, ng = 1 << hbits;
    for (int d = tid; d < pb::kGroups; d += pb::kLocThreads) gcnt[d] = 0;
    __syncthreads();
    uint2 item[pb::kLocItems];
#pragma unroll
    for (int k = 0; k < pb::kLocItems; ++k) {
      const int i = k * pb::kLocThreads + tid;
      if (i < n) {
        item[k] = g[i];
        atomicAdd(&gcnt[pb_lkey(item[k].x, lbits) >> lo], 1u);
      }
    }
    __syncthreads();
    // thread t: groups 2t and 2t + 1
    const int d0 = 2 * tid;
    const uint32_t c0 = d0 < ng ? gcnt[d0] : 0u, c1 = d0 + 1 < ng ? gcnt[d0 + 1] : 0u;
    const uint32_t st = block_excl_scan256(c0 + c1, nullptr);
    if (d0 < ng) gbeg[d0] = gcur[d0] = st;
    if (d0 + 1 < ng) gbeg[d0 + 1] = gcur[d0 + 1] = st + c0;
    rest = __syncthreads_or(c0 > (uint32_t)pb::kGroupMax || c1 > (uint32_t)pb::kGroupMax);
    if (!rest) {
#pragma unroll
      for (int k = 0; k < pb::kLocItems; ++k)
        if (k * pb::kLocThreads + tid < n) sbuf[atomicAdd(&gcur[pb_lkey(item[k].x, lbits) >> lo], 1u)] = item[k];
      __syncthreads();
      for (int i = tid; i < n; i += pb::kLocThreads) {
        const uint32_t x = sbuf[i].x;
        if (x & 1u) continue;  // the A occurrence of each pair
        const int d = (int)(pb_lkey(x, lbits) >> lo), e0 = (int)gbeg[d], e1 = e0 + (int)gcnt[d];
        int cnt = 0, other = 0;
        for (int j = e0; j < e1 && cnt < 3; ++j)
          if (((sbuf[j].x ^ x) >> 2) == 0) {
            ++cnt;
            if (j != i) other = j;
          }
        if (cnt == 2 && (sbuf[other].x & 1u)) {
          // SetDirection (LM/MemHash.cpp:189-207): B is reversed relative
          // to A when the two occurrences have different strand bits
          const uint2 y = sbuf[other];
          tab[sbuf[i].y] = y.y | (((x ^ y.x) >> 1) & 1u) << 31;
        }
      }
    }
  }
  if (rest && tid == 0) {
    const uint32_t at = atomicAdd(P.count, 1u);
    P.piece[at] = make_uint4((uint32_t)b, 0u, at, 0u);
  }
}

// The buckets in P, a block at a time: whole ones (no pieces), or pieces, of
// which whoever does a bucket's last looks for the pairs in what they left.
// (Sorted by one block each, a bucket of 600,000 equal mers took 6 ms, one of
// the 2 million of a run of N 24.)
__global__ void __launch_bounds__(pb::kLocThreads) k_pb_repeats(uint2* __restrict__ buf, uint2* __restrict__ alt,
                                                                const uint32_t* __restrict__ bstart,
                                                                const uint32_t* __restrict__ bsize, int lbits,
                                                                int npass, int dbits, int cap, PairPieces P,
                                                                uint32_t* __restrict__ tab) {
  extern __shared__ __align__(16) uint2 sbuf[];  // kCap elements
  __shared__ LocalSmem S;
  __shared__ uint32_t done;
  const uint32_t total = *P.count;
  for (uint32_t w = blockIdx.x; w < total; w += gridDim.x) {
    const uint4 piece = P.piece[w];  // bucket, number, the bucket's first, their number
    const int size = (int)bsize[piece.x];
    uint2 *const v = buf + bstart[piece.x], *const list = alt + bstart[piece.x];
    __syncthreads();  // the last bucket's table is read
    const uint2* rest = v;
    int m = size;
    if (piece.w > 0) {
      const int at = (int)piece.y * pb::kPiece;
      uint2* const left = P.left + piece.z;
      table_thin(sbuf, (uint32_t)cap, v + at, min(pb::kPiece, size - at), list, left);
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0) done = atomicAdd(&left->y, 1u);
      __syncthreads();
      if (done + 1 < piece.w) continue;
      __threadfence();  // all pieces are in the list
      rest = list;
      m = (int)*(volatile uint32_t*)&left->x;
    }
    if (m < 0 || !table_pairs(sbuf, (uint32_t)cap, rest, m, tab)) pb_sort(v, list, size, lbits, npass, dbits, S, tab);
  }
}

// ------------------------------------------------------------------ host

int pair_bucket_bufs(Ctx* c, uint64_t n, int bits, PairBucketBufs* b) {
  int sms = 0;
  MVG_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device));
  b->g = pair_bucket_geom(n, bits, sms);
  const PairBucketGeom& g = b->g;
  const int nbk = g.nbuckets;
  Workspace& ws = c->ws;
  b->alt = (uint2*)ws.get(c, 30, (size_t)n * 8 + 64);
  b->buf = (uint2*)ws.get(c, 31, (size_t)n * 8 + 64);
  // count rows, then the tiles' first slots (ntiles x nbk each)
  b->counts = (uint32_t*)ws.get(c, 32, (size_t)g.ntiles * nbk * 8 + 64);
  // chunk sums, bucket starts and sizes; the pieces of large buckets (at most
  // two per kPiece keys) and the buckets k_pb_local leaves: their list, what is
  // left of the bucket of each, their number
  const size_t tab_words = ((size_t)g.nchunks * nbk + 2 * (size_t)nbk + 67) & ~(size_t)3;
  const size_t most = 2 * (n / pb::kPiece) + 2 + nbk;
  uint32_t* tabs = (uint32_t*)ws.get(c, 33, tab_words * 4 + most * 24 + 16);
  if (!b->alt || !b->buf || !b->counts || !tabs) return report_error(MVG_ERR_NOMEM, "workspace allocation failed");
  b->offs = b->counts + (size_t)g.ntiles * nbk;
  b->csum = tabs;
  b->bstart = tabs + (size_t)g.nchunks * nbk;
  b->bsize = b->bstart + nbk;
  b->pieces.piece = (uint4*)(tabs + tab_words);
  b->pieces.left = (uint2*)(b->pieces.piece + most);
  b->pieces.count = (uint32_t*)(b->pieces.left + most);
  return 0;
}

void pair_bucket_offsets(Ctx* c, const PairBucketBufs& b) {
  const PairBucketGeom& g = b.g;
  const dim3 grid2((unsigned)((g.nbuckets + 255) / 256), (unsigned)g.nchunks);
  k_pb_csum<<<grid2, 256, 0, c->stream>>>(b.counts, g.ntiles, g.nbuckets, b.csum);
  k_pb_scan<<<1, 1024, 0, c->stream>>>(b.csum, g.nchunks, g.nbuckets, b.bstart, b.bsize, b.pieces);
  k_pb_offsets<<<grid2, 256, 0, c->stream>>>(b.counts, g.ntiles, g.nbuckets, b.csum, b.bstart, b.offs);
  c->launches += 3;
}

void pair_bucket_join(Ctx* c, const PairBucketBufs& b, uint32_t* tab) {
  const PairBucketGeom& g = b.g;
  const int cap = std::min(c->pair_bucket_cap, pb::kCap);
  const size_t smem = pb::kCap * sizeof(uint2);
  k_pb_local<<<(unsigned)g.nbuckets, pb::kLocThreads, smem, c->stream>>>(b.buf, b.bstart, b.bsize, g.lbits, cap,
                                                                         b.pieces, tab);
  c->launches++;
}

void pair_bucket_repeats(Ctx* c, const PairBucketBufs& b, uint32_t* tab) {
  const PairBucketGeom& g = b.g;
  const int cap = std::min(c->pair_bucket_cap, pb::kCap);
  k_pb_repeats<<<pb::kRepeatCtas, pb::kLocThreads, pb::kCap * sizeof(uint2), c->stream>>>(
      b.buf, b.alt, b.bstart, b.bsize, g.lbits, g.npass, g.dbits, cap, b.pieces, tab);
  c->launches++;
}

template <typename K>
static int pair_buckets_as(Ctx* c, const uint32_t* ga, uint64_t ca, const uint32_t* gb, uint64_t cb, const SeedDesc& s,
                           uint32_t* tab, PairBucketBufs& b) {
  if (int rc = pair_bucket_bufs(c, ca + cb, 2 * s.w, &b)) return rc;
  const PairBucketGeom& g = b.g;
  bool& ready = c->join_ready[sizeof(K) == 8];
  if (!ready) {  // more than 48 KB of dynamic shared memory
    MVG_CUDA_TRY(cudaFuncSetAttribute(k_pb_keys<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (16384 + 64) * 4));
    MVG_CUDA_TRY(cudaFuncSetAttribute(k_pb_scatter<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, kOneCta));
    ready = true;
  }
  const size_t hsm = (size_t)g.nbuckets * 4;
  k_pb_keys<K><<<(unsigned)g.ntiles, pb::kKeyThreads, hsm, c->stream>>>(ga, ca, gb, cb, s, b.counts, g.bbits, g.tile);
  pair_bucket_offsets(c, b);
  stage_mark(c, "seed_scatter");
  k_pb_scatter<K><<<(unsigned)g.ntiles, pb::kKeyThreads, kOneCta, c->stream>>>(ga, ca, gb, cb, s, b.offs, g.bbits, g.tile,
                                                                           b.buf);
  c->launches += 2;
  stage_mark(c, "seed_local");
  pair_bucket_join(c, b, tab);
  MVG_CUDA_TRY(cudaGetLastError());
  return 0;
}

int pair_buckets(Ctx* c, const uint32_t* ga, uint64_t ca, const uint32_t* gb, uint64_t cb, const SeedDesc& s,
                 uint32_t* tab, PairBucketBufs* b) {
  return s.w <= 15 ? pair_buckets_as<uint32_t>(c, ga, ca, gb, cb, s, tab, *b)
                   : pair_buckets_as<uint64_t>(c, ga, ca, gb, cb, s, tab, *b);
}

}  // namespace mvg

extern "C" int mvg_set_pair_bucket_cap(mvg_handle h, int cap) {
  using namespace mvg;
  if (!h || cap < 32 || cap > pb::kCap) return report_error(MVG_ERR_ARG, "cap must be in 32..3072");
  reinterpret_cast<Ctx*>(h)->pair_bucket_cap = cap;
  return 0;
}
