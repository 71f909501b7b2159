// Genome -> reference index LUT on the GPU.
//
// Construction from aligned blocks follows mauve/buildindex.py:112-130: per
// block, each side's index starts at start-1 and advances on a non-gap
// character; a column whose two characters are equal writes
// lut[genome_idx] = ref_idx when genome_idx < n (genome_idx == -1 wraps to
// n-1 as a numpy index does).  Later blocks and later columns overwrite
// earlier ones.
//
//   k_lut_count    non-gap counts of both rows per tile of 4,096 columns, and
//                  up to each block's first column within its tile
//   k_tile_scan    exclusive prefix over the tiles
//   k_lut_walk     per-column indices; each write is an atomicMax of
//                  ((column+1) << 32 | value) so the last writer in column
//                  order wins
//   k_lut_finish   keys -> int32 LUT (-1 where unwritten)
//
// fillGaps / smoothEdges / findGaps (mauve/indexutils.pyx:47-139) run
// sequentially in place in the reference.  Their decisions depend only on
// the LUT as it was before the pass, except that a fill [g-1, u] hides every
// later gap start inside (g, u] (see the proof in k_fill_resolve).  So:
//
//   k_fill_count     gap starts of the unmodified LUT per tile of 4,096 (and
//                    fixZeroIdx, which only the first gap start depends on)
//   k_tile_scan      exclusive prefix over the tiles
//   k_fill_search    gap starts in order, each with its first partner u in
//                    (g, g+width]
//   k_fill_heads     gap starts that no earlier start's reach covers are
//                    certain
//   k_fill_apply     each certain start walks its cluster forward and writes
//                    the performed fills
//
// All of it is queued without a look at the device in between: counts stay
// there, and a stage that meets an error leaves it in the error word, which
// the later stages test.  (Flags, scans and candidates as separate passes
// over the LUT, 35 launches and nine waits, took 396 us for 4.6 million
// bases in 64 blocks; this takes 189.)
#include "mvg_internal.h"
#include "prim.cuh"

namespace mvg {
namespace {

constexpr int kTile = 4096;  // columns, or LUT entries, per tile
constexpr int kLutThreads = 256;
constexpr int kGroups = kTile / 16;  // a thread's 16 consecutive columns

// Whether the error word is set, the same for all of the CTA's threads: CTAs of
// the same launch may set it at any time.
__device__ __forceinline__ bool cta_failed(const uint32_t* err) {
  return __syncthreads_or(err && threadIdx.x == 0 && *(const volatile uint32_t*)err);
}

// ------------------------------------------------------------ construction

// Sixteen characters from p, `have` of them readable (0 for the rest).
__device__ __forceinline__ uint4 load16(const uint8_t* __restrict__ p, int have) {
  if (have >= 16 && ((uintptr_t)p & 15) == 0) return *reinterpret_cast<const uint4*>(p);
  uint32_t w[4] = {0, 0, 0, 0};
  for (int k = 0; k < 16 && k < have; ++k) w[k >> 2] |= (uint32_t)p[k] << (8 * (k & 3));
  return make_uint4(w[0], w[1], w[2], w[3]);
}
// Bit k: byte k of v is set (v's bytes are 0 or 0xff).
__device__ __forceinline__ uint32_t byte_mask(uint32_t v) {
  return ((v & 0x08040201u) * 0x01010101u) >> 24;
}

struct Group {
  uint32_t bases;  // non-gap columns of the genome's row, of the reference's << 16
  uint32_t same;   // columns whose two characters are equal
};
// The group's columns [c, c + 16), cut at c1.
__device__ __forceinline__ Group load_group(const uint8_t* __restrict__ g, const uint8_t* __restrict__ r, uint64_t c,
                                            uint64_t c1) {
  Group o{0, 0};
  if (c >= c1) return o;
  const int have = c1 - c < 16 ? (int)(c1 - c) : 16;
  const uint4 x = load16(g + c, have), y = load16(r + c, have);
  const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
  uint32_t bg = 0, br = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    bg |= byte_mask(__vcmpne4(xs[k], 0x2d2d2d2du)) << (4 * k);
    br |= byte_mask(__vcmpne4(ys[k], 0x2d2d2d2du)) << (4 * k);
    o.same |= byte_mask(__vcmpeq4(xs[k], ys[k])) << (4 * k);
  }
  const uint32_t in = have < 16 ? (1u << have) - 1u : 0xffffu;
  o.bases = (bg & in) | (br & in) << 16;
  o.same &= in;
  return o;
}
__device__ __forceinline__ uint32_t group_counts(uint32_t bases) {
  return (uint32_t)__popc(bases & 0xffffu) | (uint32_t)__popc(bases >> 16) << 16;
}

// First index b in [0, n] with off[b] >= v (any offsets: stays in range).
__device__ __forceinline__ uint64_t lower_block(const uint64_t* __restrict__ off, uint64_t n, uint64_t v) {
  uint64_t lo = 0, hi = n;
  while (lo < hi) {
    const uint64_t m = (lo + hi) / 2;
    if (off[m] < v) lo = m + 1;
    else hi = m;
  }
  return lo;
}

// Tile t is columns [col_off[0] + 4096 t, + 4096).  tile: non-gap counts of
// the genome's row [0, ntiles), of the reference's [ntiles, 2 ntiles);
// blk[b]: both (reference << 16) in block b's tile before its first column.
__global__ void __launch_bounds__(kLutThreads) k_lut_count(const uint8_t* __restrict__ g, const uint8_t* __restrict__ r,
                                                           const uint64_t* __restrict__ col_off, uint64_t nblocks,
                                                           uint32_t ntiles, uint32_t* __restrict__ tile,
                                                           uint32_t* __restrict__ blk, uint32_t* err) {
  __shared__ uint32_t s_ex[kGroups], s_bases[kGroups], s_tot;
  const uint64_t t0 = col_off[0] + (uint64_t)blockIdx.x * kTile;
  const uint64_t end = col_off[nblocks], t1 = t0 + kTile < end ? t0 + kTile : end;
  for (uint64_t b = (uint64_t)blockIdx.x * kLutThreads + threadIdx.x; b < nblocks; b += (uint64_t)ntiles * kLutThreads)
    if (col_off[b + 1] < col_off[b]) set_error(err, kDevRange);
  const Group x = load_group(g, r, t0 + threadIdx.x * 16, t1);
  const uint32_t ex = block_excl_scan256(group_counts(x.bases), &s_tot);
  s_ex[threadIdx.x] = ex;
  s_bases[threadIdx.x] = x.bases;
  __syncthreads();
  if (threadIdx.x == 0) {
    tile[blockIdx.x] = s_tot & 0xffffu;
    tile[ntiles + blockIdx.x] = s_tot >> 16;
  }
  const uint64_t b1 = lower_block(col_off, nblocks, t1);
  for (uint64_t b = lower_block(col_off, nblocks, t0) + threadIdx.x; b < b1; b += kLutThreads) {
    const uint64_t at = col_off[b] - t0;
    if (at >= kTile) continue;  // offsets that decrease: reported above
    const uint32_t before = (1u << (at & 15)) - 1u;
    blk[b] = s_ex[at >> 4] + group_counts(s_bases[at >> 4] & (before | before << 16));
  }
}

// Exclusive prefix of n values in place (blockIdx.x: which of the arrays, n
// apart), their sum to total[blockIdx.x].
__global__ void __launch_bounds__(1024) k_tile_scan(uint32_t* __restrict__ v, int64_t n, uint32_t* __restrict__ total) {
  __shared__ uint32_t wsum[32];
  uint32_t* const a = v + (int64_t)blockIdx.x * n;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t carry = 0;
  for (int64_t c = 0; c < n; c += 4096) {
    uint32_t x[4], sum = 0;
    const int64_t i = c + threadIdx.x * 4;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      x[k] = i + k < n ? a[i + k] : 0u;
      sum += x[k];
    }
    const uint32_t inc = warp_incl_scan(sum);
    if (lane == 31) wsum[wid] = inc;
    __syncthreads();
    const uint32_t w = warp_incl_scan(wsum[lane]);
    uint32_t run = carry + inc - sum + (wid ? __shfl_sync(0xffffffffu, w, wid - 1) : 0u);
    carry += __shfl_sync(0xffffffffu, w, 31);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (i + k < n) a[i + k] = run;
      run += x[k];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0 && total) total[blockIdx.x] = carry;
}

// Per column: indices after this column, and the keyed write, consecutive
// threads on consecutive columns.
__global__ void __launch_bounds__(kLutThreads) k_lut_walk(const uint8_t* __restrict__ g, const uint8_t* __restrict__ r,
                                                          const uint64_t* __restrict__ col_off, uint64_t nblocks,
                                                          uint32_t ntiles, const uint32_t* __restrict__ tile,
                                                          const uint32_t* __restrict__ blk,
                                                          const int64_t* __restrict__ g_start,
                                                          const int64_t* __restrict__ r_start, int64_t n,
                                                          unsigned long long* __restrict__ keys, uint32_t* err) {
  __shared__ uint32_t s_ex[kGroups], s_bases[kGroups], s_same[kGroups];
  if (cta_failed(err)) return;  // offsets that decrease
  const uint64_t first = col_off[0], t0 = first + (uint64_t)blockIdx.x * kTile;
  const uint64_t end = col_off[nblocks], t1 = t0 + kTile < end ? t0 + kTile : end;
  const Group x = load_group(g, r, t0 + threadIdx.x * 16, t1);
  const uint32_t ex = block_excl_scan256(group_counts(x.bases), nullptr);
  s_ex[threadIdx.x] = ex;
  s_bases[threadIdx.x] = x.bases;
  s_same[threadIdx.x] = x.same;
  __syncthreads();
  const uint32_t pg = tile[blockIdx.x], pr = tile[ntiles + blockIdx.x];
  // the blocks of the tile's first and last column
  const uint64_t b0 = lower_block(col_off, nblocks, t0 + 1) - 1, b1 = lower_block(col_off, nblocks, t1) - 1;
  uint64_t b = ~0ull;
  int64_t g0 = 0, r0 = 0;  // index before the tile's first column, were it the block's
  for (uint64_t c = t0 + threadIdx.x; c < t1; c += kLutThreads) {
    const uint32_t at = (uint32_t)(c - t0), k = at >> 4, bit = at & 15;
    if (!(s_same[k] >> bit & 1)) continue;
    const uint64_t bc = b0 == b1 ? b0 : b0 + lower_block(col_off + b0, b1 + 1 - b0, c + 1) - 1;
    if (bc != b) {
      b = bc;
      const uint32_t tb = (uint32_t)((col_off[b] - first) / kTile), part = blk[b];
      g0 = g_start[b] - 1 - (int64_t)(part & 0xffffu);
      r0 = r_start[b] - 1 - (int64_t)(part >> 16);
      g0 += (int64_t)(uint32_t)(pg - tile[tb]);
      r0 += (int64_t)(uint32_t)(pr - tile[ntiles + tb]);
    }
    const uint32_t upto = (2u << bit) - 1u;
    const uint32_t cnt = s_ex[k] + group_counts(s_bases[k] & (upto | upto << 16));
    const int64_t gi = g0 + (int64_t)(cnt & 0xffffu), ri = r0 + (int64_t)(cnt >> 16);
    if (gi >= n) continue;
    const int64_t t = gi < 0 ? gi + n : gi;
    if (t < 0) {
      set_error(err, kDevRange);
      continue;
    }
    if (ri < INT32_MIN || ri > INT32_MAX) {
      set_error(err, kDevOverflow);
      continue;
    }
    const unsigned long long key = ((unsigned long long)(c + 1) << 32) | (uint32_t)(int32_t)ri;
    atomicMax(keys + t, key);
  }
}

__global__ void k_lut_finish(const unsigned long long* __restrict__ keys, int64_t n, int32_t* __restrict__ lut) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const unsigned long long k = keys[i];
    lut[i] = k ? (int32_t)(uint32_t)k : -1;
  }
}

// ------------------------------------------------------------ fixZeroIdx

// mauve/indexutils.pyx:27-44: if lut[0] == -1, the first index nx >= 10
// with lut[nx] != -1 gives ref_idx = lut[nx] - nx; lut[0] = ref_idx when
// ref_idx >= 0 and genome[0] == ref[ref_idx].  The Cython loop reads lut[nx]
// for every nx up to that index with bounds checks, so no such index (or a
// LUT of at most 10 entries) is an IndexError, as are an empty genome and
// ref_idx past the reference.  One CTA scans 256 indices per step.
struct ZeroFix {
  const uint8_t* genome;
  const uint8_t* ref;
  uint64_t glen, rlen;
  int on;
};
__device__ void fix_zero(int32_t* lut, int64_t n, const ZeroFix& z, uint32_t* err) {
  const uint8_t *const genome = z.genome, *const ref = z.ref;
  const uint64_t glen = z.glen, rlen = z.rlen;
  if (lut[0] != -1) return;
  __shared__ int64_t found;
  if (threadIdx.x == 0) found = -1;
  __syncthreads();
  for (int64_t base = 10; base < n; base += 256) {
    const int64_t i = base + threadIdx.x;
    const bool hit = i < n && lut[i] != -1;
    const int any = __syncthreads_or(hit);
    if (any) {
      // lowest hitting index: one pass over the warps' ballots
      const unsigned bal = __ballot_sync(0xffffffffu, hit);
      __shared__ unsigned wb[8];
      if ((threadIdx.x & 31) == 0) wb[threadIdx.x >> 5] = bal;
      __syncthreads();
      if (threadIdx.x == 0) {
        for (int w = 0; w < 8; ++w)
          if (wb[w]) {
            found = base + w * 32 + __ffs(wb[w]) - 1;
            break;
          }
      }
      __syncthreads();
      break;
    }
  }
  if (threadIdx.x != 0) return;
  if (found < 0) {
    set_error(err, kDevRange);
    return;
  }
  const int32_t ref_idx = (int32_t)((uint32_t)lut[found] - (uint32_t)found);
  if (ref_idx > -1) {
    if (glen == 0 || (uint64_t)ref_idx >= rlen) {
      set_error(err, kDevRange);
      return;
    }
    if (genome[0] == ref[ref_idx]) lut[0] = ref_idx;
  }
}

// ------------------------------------------------ fillGaps / smoothEdges

__global__ void __launch_bounds__(256) k_fix_zero(int32_t* lut, int64_t n, const ZeroFix z, uint32_t* err) {
  fix_zero(lut, n, z, err);
}

enum FillMode : int { kFill = 0, kSmooth = 1 };

__device__ __forceinline__ bool gap_start(int32_t lo, int32_t m, int mode) {  // of lut[i - 1], lut[i]
  if (lo == -1) return false;
  return mode == kSmooth ? m != (int32_t)((uint32_t)lo + 1u) : m == -1;
}

// A tile's gap starts: thread t of step j looks at entry 256 j + t (m[j]; the
// entry before it lo[j]), and s_at[8 j + warp] gets the tile's gap starts
// before that warp's.  Returns their number.
__device__ __forceinline__ uint32_t tile_starts(const int32_t (&lo)[kTile / 256], const int32_t (&m)[kTile / 256],
                                                int64_t n, int mode, int64_t t0, unsigned (&ball)[kTile / 256],
                                                uint32_t* s_at) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int j = 0; j < kTile / 256; ++j) {
    const int64_t i = t0 + 256 * j + threadIdx.x;
    ball[j] = __ballot_sync(0xffffffffu, i > 0 && i < n && gap_start(lo[j], m[j], mode));
    if (lane == 0) s_at[8 * j + wid] = __popc(ball[j]);
  }
  __syncthreads();
  const uint32_t v = threadIdx.x < kTile / 32 ? s_at[threadIdx.x] : 0u;
  __shared__ uint32_t total;
  const uint32_t ex = block_excl_scan256(v, &total);
  if (threadIdx.x < kTile / 32) s_at[threadIdx.x] = ex;
  __syncthreads();
  return total;
}

// The first CTA looks after fixZeroIdx: no other reads lut[0].  err may be null.
__global__ void __launch_bounds__(256) k_fill_count(int32_t* lut, int64_t n, int mode, const ZeroFix z,
                                                    uint32_t* __restrict__ tile, uint32_t* err) {
  __shared__ uint32_t s_at[kTile / 32];
  if (cta_failed(err)) return;
  if (z.on && blockIdx.x == 0) {
    fix_zero(lut, n, z, err);
    __syncthreads();
  }
  const int64_t t0 = (int64_t)blockIdx.x * kTile;
  int32_t lo[kTile / 256], m[kTile / 256];
#pragma unroll
  for (int j = 0; j < kTile / 256; ++j) {
    const int64_t i = t0 + 256 * j + threadIdx.x;
    m[j] = i < n ? lut[i] : 0;
    lo[j] = __shfl_up_sync(0xffffffffu, m[j], 1);
    if ((threadIdx.x & 31) == 0 && i > 0 && i < n) lo[j] = lut[i - 1];
  }
  unsigned ball[kTile / 256];
  const uint32_t count = tile_starts(lo, m, n, mode, t0, ball, s_at);
  if (threadIdx.x == 0) tile[blockIdx.x] = count;
}

// Gap starts g (lower = g-1, L = lut[lower]) in order, and the first u in
// g+1 .. min(n-1, g+width) with lut[u] - L == u - lower (int32 arithmetic),
// reach = u, or g when there is none.  The tile is in shared memory, its gap
// starts are listed there, and a thread per gap start tries the next eight
// entries (a substitution's partner is the next one); what is left the warp
// searches together.  (From global memory, a thread per
// entry: 36 us for 4.6 million entries that are not in L2; this takes 16.)
__global__ void __launch_bounds__(256) k_fill_search(const int32_t* __restrict__ lut, int64_t n, int width, int mode,
                                                     const uint32_t* __restrict__ tile, int32_t* __restrict__ cand,
                                                     int32_t* __restrict__ reach, int32_t* __restrict__ lval,
                                                     const uint32_t* err) {
  constexpr int kProbe = 8, kAhead = 8;
  __shared__ uint32_t s_at[kTile / 32];
  __shared__ int32_t s_lut[kTile + 1 + kProbe];  // entries t0 - 1 ..
  __shared__ uint16_t s_start[kTile];
  if (err && *(const volatile uint32_t*)err) return;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t t0 = (int64_t)blockIdx.x * kTile;
  int32_t lo[kTile / 256], m[kTile / 256];
#pragma unroll
  for (int j = 0; j < kTile / 256; ++j) {
    const int64_t i = t0 + 256 * j + threadIdx.x;
    m[j] = i < n ? lut[i] : 0;
  }
  if (threadIdx.x <= kProbe) {
    const int64_t i = threadIdx.x == 0 ? t0 - 1 : t0 + kTile + threadIdx.x - 1;
    s_lut[threadIdx.x == 0 ? 0 : kTile + threadIdx.x] = i >= 0 && i < n ? lut[i] : 0;
  }
#pragma unroll
  for (int j = 0; j < kTile / 256; ++j) s_lut[1 + 256 * j + threadIdx.x] = m[j];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kTile / 256; ++j) lo[j] = s_lut[256 * j + threadIdx.x];
  unsigned ball[kTile / 256];
  const int count = (int)tile_starts(lo, m, n, mode, t0, ball, s_at);
#pragma unroll
  for (int j = 0; j < kTile / 256; ++j)
    if (ball[j] >> lane & 1)
      s_start[s_at[8 * j + wid] + __popc(ball[j] & ((1u << lane) - 1u))] = (uint16_t)(256 * j + threadIdx.x);
  __syncthreads();
  const uint32_t first = tile[blockIdx.x];
  for (int k0 = wid * 32; k0 < count; k0 += 256) {
    const int k = k0 + lane;
    bool open = k < count;
    const int q = open ? s_start[k] : 0;
    const int64_t gs = t0 + q;
    const int32_t L = s_lut[q];
    if (open) {
      cand[first + k] = (int32_t)gs;
      lval[first + k] = L;
      // entries gs + 1 .. last that this thread tries
      const int64_t last = gs + width < n - 1 ? gs + width : n - 1;
      const int tries = last - gs < kProbe ? (int)(last - gs) : kProbe;
      int32_t u = (int32_t)gs;
      for (int d = 1; d <= tries; ++d)
        if ((int32_t)((uint32_t)s_lut[q + 1 + d] - (uint32_t)L) == d + 1) {
          u = (int32_t)gs + d;
          open = false;
          break;
        }
      open = open && last - gs > kProbe;
      reach[first + k] = u;
    }
    for (unsigned left = __ballot_sync(0xffffffffu, open); left; left &= left - 1) {
      const int src = __ffs(left) - 1;
      const int64_t g0 = t0 + __shfl_sync(0xffffffffu, q, src), l0 = g0 - 1;
      const int64_t end = g0 + width < n - 1 ? g0 + width : n - 1;
      const int32_t L0 = __shfl_sync(0xffffffffu, L, src);
      // 32 entries, then 256 at a time
      auto partner = [&](int64_t up) {
        return up <= end && (int32_t)((uint32_t)lut[up] - (uint32_t)L0) == (int32_t)(up - l0);
      };
      int64_t base = g0 + 1 + kProbe;
      unsigned hit = __ballot_sync(0xffffffffu, partner(base + lane));
      for (base += 32; !hit && base <= end;) {
        bool is[kAhead];
#pragma unroll
        for (int k = 0; k < kAhead; ++k) is[k] = partner(base + 32 * k + lane);
#pragma unroll
        for (int k = 0; k < kAhead; ++k)
          if (!hit) {
            hit = __ballot_sync(0xffffffffu, is[k]);
            base += 32;
          }
      }
      if (hit && lane == 0) reach[first + k0 + src] = (int32_t)(base - 32 + __ffs(hit) - 1);
    }
  }
}

// Sequential semantics, restated: a fill from gap start g rewrites
// [g-1, u]; afterwards every position in (g, u] continues the run, so no
// gap start of the unmodified LUT inside (g, u] is one any more, while the
// value at u (the old lut[u]) and everything after u are untouched.  Hence
// a gap start is performed iff no PERFORMED earlier start reaches it, and
// the search of a performed start sees the unmodified LUT.  A start that no
// earlier start reaches at all (performed or not) is certainly performed:
// it heads a cluster.  Its thread walks the cluster: from a performed start
// the next performed one is the first start beyond its reach; the walk ends
// at the next cluster head.  A start is a head where the largest reach before
// it is below it; reach(g) <= g + width bounds how far back that looks.
__global__ void __launch_bounds__(256) k_fill_heads(const int32_t* __restrict__ cand, const int32_t* __restrict__ reach,
                                                    const uint32_t* __restrict__ ncand_p, int width,
                                                    uint8_t* __restrict__ head, const uint32_t* err) {
  __shared__ int32_t s_warp[8];
  if (err && *(const volatile uint32_t*)err) return;
  const int64_t ncand = *ncand_p;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int64_t c0 = (int64_t)blockIdx.x * 1024; c0 < ncand; c0 += (int64_t)gridDim.x * 1024) {
    // the largest reach before this chunk
    int32_t far = -1;
    const int64_t g0 = cand[c0];
    for (int64_t j = c0 - 1 - threadIdx.x; j >= 0 && (int64_t)cand[j] + width >= g0; j -= 256) far = max(far, reach[j]);
    far = __reduce_max_sync(0xffffffffu, far);
    if (lane == 0) s_warp[wid] = far;
    __syncthreads();
    far = -1;
#pragma unroll
    for (int w = 0; w < 8; ++w) far = max(far, s_warp[w]);
    __syncthreads();
    // four consecutive starts per thread
    const int64_t k0 = c0 + threadIdx.x * 4;
    int32_t g[4], r[4], mx = -1;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const bool in = k0 + k < ncand;
      g[k] = in ? cand[k0 + k] : 0;
      r[k] = in ? reach[k0 + k] : -1;
      mx = max(mx, r[k]);
    }
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int32_t v = __shfl_up_sync(0xffffffffu, mx, d);
      if (lane >= d) mx = max(mx, v);
    }
    if (lane == 31) s_warp[wid] = mx;
    mx = __shfl_up_sync(0xffffffffu, mx, 1);
    if (lane == 0) mx = -1;
    __syncthreads();
    for (int w = 0; w < wid; ++w) mx = max(mx, s_warp[w]);
    mx = max(mx, far);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k0 + k < ncand) head[k0 + k] = mx < g[k];
      mx = max(mx, r[k]);
    }
    __syncthreads();
  }
}

// A thread per certain start walks its cluster.  A performed start with a
// partner writes lut[g-1+t] = L + t for t = 0 .. u-(g-1), runs of more than 32
// with the warp.  Adjacent performed fills share at most their end position,
// where both write the same value.  gaps (findGaps) gets u-(g-1), or -1 for a
// performed start with no partner.
__global__ void __launch_bounds__(256) k_fill_apply(int32_t* __restrict__ lut, const int32_t* __restrict__ cand,
                                                    const int32_t* __restrict__ reach,
                                                    const int32_t* __restrict__ lval,
                                                    const uint8_t* __restrict__ head,
                                                    const uint32_t* __restrict__ ncand_p, int32_t* __restrict__ gaps,
                                                    const uint32_t* err) {
  if (err && *(const volatile uint32_t*)err) return;
  const int64_t ncand = *ncand_p;
  const int lane = threadIdx.x & 31;
  for (int64_t k0 = (int64_t)blockIdx.x * 256 + (threadIdx.x & ~31); k0 < ncand; k0 += (int64_t)gridDim.x * 256) {
    int64_t cur = k0 + lane;
    bool on = cur < ncand && head[cur];
    while (__any_sync(0xffffffffu, on)) {
      int32_t u = 0, L = 0;
      int64_t gs = 0;
      bool long_run = false;
      if (on) {
        gs = cand[cur];
        u = reach[cur];
        L = lval[cur];
        if (u == gs) {
          if (gaps) gaps[gs] = -1;
        } else {
          if (gaps) gaps[gs] = (int32_t)(u - (gs - 1));
          long_run = u - gs > 31;
          if (!long_run)
            for (int32_t t = 0; t <= (int32_t)(u - (gs - 1)); ++t) lut[gs - 1 + t] = (int32_t)((uint32_t)L + (uint32_t)t);
        }
        // the next performed start of the cluster
        int64_t nx = cur + 1;
        while (nx < ncand && cand[nx] <= u) ++nx;
        on = nx < ncand && !head[nx];
        cur = nx;
      }
      for (unsigned left = __ballot_sync(0xffffffffu, long_run); left; left &= left - 1) {
        const int src = __ffs(left) - 1;
        const int64_t l0 = __shfl_sync(0xffffffffu, gs, src) - 1;
        const int32_t u0 = __shfl_sync(0xffffffffu, u, src), L0 = __shfl_sync(0xffffffffu, L, src);
        for (int64_t t = lane; t <= u0 - l0; t += 32) lut[l0 + t] = (int32_t)((uint32_t)L0 + (uint32_t)t);
      }
    }
  }
}

// ------------------------------------------------------------ analysis

__global__ void k_find_edges(const int32_t* __restrict__ lut, int64_t n, uint8_t* __restrict__ edges) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    edges[i] = i == 0 ? 1 : ((uint32_t)lut[i] - (uint32_t)lut[i - 1] != 1u);
}

__global__ void k_find_mismatches(const int32_t* __restrict__ lut, int64_t n, const uint8_t* __restrict__ genome,
                                  int64_t glen, const uint8_t* __restrict__ ref, int64_t rlen,
                                  uint8_t* __restrict__ mism, uint32_t* err) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    uint8_t v = 0;
    if (i < glen) {
      const int32_t m = lut[i];
      if (m != -1) {
        if (m < 0 || m >= rlen)
          set_error(err, kDevRange);
        else
          v = genome[i] != ref[m];
      }
    }
    mism[i] = v;
  }
}

__global__ void k_lut_max(const int32_t* __restrict__ lut, int64_t n, int* __restrict__ mx) {
  int m = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    m = max(m, lut[i]);
  for (int d = 16; d > 0; d >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, d));
  if ((threadIdx.x & 31) == 0) atomicMax(mx, m);
}

__global__ void k_lut_hist(const int32_t* __restrict__ lut, int64_t n, uint32_t* __restrict__ counts) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    atomicAdd(counts + (lut[i] < 0 ? 0 : lut[i]), 1u);
}

__global__ void k_count_dups(const uint32_t* __restrict__ counts, int64_t nc, unsigned long long* __restrict__ dup) {
  unsigned long long d = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nc; i += (int64_t)gridDim.x * blockDim.x)
    d += counts[i] > 1;
  for (int q = 16; q > 0; q >>= 1) d += __shfl_xor_sync(0xffffffffu, d, q);
  if ((threadIdx.x & 31) == 0 && d) atomicAdd(dup, d);
}

}  // namespace

// Workspace slots of this file.
enum : int {
  kWsTile = 70, kWsBlock, kWsFillTile, kWsKeys, kWsCand, kWsReach, kWsLval, kWsHead, kWsCounts, kWsMeta,
  // host-API staging
  kWsHLut, kWsHAux, kWsHGenome, kWsHRef, kWsHRowG, kWsHRowR, kWsHStarts, kWsHOff
};
static_assert(kWsHOff < Workspace::kSlots, "workspace slots");

static uint32_t* wsu32(Ctx* c, int slot, uint64_t n) { return (uint32_t*)c->ws.get(c, slot, n * 4 + 16); }

// Host reads of small device scalars through the pinned mirror.
static int read_u32(Ctx* c, const uint32_t* d, uint32_t* out) {
  MVG_CUDA_TRY(cudaMemcpyAsync(c->h_scalars, d, 4, cudaMemcpyDeviceToHost, c->stream));
  MVG_CUDA_TRY(cudaStreamSynchronize(c->stream));
  *out = (uint32_t)(c->h_scalars[0] & 0xffffffffu);
  return 0;
}

// Queues the LUT's construction from the columns [first, end) of the rows;
// errors go to c->d_err, which is cleared first.
static int lut_from_blocks_queue(Ctx* c, const int64_t* d_gs, const int64_t* d_rs, const uint64_t* d_off,
                                 const uint8_t* d_g, const uint8_t* d_r, uint64_t nblocks, uint64_t first,
                                 uint64_t end, int32_t* d_lut, int64_t n) {
  cudaStream_t st = c->stream;
  MVG_CUDA_TRY(cudaMemsetAsync(c->d_err, 0, 4, st));
  unsigned long long* keys = (unsigned long long*)c->ws.get(c, kWsKeys, (size_t)n * 8 + 16);
  if (!keys) return report_error(MVG_ERR_NOMEM, "LUT key allocation failed");
  if (n > 0) MVG_CUDA_TRY(cudaMemsetAsync(keys, 0, (size_t)n * 8, st));
  if (nblocks > 0 && end > first) {
    const uint32_t ntiles = (uint32_t)((end - first + kTile - 1) / kTile);
    uint32_t* tile = wsu32(c, kWsTile, 2 * (uint64_t)ntiles);
    uint32_t* blk = wsu32(c, kWsBlock, nblocks);
    if (!tile || !blk) return report_error(MVG_ERR_NOMEM, "LUT tile allocation failed");
    k_lut_count<<<ntiles, kLutThreads, 0, st>>>(d_g, d_r, d_off, nblocks, ntiles, tile, blk, c->d_err);
    k_tile_scan<<<2, 1024, 0, st>>>(tile, ntiles, nullptr);
    k_lut_walk<<<ntiles, kLutThreads, 0, st>>>(d_g, d_r, d_off, nblocks, ntiles, tile, blk, d_gs, d_rs, n, keys,
                                               c->d_err);
    c->launches += 3;
  }
  if (n > 0) {
    k_lut_finish<<<grid_for((uint64_t)n, 256), 256, 0, st>>>(keys, n, d_lut);
    c->launches++;
  }
  MVG_CUDA_TRY(cudaGetLastError());
  return 0;
}

int lut_fix_zero_dev(Ctx* c, int32_t* d_lut, int64_t n, const uint8_t* d_genome, uint64_t glen,
                     const uint8_t* d_ref, uint64_t rlen) {
  if (n <= 0) return report_error(MVG_ERR_RANGE, "fixZeroIdx: empty LUT");
  MVG_CUDA_TRY(cudaMemsetAsync(c->d_err, 0, 4, c->stream));
  k_fix_zero<<<1, 256, 0, c->stream>>>(d_lut, n, ZeroFix{d_genome, d_ref, glen, rlen, 1}, c->d_err);
  c->launches++;
  MVG_CUDA_TRY(cudaGetLastError());
  return check_device_error(c);
}

// Queues one fillGaps / smoothEdges / findGaps pass after fixZeroIdx (z.on).
// err: the error word whose errors turn the pass off, or null.
static int lut_fill_queue(Ctx* c, int32_t* d_lut, int64_t n, int width, int mode, int32_t* d_gaps, const ZeroFix& z,
                          uint32_t* err) {
  cudaStream_t st = c->stream;
  if (d_gaps && n > 0) MVG_CUDA_TRY(cudaMemsetAsync(d_gaps, 0, (size_t)n * 4, st));
  if (n < 2 || width < 1) {  // the reference loops never find a partner
    if (z.on) {
      k_fix_zero<<<1, 256, 0, st>>>(d_lut, n, z, err);
      c->launches++;
      MVG_CUDA_TRY(cudaGetLastError());
    }
    return 0;
  }
  const unsigned ntiles = (unsigned)((n + kTile - 1) / kTile);
  uint32_t* tile = wsu32(c, kWsFillTile, (uint64_t)ntiles + 1);
  int32_t* cand = (int32_t*)wsu32(c, kWsCand, n);
  int32_t* reach = (int32_t*)wsu32(c, kWsReach, n);
  int32_t* lval = (int32_t*)wsu32(c, kWsLval, n);
  uint8_t* head = (uint8_t*)c->ws.get(c, kWsHead, n + 16);
  if (!tile || !cand || !reach || !lval || !head) return report_error(MVG_ERR_NOMEM, "LUT fill allocation failed");
  uint32_t* count = tile + ntiles;
  const int grid = grid_for((uint64_t)n / 4 + 1, 256);
  k_fill_count<<<ntiles, 256, 0, st>>>(d_lut, n, mode, z, tile, err);
  k_tile_scan<<<1, 1024, 0, st>>>(tile, ntiles, count);
  k_fill_search<<<ntiles, 256, 0, st>>>(d_lut, n, width, mode, tile, cand, reach, lval, err);
  k_fill_heads<<<grid, 256, 0, st>>>(cand, reach, count, width, head, err);
  k_fill_apply<<<grid, 256, 0, st>>>(d_lut, cand, reach, lval, head, count, d_gaps, err);
  c->launches += 5;
  MVG_CUDA_TRY(cudaGetLastError());
  return 0;
}

// like every entry point, returns once the LUT is final (callers read it on
// other streams)
int lut_fill_dev(Ctx* c, int32_t* d_lut, int64_t n, int width, int mode, int32_t* d_gaps) {
  if (int rc = lut_fill_queue(c, d_lut, n, width, mode, d_gaps, ZeroFix{}, nullptr)) return rc;
  MVG_CUDA_TRY(cudaStreamSynchronize(c->stream));
  return 0;
}

int lut_find_edges_dev(Ctx* c, const int32_t* d_lut, int64_t n, uint8_t* d_edges) {
  if (n <= 0) return 0;
  k_find_edges<<<grid_for((uint64_t)n, 256), 256, 0, c->stream>>>(d_lut, n, d_edges);
  c->launches++;
  MVG_CUDA_TRY(cudaGetLastError());
  MVG_CUDA_TRY(cudaStreamSynchronize(c->stream));
  return 0;
}

int lut_find_mismatches_dev(Ctx* c, const int32_t* d_lut, int64_t n, const uint8_t* d_genome, uint64_t glen,
                            const uint8_t* d_ref, uint64_t rlen, uint8_t* d_mism) {
  if (glen > (uint64_t)n) return report_error(MVG_ERR_RANGE, "findMismatches: genome longer than the LUT");
  if (n <= 0) return 0;
  MVG_CUDA_TRY(cudaMemsetAsync(c->d_err, 0, 4, c->stream));
  k_find_mismatches<<<grid_for((uint64_t)n, 256), 256, 0, c->stream>>>(d_lut, n, d_genome, (int64_t)glen, d_ref,
                                                                      (int64_t)rlen, d_mism, c->d_err);
  c->launches++;
  MVG_CUDA_TRY(cudaGetLastError());
  return check_device_error(c);
}

int lut_duplicate_mappings_dev(Ctx* c, const int32_t* d_lut, int64_t n, int64_t* result) {
  if (n <= 0) {
    *result = -1;
    return 0;
  }
  cudaStream_t st = c->stream;
  uint32_t* meta = wsu32(c, kWsMeta, 8);
  if (!meta) return report_error(MVG_ERR_NOMEM, "allocation failed");
  MVG_CUDA_TRY(cudaMemsetAsync(meta, 0, 32, st));
  k_lut_max<<<grid_for((uint64_t)n, 256), 256, 0, st>>>(d_lut, n, (int*)meta);
  c->launches++;
  uint32_t mx = 0;
  if (int rc = read_u32(c, meta, &mx)) return rc;
  const int64_t nc = (int64_t)mx + 1;
  uint32_t* counts = wsu32(c, kWsCounts, (uint64_t)nc);
  if (!counts) return report_error(MVG_ERR_NOMEM, "allocation failed");
  MVG_CUDA_TRY(cudaMemsetAsync(counts, 0, (size_t)nc * 4, st));
  unsigned long long* dup = (unsigned long long*)(meta + 2);
  k_lut_hist<<<grid_for((uint64_t)n, 256), 256, 0, st>>>(d_lut, n, counts);
  k_count_dups<<<grid_for((uint64_t)nc, 256), 256, 0, st>>>(counts, nc, dup);
  c->launches += 2;
  MVG_CUDA_TRY(cudaMemcpyAsync(c->h_scalars, dup, 8, cudaMemcpyDeviceToHost, st));
  MVG_CUDA_TRY(cudaStreamSynchronize(st));
  *result = (int64_t)c->h_scalars[0] - 1;
  return 0;
}

}  // namespace mvg

// ------------------------------------------------------------------ C ABI

using namespace mvg;

namespace {

Ctx* ctx_of(mvg_handle h) { return reinterpret_cast<Ctx*>(h); }

// Host buffer -> workspace slot (async on the handle's stream).
template <typename T>
T* stage_in(Ctx* c, int slot, const T* host, uint64_t count) {
  T* d = (T*)c->ws.get(c, slot, count * sizeof(T) + 16);
  if (d && count) {
    if (cudaMemcpyAsync(d, host, count * sizeof(T), cudaMemcpyHostToDevice, c->stream) != cudaSuccess) return nullptr;
  }
  return d;
}

int finish_out(Ctx* c, void* host, const void* dev, size_t bytes) {
  if (bytes) MVG_CUDA_TRY(cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, c->stream));
  MVG_CUDA_TRY(cudaStreamSynchronize(c->stream));
  return 0;
}

int check_lut_len(uint64_t n) {
  if (n > (uint64_t)INT32_MAX) return report_error(MVG_ERR_CAPACITY, "LUT longer than 2^31-1 entries");
  return 0;
}

int queue_blocks(Ctx* c, const int64_t* d_gs, const int64_t* d_rs, const uint64_t* d_off, const uint8_t* d_g,
               const uint8_t* d_r, uint64_t nblocks, uint64_t first, uint64_t end, int32_t* d_lut, uint64_t n) {
  if (int rc = check_lut_len(n)) return rc;
  if (end >= 0xffffffffull) return report_error(MVG_ERR_CAPACITY, "more than 2^32-2 alignment columns");
  return lut_from_blocks_queue(c, d_gs, d_rs, d_off, d_g, d_r, nblocks, first, end, d_lut, (int64_t)n);
}

// buildIndex's passes over a LUT whose construction is queued, and the wait
// for them.
int index_passes(Ctx* c, int32_t* d_lut, int64_t n, const ZeroFix& zero, int fill_gaps, int max_gap_width,
                 int smooth_edges, int smoothing_radius) {
  if (fill_gaps) {
    if (n <= 0) {
      if (int rc = check_device_error(c)) return rc;
      return report_error(MVG_ERR_RANGE, "fixZeroIdx: empty LUT");
    }
    if (int rc = lut_fill_queue(c, d_lut, n, max_gap_width, kFill, nullptr, zero, c->d_err)) return rc;
  }
  if (smooth_edges)
    if (int rc = lut_fill_queue(c, d_lut, n, smoothing_radius, kSmooth, nullptr, ZeroFix{}, c->d_err)) return rc;
  return check_device_error(c);
}

// First and last column offset of blocks on the device.
int read_cols(Ctx* c, const uint64_t* d_col_off, uint64_t nblocks, const uint8_t* d_g, const uint8_t* d_r,
              uint64_t* first, uint64_t* end) {
  *first = *end = 0;
  if (!nblocks) return 0;
  MVG_CUDA_TRY(cudaMemcpyAsync(c->h_scalars, d_col_off, 8, cudaMemcpyDeviceToHost, c->stream));
  MVG_CUDA_TRY(cudaMemcpyAsync(c->h_scalars + 1, d_col_off + nblocks, 8, cudaMemcpyDeviceToHost, c->stream));
  MVG_CUDA_TRY(cudaStreamSynchronize(c->stream));
  *first = c->h_scalars[0];
  *end = c->h_scalars[1];
  if (*end < *first) return report_error(MVG_ERR_ARG, "column offsets decrease");
  if (*end && (!d_g || !d_r)) return report_error(MVG_ERR_ARG, "bad argument");
  return 0;
}

}  // namespace

extern "C" {

int mvg_lut_from_blocks_dev(mvg_handle h, const int64_t* d_genome_start, const int64_t* d_ref_start,
                            const uint64_t* d_col_off, const uint8_t* d_genome_rows, const uint8_t* d_ref_rows,
                            uint64_t nblocks, int32_t* d_lut, uint64_t n) {
  if (!h || (nblocks && (!d_genome_start || !d_ref_start || !d_col_off)) || (n && !d_lut))
    return report_error(MVG_ERR_ARG, "bad argument");
  Ctx* c = ctx_of(h);
  MVG_CUDA_TRY(cudaSetDevice(c->device));
  uint64_t first, end;
  if (int rc = read_cols(c, d_col_off, nblocks, d_genome_rows, d_ref_rows, &first, &end)) return rc;
  if (int rc = queue_blocks(c, d_genome_start, d_ref_start, d_col_off, d_genome_rows, d_ref_rows, nblocks, first, end,
                            d_lut, n))
    return rc;
  return check_device_error(c);
}

int mvg_lut_from_blocks(mvg_handle h, const int64_t* genome_start, const int64_t* ref_start, const uint64_t* col_off,
                        const uint8_t* genome_rows, const uint8_t* ref_rows, uint64_t nblocks, int32_t* lut,
                        uint64_t n) {
  if (!h || (nblocks && (!genome_start || !ref_start || !col_off)) || (n && !lut))
    return report_error(MVG_ERR_ARG, "bad argument");
  Ctx* c = ctx_of(h);
  MVG_CUDA_TRY(cudaSetDevice(c->device));
  if (int rc = check_lut_len(n)) return rc;
  uint64_t ncols = 0;
  if (nblocks) {
    for (uint64_t b = 0; b < nblocks; ++b)
      if (col_off[b + 1] < col_off[b]) return report_error(MVG_ERR_ARG, "column offsets decrease");
    ncols = col_off[nblocks];
    if (ncols && (!genome_rows || !ref_rows)) return report_error(MVG_ERR_ARG, "bad argument");
  }
  const int64_t* d_gs = stage_in(c, kWsHStarts, genome_start, nblocks);
  const int64_t* d_rs = stage_in(c, kWsHAux, ref_start, nblocks);
  const uint64_t* d_off = stage_in(c, kWsHOff, col_off, nblocks + 1);
  const uint8_t* d_g = stage_in(c, kWsHRowG, genome_rows, ncols);
  const uint8_t* d_r = stage_in(c, kWsHRowR, ref_rows, ncols);
  int32_t* d_lut = (int32_t*)c->ws.get(c, kWsHLut, n * 4 + 16);
  if (!d_gs || !d_rs || !d_off || !d_g || !d_r || !d_lut) return report_error(MVG_ERR_NOMEM, "staging failed");
  if (int rc = queue_blocks(c, d_gs, d_rs, d_off, d_g, d_r, nblocks, nblocks ? col_off[0] : 0, ncols, d_lut, n))
    return rc;
  if (int rc = check_device_error(c)) return rc;
  return finish_out(c, lut, d_lut, n * 4);
}

int mvg_lut_fix_zero_idx_dev(mvg_handle h, int32_t* d_lut, uint64_t n, const uint8_t* d_genome, uint64_t genome_len,
                             const uint8_t* d_ref, uint64_t ref_len) {
  if (!h || (n && !d_lut) || (genome_len && !d_genome) || (ref_len && !d_ref))
    return report_error(MVG_ERR_ARG, "bad argument");
  Ctx* c = ctx_of(h);
  MVG_CUDA_TRY(cudaSetDevice(c->device));
  if (int rc = check_lut_len(n)) return rc;
  return lut_fix_zero_dev(c, d_lut, (int64_t)n, d_genome, genome_len, d_ref, ref_len);
}

int mvg_lut_fix_zero_idx(mvg_handle h, int32_t* lut, uint64_t n, const uint8_t* genome, uint64_t genome_len,
                         const uint8_t* ref, uint64_t ref_len) {
  if (!h || (n && !lut) || (genome_len && !genome) || (ref_len && !ref)) return report_error(MVG_ERR_ARG, "bad argument");
  Ctx* c = ctx_of(h);
  MVG_CUDA_TRY(cudaSetDevice(c->device));
  if (int rc = check_lut_len(n)) return rc;
  int32_t* d_lut = stage_in(c, kWsHLut, lut, n);
  const uint8_t* d_g = stage_in(c, kWsHGenome, genome, genome_len);
  const uint8_t* d_r = stage_in(c, kWsHRef, ref, ref_len);
  if (!d_lut || !d_g || !d_r) return report_error(MVG_ERR_NOMEM, "staging failed");
  if (int rc = lut_fix_zero_dev(c, d_lut, (int64_t)n, d_g, genome_len, d_r, ref_len)) return rc;
  return finish_out(c, lut, d_lut, 4);
}

static int fill_common(mvg_handle h, int32_t* lut, uint64_t n, int width, int mode, int32_t* gaps, bool host) {
  if (!h || (n && !lut)) return report_error(MVG_ERR_ARG, "bad argument");
  Ctx* c = ctx_of(h);
  MVG_CUDA_TRY(cudaSetDevice(c->device));
  if (int rc = check_lut_len(n)) return rc;
  if (!host) return lut_fill_dev(c, lut, (int64_t)n, width, mode, gaps);
  int32_t* d_lut = stage_in(c, kWsHLut, lut, n);
  int32_t* d_gaps = gaps ? (int32_t*)c->ws.get(c, kWsHAux, n * 4 + 16) : nullptr;
  if (!d_lut || (gaps && !d_gaps)) return report_error(MVG_ERR_NOMEM, "staging failed");
  if (int rc = lut_fill_dev(c, d_lut, (int64_t)n, width, mode, d_gaps)) return rc;
  if (gaps && n) MVG_CUDA_TRY(cudaMemcpyAsync(gaps, d_gaps, n * 4, cudaMemcpyDeviceToHost, c->stream));
  return finish_out(c, lut, d_lut, n * 4);
}

int mvg_lut_fill_gaps(mvg_handle h, int32_t* lut, uint64_t n, int max_gap_width) {
  return fill_common(h, lut, n, max_gap_width, kFill, nullptr, true);
}
int mvg_lut_fill_gaps_dev(mvg_handle h, int32_t* d_lut, uint64_t n, int max_gap_width) {
  return fill_common(h, d_lut, n, max_gap_width, kFill, nullptr, false);
}
int mvg_lut_smooth_edges(mvg_handle h, int32_t* lut, uint64_t n, int smoothing_radius) {
  return fill_common(h, lut, n, smoothing_radius, kSmooth, nullptr, true);
}
int mvg_lut_smooth_edges_dev(mvg_handle h, int32_t* d_lut, uint64_t n, int smoothing_radius) {
  return fill_common(h, d_lut, n, smoothing_radius, kSmooth, nullptr, false);
}
int mvg_lut_find_gaps(mvg_handle h, int32_t* lut, uint64_t n, int32_t* gaps) {
  if (n && !gaps) return report_error(MVG_ERR_ARG, "bad argument");
  return fill_common(h, lut, n, 300, kFill, gaps, true);
}
int mvg_lut_find_gaps_dev(mvg_handle h, int32_t* d_lut, uint64_t n, int32_t* d_gaps) {
  if (n && !d_gaps) return report_error(MVG_ERR_ARG, "bad argument");
  return fill_common(h, d_lut, n, 300, kFill, d_gaps, false);
}

int mvg_lut_find_edges(mvg_handle h, const int32_t* lut, uint64_t n, uint8_t* edges) {
  if (!h || (n && (!lut || !edges))) return report_error(MVG_ERR_ARG, "bad argument");
  Ctx* c = ctx_of(h);
  MVG_CUDA_TRY(cudaSetDevice(c->device));
  if (int rc = check_lut_len(n)) return rc;
  const int32_t* d_lut = stage_in(c, kWsHLut, lut, n);
  uint8_t* d_e = (uint8_t*)c->ws.get(c, kWsHAux, n + 16);
  if (!d_lut || !d_e) return report_error(MVG_ERR_NOMEM, "staging failed");
  if (int rc = lut_find_edges_dev(c, d_lut, (int64_t)n, d_e)) return rc;
  return finish_out(c, edges, d_e, n);
}

int mvg_lut_find_mismatches(mvg_handle h, const int32_t* lut, uint64_t n, const uint8_t* genome, uint64_t genome_len,
                            const uint8_t* ref, uint64_t ref_len, uint8_t* mismatches) {
  if (!h || (n && (!lut || !mismatches)) || (genome_len && !genome) || (ref_len && !ref))
    return report_error(MVG_ERR_ARG, "bad argument");
  Ctx* c = ctx_of(h);
  MVG_CUDA_TRY(cudaSetDevice(c->device));
  if (int rc = check_lut_len(n)) return rc;
  const int32_t* d_lut = stage_in(c, kWsHLut, lut, n);
  const uint8_t* d_g = stage_in(c, kWsHGenome, genome, genome_len);
  const uint8_t* d_r = stage_in(c, kWsHRef, ref, ref_len);
  uint8_t* d_m = (uint8_t*)c->ws.get(c, kWsHAux, n + 16);
  if (!d_lut || !d_g || !d_r || !d_m) return report_error(MVG_ERR_NOMEM, "staging failed");
  if (int rc = lut_find_mismatches_dev(c, d_lut, (int64_t)n, d_g, genome_len, d_r, ref_len, d_m)) return rc;
  return finish_out(c, mismatches, d_m, n);
}

int mvg_lut_find_duplicate_mappings(mvg_handle h, const int32_t* lut, uint64_t n, int64_t* result) {
  if (!h || !result || (n && !lut)) return report_error(MVG_ERR_ARG, "bad argument");
  Ctx* c = ctx_of(h);
  MVG_CUDA_TRY(cudaSetDevice(c->device));
  if (int rc = check_lut_len(n)) return rc;
  const int32_t* d_lut = stage_in(c, kWsHLut, lut, n);
  if (!d_lut) return report_error(MVG_ERR_NOMEM, "staging failed");
  return lut_duplicate_mappings_dev(c, d_lut, (int64_t)n, result);
}

int mvg_build_index_lut_dev(mvg_handle h, const int64_t* d_genome_start, const int64_t* d_ref_start,
                            const uint64_t* d_col_off, const uint8_t* d_genome_rows, const uint8_t* d_ref_rows,
                            uint64_t nblocks, const uint8_t* d_genome, uint64_t genome_len, const uint8_t* d_ref,
                            uint64_t ref_len, int fill_gaps, int max_gap_width, int smooth_edges,
                            int smoothing_radius, int32_t* d_lut, uint64_t n) {
  if (fill_gaps && ((genome_len && !d_genome) || (ref_len && !d_ref))) return report_error(MVG_ERR_ARG, "bad argument");
  if (!h || (nblocks && (!d_genome_start || !d_ref_start || !d_col_off)) || (n && !d_lut))
    return report_error(MVG_ERR_ARG, "bad argument");
  Ctx* c = ctx_of(h);
  MVG_CUDA_TRY(cudaSetDevice(c->device));
  uint64_t first, end;
  if (int rc = read_cols(c, d_col_off, nblocks, d_genome_rows, d_ref_rows, &first, &end)) return rc;
  if (int rc = queue_blocks(c, d_genome_start, d_ref_start, d_col_off, d_genome_rows, d_ref_rows, nblocks, first, end,
                            d_lut, n))
    return rc;
  return index_passes(c, d_lut, (int64_t)n, ZeroFix{d_genome, d_ref, genome_len, ref_len, 1}, fill_gaps, max_gap_width,
                      smooth_edges, smoothing_radius);
}

int mvg_build_index_lut(mvg_handle h, const int64_t* genome_start, const int64_t* ref_start, const uint64_t* col_off,
                        const uint8_t* genome_rows, const uint8_t* ref_rows, uint64_t nblocks, const uint8_t* genome,
                        uint64_t genome_len, const uint8_t* ref, uint64_t ref_len, int fill_gaps, int max_gap_width,
                        int smooth_edges, int smoothing_radius, int32_t* lut, uint64_t n) {
  if (!h || (nblocks && (!genome_start || !ref_start || !col_off)) || (n && !lut))
    return report_error(MVG_ERR_ARG, "bad argument");
  if (fill_gaps && ((genome_len && !genome) || (ref_len && !ref))) return report_error(MVG_ERR_ARG, "bad argument");
  Ctx* c = ctx_of(h);
  MVG_CUDA_TRY(cudaSetDevice(c->device));
  if (int rc = check_lut_len(n)) return rc;
  uint64_t ncols = 0;
  if (nblocks) {
    for (uint64_t b = 0; b < nblocks; ++b)
      if (col_off[b + 1] < col_off[b]) return report_error(MVG_ERR_ARG, "column offsets decrease");
    ncols = col_off[nblocks];
    if (ncols && (!genome_rows || !ref_rows)) return report_error(MVG_ERR_ARG, "bad argument");
  }
  const int64_t* d_gs = stage_in(c, kWsHStarts, genome_start, nblocks);
  const int64_t* d_rs = stage_in(c, kWsHAux, ref_start, nblocks);
  const uint64_t* d_off = stage_in(c, kWsHOff, col_off, nblocks + 1);
  const uint8_t* d_gr = stage_in(c, kWsHRowG, genome_rows, ncols);
  const uint8_t* d_rr = stage_in(c, kWsHRowR, ref_rows, ncols);
  const uint8_t* d_g = fill_gaps ? stage_in(c, kWsHGenome, genome, genome_len) : nullptr;
  const uint8_t* d_r = fill_gaps ? stage_in(c, kWsHRef, ref, ref_len) : nullptr;
  int32_t* d_lut = (int32_t*)c->ws.get(c, kWsHLut, n * 4 + 16);
  if (!d_gs || !d_rs || !d_off || !d_gr || !d_rr || !d_lut || (fill_gaps && (!d_g || !d_r)))
    return report_error(MVG_ERR_NOMEM, "staging failed");
  if (int rc = queue_blocks(c, d_gs, d_rs, d_off, d_gr, d_rr, nblocks, nblocks ? col_off[0] : 0, ncols, d_lut, n))
    return rc;
  if (int rc = index_passes(c, d_lut, (int64_t)n, ZeroFix{d_g, d_r, genome_len, ref_len, 1}, fill_gaps, max_gap_width,
                            smooth_edges, smoothing_radius))
    return rc;
  return finish_out(c, lut, d_lut, n * 4);
}

}  // extern "C"
