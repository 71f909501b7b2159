// The banded NWSmall kernel on a ring schedule (included by gapdp.cu after
// gapdp_strips.cuh, whose recurrence, profile and nibbles it shares; the bound
// is gapdp_kernel.cuh's).
//
// One warp solves one problem.  Rows are cut into groups of R (RingBand,
// band.h); lane g mod 32 runs group g, and the 32 lanes form a ring: lane t
// receives the bottom row of the group above it from lane t-1, lane 0 from
// lane 31, through one rotating shuffle per step.  Every group is as wide as
// the band (W columns) and starts one step after its predecessor reached the
// group's first column, so a lane never sweeps the staircase that a 32*R-row
// strip spans on a diagonal band, and there is no ramp-up or ramp-down per
// strip: the ring runs from the first group's start to the last group's end.
// A lane idles between its groups when the band is narrow for R; the host
// picks the smallest R whose schedule is valid (ring_eligible), which keeps
// lanes busy most of the time.
//
// Values are scaled by 16 with the strips' tags.  Cells outside the band are
// kRingNeg; scores added along the band's edge let such a value drift by at
// most 2,560 a row, and kRingScaledMax keeps it below every real score.
//
// Exactness: the kept region is a union of group rectangles.  A banded score
// is accepted only when it is strictly above an upper bound on every path
// that leaves the region, as in the strip kernel: each cell a path can leave
// from (the bottom row of a group left of the next group's first column, the
// right-most column of a group short of LB, row 0 right of group 0, column 0
// below the last group that reaches it) contributes its score plus
// min(sum of A's best-base scores below it, sum of B's right of it).  Prefix
// sums of both are staged in shared memory with the sequences.
//
// Traceback words: each lane writes its R nibbles per step as one stream
// (ring_tb_at), so every store is one coalesced 128-byte row.
#pragma once
#include <limits.h>

#include "band.h"

namespace mvg {

struct RingJob {
  const uint8_t* sa;
  const uint64_t* oa;
  const uint8_t* sb;
  const uint64_t* ob;
  const uint32_t* order;   // problem ids of this launch, longest first
  const uint8_t* rows_of;  // group height of each
  const uint64_t* tb_off;  // byte offset of each slot's traceback words
  int nwork;
  uint32_t* tb;
  int32_t* scores;
  uint8_t* end_edge;
  const int32_t* band_delta;
  const int32_t* band_half;
  uint8_t* accept;
  uint32_t base_max;
  unsigned* counter;
  unsigned long long* cells;  // kept cells inside the matrix, summed over problems
};

constexpr int kRingThreads = 128;
constexpr int kRingA = 256;  // rows of A staged per warp (codes of the next groups to start)
constexpr int32_t kRingNeg = -(1 << 30);
constexpr int kRingScaledMax = 200000;  // min(LA, LB) up to which scaled scores and drift fit

// Shared memory of one warp of a launch whose tallest groups have RMAX rows.
template <int RMAX>
struct RingSmem {
  int4 prof[RMAX][32];  // [4 * (row / 4) + base][lane]: the scores of four rows of the lane's group
  int2 colB[128];       // per staged column: 512 times the base's code, best scores of B up to it
  int32_t prefA[kRingA];  // per staged row: best scores of A up to it
  __align__(16) uint8_t codeA[kRingA];
  int32_t score[16];    // [4 * a + b], scaled and tagged
};

// Inclusive sum over the warp's lanes.
__device__ __forceinline__ int32_t ring_scan(int32_t v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int32_t t = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= d) v += t;
  }
  return v;
}

template <int R, int RMAX>
__device__ void ring_solve(const RingJob& J, RingSmem<RMAX>& sm, int w) {
  constexpr int NW = (R + 7) / 8, NQ = (R + 3) / 4;
  constexpr int32_t kOpenD = kOpen2 * 16 + 3, kOpenI = kOpen2 * 16 + 6, kFree = kOpen2 * 16;
  const int lane = threadIdx.x & 31;
  const int src = (lane + 31) & 31;  // the ring's previous lane
  const uint32_t p = J.order[w];
  const uint64_t a0 = J.oa[p], b0 = J.ob[p];
  const int LA = (int)(J.oa[p + 1] - a0), LB = (int)(J.ob[p + 1] - b0);
  const uint8_t* A = J.sa + a0;
  const uint8_t* B = J.sb + b0;
  const RingBand b = make_ring_band(LA, LB, J.band_delta[p], J.band_half[p], R);
  const int G = b.G, W = b.W, lo0 = b.lo0;
  const int S = (int)b.steps;
  const int32_t totA = warp_best_sum(A, 0, LA, J.base_max);
  const int32_t totB = warp_best_sum(B, 0, LB, J.base_max);

  // warp-uniform: the next group to start, its first column, and the band
  // centre floor((gR+1)*LB/LA) of that group kept as quotient f, remainder m
  int gnext = 0;
  int f = LB / LA, m = LB % LA;
  const int qR = (int)((int64_t)R * LB / LA), rR = (int)((int64_t)R * LB % LA);
  const int shift = b.delta - b.half;
  int lo_next = f + shift;  // == lo0
  int lo_started = lo0;     // first column of the last group started
  int filled = lo0 - 1;     // colB holds columns (filled - 128, filled]
  int filledA = 0;          // codeA and prefA hold rows [filledA - kRingA, filledA) of A
  int32_t sumA = 0, sumB = filled > 0 ? warp_best_sum(B, 0, filled, J.base_max) : 0;

  // this lane's group
  int my_g = -1, j = INT_MIN / 2, my_end = INT_MIN, j_end = INT_MIN, prev_hi = INT_MIN, next_lo = INT_MIN;
  int exit_col = INT_MIN, end_col = INT_MIN;  // right-edge exits; the end cell
  int32_t topV = kRingNeg, left_a = 0;
  uint32_t codes[(R + 15) / 16];  // the group's rows of A, two bits each
  int32_t V[R], I[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    V[r] = kRingNeg;
    I[r] = kRingNeg;
  }
  int32_t pubV = kRingNeg, pubD = kRingNeg | 1;  // this lane's bottom row, last column
  int32_t dg = kRingNeg;                         // V above-left of the next column
  int32_t raw = kRingNeg;                        // V the previous lane published one step ago
  int32_t bound = kNeg, endsc = kNeg;
  int end_lane_edge = 0;
  uint32_t kept = 0;
  uint32_t acc = 0;
  uint32_t* tbp = J.tb + J.tb_off[w] / 4 + lane;

  for (int s = 0; s < S; ++s) {
    const int32_t rV = __shfl_sync(0xffffffffu, pubV, src);
    const int32_t rD = __shfl_sync(0xffffffffu, pubD, src);
    ++j;
    if (gnext < G && s - gnext == lo_next - lo0) {
      const int g = gnext;
      __syncwarp();
      if (filledA < (g + 1) * R) {  // rows of A about to start, staged 128 at a time
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int i = filledA + k * 32 + lane;
          const uint32_t code = i < LA ? A[i] & 3u : 0u;
          const int32_t incl = sumA + ring_scan(i < LA ? best_of(J.base_max, code) : 0);
          sm.codeA[i & (kRingA - 1)] = (uint8_t)code;
          sm.prefA[i & (kRingA - 1)] = incl;
          sumA = __shfl_sync(0xffffffffu, incl, 31);
        }
        __syncwarp();
        filledA += 128;
      }
      // the group's profile: lane x writes base x / 8 of rows x mod 8, 8 + x mod 8, ...
#pragma unroll
      for (int k = 0; k < (R + 7) / 8; ++k) {
        const int r = 8 * k + (lane & 7), base = lane >> 3;
        if (R % 8 == 0 || r < R) {
          const int32_t sc = sm.score[4 * sm.codeA[(g * R + r) & (kRingA - 1)] + base];
          reinterpret_cast<int32_t*>(&sm.prof[4 * (r >> 2) + base][g & 31])[r & 3] = sc;
        }
      }
      __syncwarp();
      const int lo_prev = lo_started;
      f += qR;
      m += rR;
      if (m >= LA) {
        m -= LA;
        ++f;
      }
      const int lo_after = f + shift;
      if (lane == (g & 31)) {
        const int my_lo = lo_next;
        my_g = g;
        j = my_lo;
        my_end = my_lo + W - 1;
        j_end = my_end < LB ? my_end : LB;
        prev_hi = g == 0 ? INT_MIN : lo_prev + W - 1;
        next_lo = g + 1 < G ? lo_after : INT_MIN;
        exit_col = my_end < LB ? my_end : INT_MIN;
        end_col = g == G - 1 ? LB : INT_MIN;
#pragma unroll
        for (int q = 0; q < (R + 15) / 16; ++q) codes[q] = 0;
#pragma unroll
        for (int r = 0; r < R; r += 2) {  // R is even and groups start at even rows
          const uint32_t two = *reinterpret_cast<const uint16_t*>(&sm.codeA[(g * R + r) & (kRingA - 1)]);
          codes[r >> 4] |= ((two & 3u) | ((two >> 6) & 12u)) << (2 * (r & 15));
        }
        const int rows_here = LA - g * R < R ? LA - g * R : R;
        left_a = totA - sm.prefA[(g * R + rows_here - 1) & (kRingA - 1)];
        // cells of this group inside the matrix
        const int c0 = my_lo < 1 ? 1 : my_lo;
        if (j_end >= c0) kept += (uint32_t)rows_here * (uint32_t)(j_end - c0 + 1);
        topV = g == 0 ? kFree : kRingNeg;
        // column 0 is (-inf, 0, -inf) below row 0
        const int32_t left = my_lo == 1 ? kFree : kRingNeg;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          V[r] = left;
          I[r] = kRingNeg;
        }
        // cell above-left of the first column: (gR, my_lo - 1)
        const int x = my_lo - 1;
        if (g == 0)  // row 0: M(0,0) = 0, I(0,j) = 0 for j >= 1
          dg = x == 0 ? (LA > 1 ? kGap * 16 : kFree) : x >= 1 ? kFree : kRingNeg;
        else if (x <= 0)
          dg = x == 0 ? kFree : kRingNeg;
        else
          dg = x >= lo_prev ? raw : kRingNeg;  // the predecessor computed it two steps ago
      }
      lo_started = lo_next;
      lo_next = lo_after;
      ++gnext;
    }
    // B of the running groups' columns: up to s - (gnext - 32) + lo0
    if (filled < s + 32 - gnext + lo0) {
      const int x = filled + 1 + lane;
      const bool in = x >= 1 && x <= LB;
      const uint32_t code = in ? B[x - 1] & 3u : 0u;
      const int32_t incl = sumB + ring_scan(in ? best_of(J.base_max, code) : 0);
      __syncwarp();
      sm.colB[x & 127] = make_int2((int)(code * 512u), incl);
      __syncwarp();
      sumB = __shfl_sync(0xffffffffu, incl, 31);
      filled += 32;
    }
    // the cell above: the predecessor's bottom row while inside its range;
    // for group 0 row 0 (I = 0 right of column 0; M(0,0) is set below)
    const bool from_ring = j <= prev_hi;
    int32_t uV = from_ring ? rV : topV;
    const int32_t uD = from_ring ? rD : kRingNeg | 1;
    uint32_t nw[NW];
#pragma unroll
    for (int q = 0; q < NW; ++q) nw[q] = 0;
    pubV = kRingNeg;
    pubD = kRingNeg | 1;
    if (j <= j_end && j >= 1) {
      const int2 col = sm.colB[j & 127];
      const char* prof = reinterpret_cast<const char*>(&sm.prof[0][lane]) + col.x;
      int32_t sc[4 * NQ];
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const int4 v = *reinterpret_cast<const int4*>(prof + q * 2048);
        sc[4 * q] = v.x;
        sc[4 * q + 1] = v.y;
        sc[4 * q + 2] = v.z;
        sc[4 * q + 3] = v.w;
      }
      if (j == exit_col) {  // every row's best state may leave the band to the right
        const int rows_here = LA - my_g * R < R ? LA - my_g * R : R;
        const int32_t leftB = totB - col.y;
        int32_t up = dg, D = uD, left = left_a;
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (r < rows_here) left += best_of(J.base_max, codes[r >> 4] >> (2 * (r & 15)));
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int32_t M = up + sc[r];
          const int32_t best = (__viaddmax_s32(M, kGap * 16, max(D, I[r])) >> 4) - kOpen2;
          left -= best_of(J.base_max, codes[r >> 4] >> (2 * (r & 15)));
          if (r < rows_here) bound = __viaddmax_s32(best, min(left, leftB), bound);
          D = __viaddmax_s32(M, kOpenD, D) & ~4;
          up = V[r];
        }
      }
      if (j == end_col) {  // the end cell (LA, LB)
        const int last = LA - 1 - my_g * R;
        int32_t up = dg, D = uD;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int32_t M = up + sc[r];
          if (r == last) {
            const int32_t eM = (M >> 4) - kGap, eD = (D >> 4) - kOpen2, eI = (I[r] >> 4) - kOpen2;
            endsc = max(eM, max(eD, eI));
            end_lane_edge = eM == endsc ? 'M' : eD == endsc ? 'D' : 'I';
          }
          D = __viaddmax_s32(M, kOpenD, D) & ~4;
          up = V[r];
        }
      }
      int32_t up = dg, D = uD;
      int32_t lastM = 0, lastDI = 0;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int32_t M = up + sc[r];
        const int32_t v = __vimax3_s32(M, D, I[r]);
        if (r == R - 1) {
          lastM = M;
          lastDI = max(D, I[r]);
        }
        const int32_t nd = __viaddmax_s32(M, kOpenD, D);
        const int32_t ni = __viaddmax_s32(M, kOpenI, I[r]);
        up = V[r];
        nw[r >> 3] = __funnelshift_r(nw[r >> 3], (uint32_t)(v ^ nd ^ ni), 4);
        V[r] = v & ~3;
        D = nd & ~4;
        I[r] = ni & ~8;
      }
      if constexpr (R % 8 != 0) nw[NW - 1] >>= 32 - 4 * (R % 8);
      pubV = V[R - 1];
      pubD = D;
      if (j < next_lo) {  // bottom-row exit: max(M, D, I)
        const int32_t best = (__viaddmax_s32(lastM, kGap * 16, lastDI) >> 4) - kOpen2;
        bound = max(bound, best + min(left_a, totB - col.y));
      }
    } else if (j <= my_end && j <= 0 && my_g >= 0) {
      // the left boundary column (D = 0 below row 0) or outside the matrix
      const int32_t left = j == 0 ? kFree : kRingNeg;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        V[r] = left;
        I[r] = kRingNeg;
      }
      pubV = left;
      if (my_g == 0 && j == 0) uV = LA > 1 ? kGap * 16 : kFree;  // cell (0, 0)
    }
    if constexpr (R < 8 && 8 % R == 0) {
      constexpr int kPer = 8 / R;
      acc |= nw[0] << (4 * R * (s % kPer));
      if ((s % kPer) == kPer - 1 || s == S - 1) {
        *tbp = acc;
        tbp += 32;
        acc = 0;
      }
    } else {
#pragma unroll
      for (int q = 0; q < NW; ++q) tbp[q * 32] = nw[q];
      tbp += NW * 32;
    }
    dg = uV;
    raw = rV;
  }
  // paths along row 0 past group 0, and down column 0 past the last group
  // that reaches it (both score 0 up to the exit)
  const int hi0 = lo0 + W - 1;
  const int32_t pb0 = hi0 < LB ? warp_best_sum(B, 0, hi0, J.base_max) : 0;
  int gcol = 0;
  while (gcol + 1 < G && ring_lo(b, gcol + 1) <= 1) ++gcol;
  const int last_col0 = (gcol + 1) * R;
  const int32_t pa0 = last_col0 < LA ? warp_best_sum(A, 0, last_col0, J.base_max) : 0;
  if (lane == 0) {
    if (hi0 < LB) bound = max(bound, min(totA, totB - pb0));
    if (last_col0 < LA) bound = max(bound, min(totA - pa0, totB));
  }
  unsigned long long kept64 = kept;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    bound = max(bound, __shfl_xor_sync(0xffffffffu, bound, d));
    kept64 += __shfl_xor_sync(0xffffffffu, kept64, d);
  }
  const int end_lane = (G - 1) & 31;
  const int32_t sc = __shfl_sync(0xffffffffu, endsc, end_lane);
  if (lane == end_lane) {
    J.scores[p] = sc;
    J.end_edge[p] = (uint8_t)end_lane_edge;
  }
  if (lane == 0) {
    J.accept[p] = sc > bound ? 1 : 0;
    if (J.cells) atomicAdd(J.cells, kept64);
  }
}

// Problems of all heights up to RMAX (above the previous launch's), claimed
// longest first.  One launch for several heights: a launch per height ends in
// the chain of steps of its longest problem, and those tails added up.
// 4 and 2 CTAs per SM (128 and 218 registers): 30,011 recoded-pair gaps took
// 15.8 ms, against 16.6 at 5 and 17.7 at 6 of the low launch.
template <int RMAX>
__global__ void __launch_bounds__(kRingThreads, RMAX == 12 ? 4 : 2) k_gapdp_ring(RingJob J) {
  extern __shared__ __align__(16) uint8_t ring_smem[];
  const int lane = threadIdx.x & 31;
  RingSmem<RMAX>& sm = reinterpret_cast<RingSmem<RMAX>*>(ring_smem)[threadIdx.x >> 5];
  if (lane < 16)
    sm.score[lane] = ((int32_t)((c_score_rows[lane >> 2] >> (8 * (lane & 3))) & 255u) - kScoreBias) * 16 + 2;
  __syncwarp();
  for (;;) {
    int w = 0;
    if (lane == 0) w = (int)atomicAdd(J.counter, 1u);
    w = __shfl_sync(0xffffffffu, w, 0);
    if (w >= J.nwork) break;
    const int R = J.rows_of[w];
    if constexpr (RMAX == 12) {
      if (R == 4)
        ring_solve<4>(J, sm, w);
      else if (R == 6)
        ring_solve<6>(J, sm, w);
      else if (R == 8)
        ring_solve<8>(J, sm, w);
      else
        ring_solve<12>(J, sm, w);
    } else {
      if (R == 16)
        ring_solve<16>(J, sm, w);
      else if (R == 24)
        ring_solve<24>(J, sm, w);
      else
        ring_solve<32>(J, sm, w);
    }
  }
}

// BitTraceBack (MU/bittraceback.cpp:138-210) over the ring layout, one warp
// per accepted problem, by runs of equal moves as walk_path finds them (lane l
// reads the nibble l + 1 moves on; the words a window further along are
// prefetched to L2).  The path is written from the end of its slot and moved
// to the head.
template <int R>
__device__ void ring_walk(const uint32_t* T, const RingBand& b, char* path, char X, uint32_t* err, int64_t* path_len) {
  const int lane = threadIdx.x & 31;
  const int64_t limit = (int64_t)b.LA + b.LB;
  int pa = b.LA, pb = b.LB;
  int64_t n = 0;
  bool fail = false;
  for (;;) {
    const int di = X != 'I', dj = X != 'D';
    const int i = pa - di * (lane + 1), j = pb - dj * (lane + 1);
    bool valid = false, more = false;
    uint32_t bits = 0;
    auto word_of = [&](int ci, int cj, int& sh) -> const uint32_t* {
      const int g = (ci - 1) / R, r = (ci - 1) % R;
      const int64_t s = (int64_t)cj + g - b.lo0;
      if (s < 0 || s >= b.steps) return nullptr;
      int64_t word;
      ring_tb_at(R, s, r, word, sh);
      return T + word * 32 + (g & 31);
    };
    if (i >= 1 && j >= 1) {
      int sh = 0;
      if (const uint32_t* at = word_of(i, j, sh)) {
        valid = true;
        bits = (*at >> sh) & 15u;
        more = X == 'M' ? (bits & 3u) == 3u : X == 'D' ? !(bits & 4u) : !(bits & 8u);
      }
      if (i > 32 && j > 32)
        if (const uint32_t* at = word_of(i - 32, j - 32, sh)) asm volatile("prefetch.global.L2 [%0];" ::"l"(at));
    }
    const uint32_t stop = ~__ballot_sync(0xffffffffu, more);
    const int run = stop ? __ffs(stop) - 1 : 32;
    const int count = run < 32 ? run + 1 : 32;
    if (n + count > limit) {
      fail = true;
      break;
    }
    if (lane < count) path[limit - n - 1 - lane] = X;
    n += count;
    pa -= di * count;
    pb -= dj * count;
    if (run == 32) continue;  // X also at the new cell
    bits = __shfl_sync(0xffffffffu, bits, run);
    valid = __shfl_sync(0xffffffffu, valid ? 1 : 0, run) != 0;
    if (pa < 0 || pb < 0) {
      fail = true;
      break;
    }
    if (pa == 0 || pb == 0) {  // along row 0 or column 0 to the origin
      X = pa == 0 ? 'I' : 'D';
      const int rest = pa + pb;
      if (n + rest > limit) {
        fail = true;
        break;
      }
      for (int l = lane; l < rest; l += 32) path[limit - n - 1 - l] = X;
      n += rest;
      break;
    }
    if (!valid) {  // outside an accepted band cannot happen
      fail = true;
      break;
    }
    if (X == 'M')
      X = (bits & 3u) == 3u ? 'M' : (bits & 3u) == 0u ? 'D' : 'I';
    else
      X = (bits & (X == 'D' ? 4u : 8u)) ? 'M' : X;
  }
  if (fail && lane == 0) set_error(err, kDevCapacity);
  if (lane == 0) *path_len = n;
  __syncwarp();
  walk_compact(path, limit, n, lane, 32, [] { __syncwarp(); });
}

__global__ void __launch_bounds__(128) k_ring_walk(RingJob J, const uint64_t* __restrict__ path_off,
                                                   char* __restrict__ paths, int64_t* __restrict__ path_len,
                                                   uint32_t* err) {
  const int w = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (w >= J.nwork) return;
  const uint32_t p = J.order[w];
  if (!J.accept[p]) return;
  const int LA = (int)(J.oa[p + 1] - J.oa[p]), LB = (int)(J.ob[p + 1] - J.ob[p]);
  const int R = J.rows_of[w];
  const RingBand b = make_ring_band(LA, LB, J.band_delta[p], J.band_half[p], R);
  const uint32_t* T = J.tb + J.tb_off[w] / 4;
  char* path = paths + path_off[p];
  const char X = (char)J.end_edge[p];
  int64_t* len = path_len + p;
  switch (R) {
    case 4: ring_walk<4>(T, b, path, X, err, len); break;
    case 6: ring_walk<6>(T, b, path, X, err, len); break;
    case 8: ring_walk<8>(T, b, path, X, err, len); break;
    case 12: ring_walk<12>(T, b, path, X, err, len); break;
    case 16: ring_walk<16>(T, b, path, X, err, len); break;
    case 24: ring_walk<24>(T, b, path, X, err, len); break;
    default: ring_walk<32>(T, b, path, X, err, len); break;
  }
}

}  // namespace mvg
