// The full gap DP (NWSmall) in strips on a grid-wide pipeline (included by
// gapdp.cu after gapdp_kernel.cuh).
//
// The matrix is cut into strips of 32*R rows; one warp runs one strip, lane t
// owning rows [t*R, t*R+R) and running t columns behind lane 0 (step s: lane
// t at column offset x = s - t).  A strip is the unit of work: the strips of
// a large problem are consecutive entries of one grid-wide queue, so they run
// on as many warps as are free, wherever they are, each following its
// predecessor some 70 columns behind through the predecessor's bottom row in
// global memory.  A row's columns are 64-bit words set to kStUnwritten before
// the pass: a reader sees by the word itself whether it is there, so there
// are no flags, fences or progress words (with a progress word released every
// 32 columns, warps spent 40% of their time on the fence and on the two L2
// round trips before each chunk).  A unit is claimed only after its
// predecessor was, by a warp that is running, so every wait ends; a bounded
// spin turns a fault of that reasoning into an error.  Problems are claimed in
// groups of kStGroup, strip by strip: first all their first strips, then all
// their second ones, and so on.  A strip claimed right after its predecessor
// would hold a warp for as long as the strips above it take to get going.
//
// Before, a CTA's 8 warps shared a problem, and a batch took as long as one
// CTA needed for its 20 kbp pairs.  Measured on 4,000 pairs of 10-20,000 bp
// (1.05e11 cells): forward pass 70.3 -> 27.5 ms, traceback 20.8 -> 3.3 ms.
//
// Cell recurrence.  With extension 0 and open and close both -200, carrying
//   M(i,j) as the reference's M plus the open (Mg),  D~, I~ = D, I - 400,
//   V(i,j) = max(Mg, D~, I~)
// gives
//   Mg(i,j)   = s(i,j) + V(i-1,j-1)
//   D~(i+1,j) = max(Mg(i,j) - 400, D~(i,j)),  I~(i,j+1) = max(Mg(i,j) - 400, I~(i,j))
// which is two add-max, one three-way max and one add per cell, and two
// values per row and column boundary (V and the next D~ or I~) instead of
// three.  All comparisons are the reference's with the same constant added to
// both sides, so every decision and every tie is the same.  Row 0 and column
// 0 are V = -400 (V(0,0) = -200; -400 for LA == 1, where NWSmall's last-row
// case adds the close, MU/nwsmall.cpp:616-624) with D~(1,j) = I~(i,1) = -inf:
// the free terminal opens need no case of their own.
//
// Scores come from a per-warp query profile in shared memory (the four
// scores of a lane's row against A, C, G, T), one 128-bit load per four
// cells; a lane's address depends on its column's base only in units of 512
// bytes, so the loads are conflict-free.  That takes the table lookup off the
// integer pipe (max, add-max and byte permute issue at 64 lanes per clock and
// SM there, measured), which bounds this kernel: three of the four remaining
// operations per cell go through it.
//
// What a strip leaves for the traceback (per problem slot, StripShape):
//   rows    the bottom row of every strip but the last, (V, next D~) per column;
//   states  checkpointed problems: every kStBlock steps (or a multiple), all
//           lanes' state;
//   bits    direct problems: the traceback nibbles of every step.
// Nibbles belong to the cell that the move arrives at: bits 0-1 where V comes
// from (3 = M, 0 = D, 1 = I, ties in that order), bit 2 set if the next row's
// D comes from M, bit 3 if the next column's I does.  They fall out of the
// maxima themselves: values are scaled by 16 and carry tags in their low
// bits (V's candidates M 2, D 1, I 0; D's M 5, D 1; I's M 8, I 0), so a
// maximum brings its tie-broken source along, and the exclusive or of the
// three results has the nibble in its low bits.
#pragma once
#include "mvg_common.cuh"

namespace mvg {

constexpr int kStWarps = 4;
constexpr int kStGroup = 1024;             // problems whose strips are claimed level by level
constexpr unsigned long long kStUnwritten = 0x8080808080808080ull;  // V far below any score
constexpr int kStBlockBits = 6;
constexpr int kStBlock = 1 << kStBlockBits;  // steps of a block, and between stored states where there is room
constexpr int kStDirectCols = 700;         // direct bits up to this LB ...
constexpr int64_t kStDirectCells = 4 << 20;  // ... and this many cells
constexpr int kStScaledMax = 400000;       // min(LA, LB) up to which scaled scores fit 32 bits
constexpr int32_t kOpen2 = 2 * kGap;       // open plus close

// How a problem is run: rows per lane, strips, and what is stored for the
// traceback: its bits, or the state every 1 << every steps (a block, or a
// multiple).  The bits of a problem of few columns cost less than computing
// most of its blocks again.
struct StripShape {
  int LA, LB, R, n, S, every;
  bool direct;
};

MVG_HD uint64_t strip_rows_bytes(const StripShape& h) { return ((uint64_t)(h.n - 1) * h.LB * 8 + 255) & ~255ull; }
// stored states of a strip
MVG_HD int strip_states(const StripShape& h) { return (h.S - 1) >> h.every; }
// one state: R (V, next I~) pairs and (V above-left, next D~) per lane
MVG_HD uint64_t strip_state_bytes(const StripShape& h) { return (uint64_t)(h.R + 1) * 32 * 8; }
MVG_HD uint64_t strip_slot_bytes(const StripShape& h) {
  const uint64_t rest = h.direct ? (uint64_t)h.n * h.S * 16 * h.R : (uint64_t)h.n * strip_states(h) * strip_state_bytes(h);
  return (strip_rows_bytes(h) + rest + 255) & ~255ull;
}

MVG_HD StripShape strip_shape(int LA, int LB, int max_rows, bool ckpt) {
  StripShape h;
  h.LA = LA;
  h.LB = LB;
  h.R = max_rows < 8 || LA <= 128 ? 4 : 8;
  h.n = (LA + 32 * h.R - 1) / (32 * h.R);
  h.S = LB + 31;
  h.every = kStBlockBits;
  const int least = LA < LB ? LA : LB;
  h.direct = least <= kStScaledMax && (!ckpt || (LB <= kStDirectCols && (int64_t)LA * LB <= kStDirectCells));
  return h;
}

// The shape of a problem whose slot would take more than `limit`: checkpointed
// in the taller strips, with as many states as fit.
inline StripShape strip_shape_within(StripShape h, uint64_t limit) {
  if (strip_slot_bytes(h) <= limit) return h;
  h.direct = false;
  h.R = h.LA <= 128 ? 4 : 8;
  h.n = (h.LA + 32 * h.R - 1) / (32 * h.R);
  while (strip_slot_bytes(h) > limit && strip_states(h) > 0) ++h.every;
  return h;
}

// A slot as the kernels get it: its byte offset in the arena (a multiple of
// 256) with the shape below it.
inline uint64_t strip_slot(uint64_t offset, const StripShape& h) {
  return offset | (uint64_t)(h.every << 2 | (h.R == 8 ? 2 : 0) | (h.direct ? 1 : 0));
}
MVG_HD uint64_t strip_slot_offset(uint64_t slot) { return slot & ~255ull; }

// The shape of problem p in slot w.  SPARSE: as the slot has it.  A pass whose
// slots were not cut to fit a bound takes it from the lengths: with the states'
// interval and the slot's shape in registers the batch's forward pass took 2%
// longer.
template <bool SPARSE, class Job>
__device__ __forceinline__ StripShape strip_shape_of(const Job& J, uint32_t p, int w) {
  const int LA = (int)(J.oa[p + 1] - J.oa[p]), LB = (int)(J.ob[p + 1] - J.ob[p]);
  if (!SPARSE) return strip_shape(LA, LB, J.max_rows, J.ckpt);
  const uint64_t slot = J.slots[w];
  StripShape h;
  h.LA = LA;
  h.LB = LB;
  h.R = slot & 2 ? 8 : 4;
  h.n = (LA + 32 * h.R - 1) / (32 * h.R);
  h.S = LB + 31;
  h.every = (int)(slot >> 2 & 63);
  h.direct = slot & 1;
  return h;
}

// The least arena bound at which a problem is taken: its cell states at 16
// bytes each, every 128 columns and 32 * max_rows rows (or its nibbles), as
// the entry point has always had it.  The rows alone, which a slot cannot do
// without, are half of that at most.
MVG_HD uint64_t strip_least_bytes(const StripShape& h, int max_rows, bool ckpt) {
  const uint64_t n = ((uint64_t)h.LA + 32 * max_rows - 1) / (32 * max_rows), LB = h.LB;
  return ckpt ? ((n - 1) * LB + n * ((LB + 127) / 128 - 1) * 32 * max_rows) * 16 : n * (LB + 31) * 16 * max_rows;
}

struct StripJob {
  const uint8_t* sa;
  const uint64_t* oa;
  const uint8_t* sb;
  const uint64_t* ob;
  const uint32_t* order;       // slot -> problem: pipelined problems first, each part largest first
  const uint64_t* slots;       // strip_slot
  const uint2* units;          // pipelined strips in claim order: slot, strip
  int nwork, npipe, nunits;
  int max_rows;
  bool ckpt;
  uint8_t* arena;
  int32_t* scores;
  uint8_t* end_edge;
  unsigned* counter;  // [0] claims, [1] set when a wait gave up
  uint32_t* err;
  long long spin_limit;
};

// Before a pass: the pipelined slots' rows unwritten.  Slots along grid.x,
// shares of a slot's rows along grid.y.
template <bool SPARSE>
__global__ void k_strip_unwritten(StripJob J) {
  for (int w = blockIdx.x; w < J.npipe; w += gridDim.x) {
    const uint32_t p = J.order[w];
    const StripShape h = strip_shape_of<SPARSE>(J, p, w);
    ulonglong2* rows = reinterpret_cast<ulonglong2*>(J.arena + strip_slot_offset(J.slots[w]));
    const int64_t n = (int64_t)(strip_rows_bytes(h) / 16);
    for (int64_t i = (int64_t)blockIdx.y * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.y * blockDim.x)
      rows[i] = make_ulonglong2(kStUnwritten, kStUnwritten);
  }
}

template <bool BITS>
struct StripConst {
  static constexpr int32_t scale = BITS ? 16 : 1;
  static constexpr int32_t neg = BITS ? -(1 << 30) : kNeg;  // never added to
  static constexpr int32_t open_d = kOpen2 * scale + (BITS ? 3 : 0);
  static constexpr int32_t open_i = kOpen2 * scale + (BITS ? 6 : 0);
  static constexpr int32_t d_tag = BITS ? 1 : 0;
};

// One lane's rows at one column.  up: V above-left of row 0; D: D~ of row 0.
// Leaves the D~ of the row below in D and the nibbles in bits 32 - 4R .. 31.
// cap: the row whose (Mg, D~, I~) go to e (-1: none).
template <int R, bool BITS, bool CAP>
__device__ __forceinline__ void strip_column(int32_t (&V)[R], int32_t (&I)[R], const int32_t (&sc)[R], int32_t up,
                                             int32_t& D, uint32_t& nib, int cap, int32_t (&e)[3]) {
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int32_t M = up + sc[r];
    const int32_t v = __vimax3_s32(M, D, I[r]);
    if (CAP && r == cap) {
      e[0] = M;
      e[1] = D;
      e[2] = I[r];
    }
    const int32_t nd = __viaddmax_s32(M, StripConst<BITS>::open_d, D);
    const int32_t ni = __viaddmax_s32(M, StripConst<BITS>::open_i, I[r]);
    up = V[r];
    if (BITS) {
      nib = __funnelshift_r(nib, (uint32_t)(v ^ nd ^ ni), 4);
      V[r] = v & ~3;
      D = nd & ~4;
      I[r] = ni & ~8;
    } else {
      V[r] = v;
      D = nd;
      I[r] = ni;
    }
  }
}

// Shared memory of one warp: the profile and 32 columns of input (V and D~ of
// the row above, and 512 times the base's code).
struct StripSmem {
  int4 prof[8][32];  // [4 * (row / 4) + base][lane]: the scores of four rows
  int4 ring[32];
};

// Lane 0's input of step s in place of what the shuffles brought it.
__device__ __forceinline__ void strip_input(const StripSmem& sm, int s, int lane, int32_t& V, int32_t& D, uint32_t& sel) {
  const uint32_t at = (uint32_t)__cvta_generic_to_shared(&sm.ring[s & 31]);
  asm volatile(
      "{.reg .pred p; .reg .b32 t; setp.eq.s32 p, %4, 0; @p ld.shared.v4.b32 {%0, %1, %2, t}, [%3];}"
      : "+r"(V), "+r"(D), "+r"(sel)
      : "r"(at), "r"(lane)
      : "memory");
}

template <int R, bool BITS>
__device__ __forceinline__ void strip_profile(StripSmem& sm, const uint8_t* A, int row0, int LA) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int q = 0; q < R / 4; ++q) {
    uint32_t row[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = row0 + lane * R + 4 * q + r;
      row[r] = c_score_rows[(i < LA ? A[i] : 0u) & 3u];
    }
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      int32_t s[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        s[r] = (int32_t)((row[r] >> (8 * b)) & 255u) - kScoreBias;
        if (BITS) s[r] = s[r] * 16 + 2;
      }
      sm.prof[4 * q + b][lane] = make_int4(s[0], s[1], s[2], s[3]);
    }
  }
}

template <int R>
__device__ __forceinline__ void strip_scores(const StripSmem& sm, uint32_t sel, int32_t (&sc)[R]) {
  const char* at = reinterpret_cast<const char*>(&sm.prof[0][threadIdx.x & 31]) + sel;
#pragma unroll
  for (int q = 0; q < R / 4; ++q) {
    const int4 v = *reinterpret_cast<const int4*>(at + q * 2048);
    sc[4 * q] = v.x;
    sc[4 * q + 1] = v.y;
    sc[4 * q + 2] = v.z;
    sc[4 * q + 3] = v.w;
  }
}

// A direct slot's nibbles: 4R bits per lane and step, lane-minor.
template <int R>
__device__ __forceinline__ void store_nibbles(void* bits, int64_t at, uint32_t nib) {
  if (R == 8)
    reinterpret_cast<uint32_t*>(bits)[at] = nib;
  else
    reinterpret_cast<uint16_t*>(bits)[at] = (uint16_t)(nib >> 16);
}

// Runs strip k; piped: the previous strip may still be running.  False: a
// wait gave up.
template <int R, bool BITS>
__device__ bool strip_run(const StripJob& J, StripSmem& sm, const StripShape& h, uint8_t* slot, uint32_t p, int k,
                          bool piped) {
  using C = StripConst<BITS>;
  const int lane = threadIdx.x & 31;
  const int LA = h.LA, LB = h.LB, S = h.S;
  const uint8_t* B = J.sb + J.ob[p];
  unsigned long long* rows = reinterpret_cast<unsigned long long*>(slot);
  const unsigned long long* row_in = rows + (int64_t)(k - 1) * LB;
  unsigned long long* row_out = rows + (int64_t)k * LB;
  uint8_t* rest = slot + strip_rows_bytes(h);
  const int row0 = k * 32 * R;
  __syncwarp();
  strip_profile<R, BITS>(sm, J.sa + J.oa[p], row0, LA);

  // the next 32 columns' input, fetched a chunk ahead: V (low word) and D~ of
  // the row above, the base
  unsigned long long above = 0;
  uint32_t code = 0;
  auto load_row = [&](int x) {
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(above) : "l"(row_in + x) : "memory");
  };
  auto fetch = [&](int x) {
    if (x >= LB) return;
    if (k > 0) load_row(x);
    code = B[x] & 3u;
  };
  auto stage = [&](int x) -> bool {
    if (piped && k > 0) {
      bool missing = x < LB && above == kStUnwritten;
      for (long long spins = 0; __ballot_sync(0xffffffffu, missing);) {
        spins += 32;  // a poll of L2 takes as long as some tens of polls of shared memory
        int stop = lane == 0 && (spins > J.spin_limit || *(volatile unsigned*)&J.counter[1]);
        if (__shfl_sync(0xffffffffu, stop, 0)) {
          if (lane == 0) {
            *(volatile unsigned*)&J.counter[1] = 1u;
            set_error(J.err, kDevWatchdog);
          }
          return false;
        }
        __nanosleep(40);
        if (missing) {
          load_row(x);
          missing = above == kStUnwritten;
        }
      }
    }
    int4 v = make_int4(kOpen2 * C::scale, C::neg | C::d_tag, (int)(code * 512u), 0);
    if (k > 0) {
      v.x = (int32_t)(uint32_t)above;
      v.y = (int32_t)(uint32_t)(above >> 32);
    }
    __syncwarp();
    sm.ring[x & 31] = v;
    __syncwarp();
    return true;
  };
  fetch(lane);

  int32_t V[R], I[R], e[3] = {0, 0, 0};
#pragma unroll
  for (int r = 0; r < R; ++r) {
    V[r] = kOpen2 * C::scale;
    I[r] = C::neg;
  }
  int32_t dg = (k == 0 && lane == 0 && LA > 1 ? kGap : kOpen2) * C::scale;
  int32_t D = 0;
  uint32_t sel = 0;
  const bool writes = lane == 31 && k + 1 < h.n;
  const int cap_row = k == h.n - 1 && lane == (LA - 1 - row0) / R ? (LA - 1 - row0) % R : -1;

  auto step = [&](int s, auto checked) {
    constexpr bool kChecked = decltype(checked)::value;
    int32_t uV = __shfl_up_sync(0xffffffffu, V[R - 1], 1);
    int32_t uD = __shfl_up_sync(0xffffffffu, D, 1);
    sel = __shfl_up_sync(0xffffffffu, sel, 1);
    strip_input(sm, s, lane, uV, uD, sel);
    const int x = s - lane;
    if (!kChecked || (x >= 0 && x < LB)) {
      int32_t sc[R];
      strip_scores<R>(sm, sel, sc);
      uint32_t nib = 0;
      D = uD;
      strip_column<R, BITS, kChecked>(V, I, sc, dg, D, nib, kChecked && x == LB - 1 ? cap_row : -1, e);
      dg = uV;
      if (writes)
        asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(row_out + x),
                     "l"((unsigned long long)(uint32_t)V[R - 1] | (unsigned long long)(uint32_t)D << 32)
                     : "memory");
      if (BITS) store_nibbles<R>(rest, ((int64_t)k * S + s) * 32 + lane, nib);
    }
  };

  for (int s0 = 0; s0 < S; s0 += 32) {
    if (!stage(s0 + lane)) return false;
    fetch(s0 + 32 + lane);
    if (!BITS && s0 > 0 && (s0 & ((1 << h.every) - 1)) == 0) {
      int2* st = reinterpret_cast<int2*>(rest) +
                 ((int64_t)k * strip_states(h) + (s0 >> h.every) - 1) * ((R + 1) * 32) + lane;
#pragma unroll
      for (int r = 0; r < R; ++r) st[r * 32] = make_int2(V[r], I[r]);
      st[R * 32] = make_int2(dg, D);
    }
    if (s0 >= 32 && s0 + 32 < LB) {
#pragma unroll 16
      for (int q = 0; q < 32; ++q) step(s0 + q, std::false_type{});
    } else {
      const int end = S - s0 < 32 ? S - s0 : 32;
#pragma unroll 1
      for (int q = 0; q < end; ++q) step(s0 + q, std::true_type{});
    }
  }
  if (cap_row >= 0) {
    int32_t sc = e[0], eD = e[1], eI = e[2];
    if (BITS) {
      sc >>= 4;
      eD >>= 4;
      eI >>= 4;
    }
    sc -= kGap;
    char edge = 'M';
    if (eD - kOpen2 > sc) {
      sc = eD - kOpen2;
      edge = 'D';
    }
    if (eI - kOpen2 > sc) {
      sc = eI - kOpen2;
      edge = 'I';
    }
    J.scores[p] = sc;
    J.end_edge[p] = (uint8_t)edge;
  }
  return true;
}

// 5 CTAs of 4 warps per SM and 16 steps unrolled (96 registers): on the
// 4,000-pair batch 22.7 ms against 23.8 at 4 steps, 24.5 at 7 CTAs and 4 steps
// (72 registers) and 32.5 at 9 CTAs; 2 or 8 warps per CTA measure the same.
template <bool SPARSE>
__global__ void __launch_bounds__(kStWarps * 32, 5) k_gapdp_strips(StripJob J) {
  __shared__ StripSmem smem[kStWarps];
  const int lane = threadIdx.x & 31;
  StripSmem& sm = smem[threadIdx.x >> 5];
  for (;;) {
    int u = 0;
    if (lane == 0) u = (int)atomicAdd(&J.counter[0], 1u);
    u = __shfl_sync(0xffffffffu, u, 0);
    const bool piped = u < J.nunits;
    const uint2 unit = piped ? J.units[u] : make_uint2((uint32_t)(J.npipe + (u - J.nunits)), 0u);
    const int w = (int)unit.x;
    if (w >= J.nwork) break;
    const uint32_t p = J.order[w];
    const StripShape h = strip_shape_of<SPARSE>(J, p, w);
    uint8_t* slot = J.arena + strip_slot_offset(J.slots[w]);
    int k = (int)unit.y;
    const int end = piped ? k + 1 : h.n;
    bool ok = true;
    for (; k < end && ok; ++k) {
      if (h.R == 8)
        ok = h.direct ? strip_run<8, true>(J, sm, h, slot, p, k, piped) : strip_run<8, false>(J, sm, h, slot, p, k, piped);
      else
        ok = h.direct ? strip_run<4, true>(J, sm, h, slot, p, k, piped) : strip_run<4, false>(J, sm, h, slot, p, k, piped);
    }
    if (!ok) break;
  }
}

// ------------------------------------------------------------- traceback

// BitTraceBack (MU/bittraceback.cpp:138-210).  The walk needs the nibbles of
// the cells it arrives at, kStBlock steps of a strip at a time.  Inside what
// is in shared memory a whole run of equal moves is found at once: lane l
// looks at the cell l + 1 moves on, and a ballot gives the run's length.
//
// A direct problem is walked by one warp, which copies its blocks to shared
// memory.  A checkpointed problem is walked by a CTA: its blocks are computed
// again from the stored states and the row above with the forward pass's
// recurrences, on values relative to one of the block's (so that scaled
// scores fit 32 bits at any length).  A path crosses a strip of 256 rows in
// about 290 steps, so the kWalkWarps blocks up to the walk's step are
// computed at once, one per warp, and the first warp walks them: a block is a
// serial chain of 64 steps, and the longest paths, which end the pass, took
// one such chain per block when one warp did everything.
constexpr int kWalkWarps = 512 / kStBlock;
struct WalkJob {
  const uint8_t* sa;
  const uint64_t* oa;
  const uint8_t* sb;
  const uint64_t* ob;
  const uint32_t* order;
  const uint64_t* slots;
  const uint32_t* todo;  // slots: the first nck checkpointed, the others direct, each part largest first
  int nwork, nck, max_rows;
  bool ckpt;
  const uint8_t* arena;
  const uint8_t* end_edge;
  const uint64_t* path_off;
  char* paths;
  int64_t* path_len;
  uint32_t* err;
  int32_t* env;  // optional: the path's extreme deviations from the diagonal
  unsigned* counter;  // [0] claims of CTAs, [1] claims of warps
};

struct WalkSmem {
  StripSmem strip[kWalkWarps];
  uint32_t nib[kWalkWarps * kStBlock * 32];  // [step][lane] (uint16_t for R = 4); direct: a block per warp
  int claim, want_k, want_s, want_n;         // a CTA's problem; the strip, the step and the blocks it walks
  int64_t path_n;
};
constexpr size_t kWalkSmem = sizeof(WalkSmem);

// The state of strip k at step s0 from the one at step sa (st; null: the
// strip's start), left in sm.prof as a stored state: for slots whose states are
// some blocks apart.  Not inlined, and without the caller's structures: this is
// the exception, walk_block's registers are the rule's.
template <int R>
__device__ __noinline__ void walk_to(StripSmem& sm, const uint8_t* A, int LA, const uint8_t* B, int LB,
                                     const int2* row_in, const int2* st, int k, int sa, int s0) {
  const int lane = threadIdx.x & 31;
  int32_t V[R], I[R], dg = k == 0 && lane == 0 && LA > 1 ? kGap : kOpen2, D = 0, e[3];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int2 v = st ? st[r * 32] : make_int2(kOpen2, kNeg);
    V[r] = v.x;
    I[r] = v.y;
  }
  if (st) {
    dg = st[R * 32].x;
    D = st[R * 32].y;
  }
  __syncwarp();
  strip_profile<R, false>(sm, A, k * 32 * R, LA);
  const int x0 = sa - 1 - lane;
  uint32_t sel = x0 >= 0 && x0 < LB ? (B[x0] & 3u) * 512u : 0u;
  for (int c = sa; c < s0; c += 32) {
    const int xc = c + lane;
    int4 in = make_int4(kOpen2, kNeg, 0, 0);
    if (xc < LB) {
      if (k > 0) {
        const int2 above = row_in[xc];
        in.x = above.x;
        in.y = above.y;
      }
      in.z = (int)((B[xc] & 3u) * 512u);
    }
    __syncwarp();
    sm.ring[xc & 31] = in;
    __syncwarp();
#pragma unroll 1
    for (int q = 0; q < 32; ++q) {
      int32_t uV = __shfl_up_sync(0xffffffffu, V[R - 1], 1);
      int32_t uD = __shfl_up_sync(0xffffffffu, D, 1);
      sel = __shfl_up_sync(0xffffffffu, sel, 1);
      strip_input(sm, c + q, lane, uV, uD, sel);
      const int x = c + q - lane;
      if (x >= 0 && x < LB) {
        int32_t sc[R];
        strip_scores<R>(sm, sel, sc);
        uint32_t nib = 0;
        D = uD;
        strip_column<R, false, false>(V, I, sc, dg, D, nib, -1, e);
        dg = uV;
      }
    }
  }
  __syncwarp();
  int2* to = reinterpret_cast<int2*>(sm.prof) + lane;
  static_assert((R + 1) * 32 * 8 <= sizeof(sm.prof), "a state fits the profile");
#pragma unroll
  for (int r = 0; r < R; ++r) to[r * 32] = make_int2(V[r], I[r]);
  to[R * 32] = make_int2(dg, D);
}

// Steps s0 .. s1 of strip k computed again; step s goes to nib[s & mask].
template <int R, bool SPARSE>
__device__ void walk_block(const WalkJob& J, StripSmem& sm, void* nibs, int mask, const StripShape& h,
                           const uint8_t* slot, uint32_t p, int k, int s0, int s1) {
  const int lane = threadIdx.x & 31;
  const int LB = h.LB;
  const uint8_t* B = J.sb + J.ob[p];
  const int2* row_in = reinterpret_cast<const int2*>(slot) + (int64_t)(k - 1) * LB;
  int32_t V[R], I[R], dg, D, e[3];
  if (s0 == 0) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      V[r] = kOpen2;
      I[r] = kNeg;
    }
    dg = k == 0 && lane == 0 && h.LA > 1 ? kGap : kOpen2;
    D = 0;
  } else {
    const int sa = SPARSE ? s0 & ~((1 << h.every) - 1) : s0;
    const int2* st = reinterpret_cast<const int2*>(slot + strip_rows_bytes(h)) +
                     ((int64_t)k * strip_states(h) + (sa >> h.every) - 1) * ((R + 1) * 32) + lane;
    if (SPARSE && sa != s0) {
      walk_to<R>(sm, J.sa + J.oa[p], h.LA, B, LB, row_in, sa > 0 ? st : nullptr, k, sa, s0);
      st = reinterpret_cast<const int2*>(sm.prof) + lane;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int2 v = st[r * 32];
      V[r] = v.x;
      I[r] = v.y;
    }
    const int2 v = st[R * 32];
    dg = v.x;
    D = v.y;
  }
  int2 above = make_int2(kOpen2, kNeg);
  uint32_t code = 0;
  auto fetch = [&](int x) {
    if (x >= LB || x > s1) return;
    if (k > 0) above = row_in[x];
    code = B[x] & 3u;
  };
  fetch(s0 + lane);
  __syncwarp();
  strip_profile<R, true>(sm, J.sa + J.oa[p], k * 32 * R, h.LA);
  const int32_t base = __shfl_sync(0xffffffffu, V[R - 1], 0);
  auto scaled = [&](int32_t v) { return max(v - base, -(1 << 26)) * 16; };
#pragma unroll
  for (int r = 0; r < R; ++r) {
    V[r] = scaled(V[r]);
    I[r] = scaled(I[r]);
  }
  dg = scaled(dg);
  D = scaled(D) | 1;
  // the base of the column each lane has just left (lane t - 1 hands it on)
  const int x0 = s0 - 1 - lane;
  uint32_t sel = x0 >= 0 && x0 < LB ? (B[x0] & 3u) * 512u : 0u;
  auto step = [&](int s, auto checked) {
    int32_t uV = __shfl_up_sync(0xffffffffu, V[R - 1], 1);
    int32_t uD = __shfl_up_sync(0xffffffffu, D, 1);
    sel = __shfl_up_sync(0xffffffffu, sel, 1);
    strip_input(sm, s, lane, uV, uD, sel);
    const int x = s - lane;
    if (!decltype(checked)::value || (x >= 0 && x < LB)) {
      int32_t sc[R];
      strip_scores<R>(sm, sel, sc);
      uint32_t nib = 0;
      D = uD;
      strip_column<R, true, false>(V, I, sc, dg, D, nib, -1, e);
      dg = uV;
      store_nibbles<R>(nibs, (s & mask) * 32 + lane, nib);
    }
  };
  for (int c = s0; c <= s1; c += 32) {
    __syncwarp();
    sm.ring[(c + lane) & 31] = make_int4(scaled(above.x), scaled(above.y) | 1, (int)(code * 512u), 0);
    __syncwarp();
    fetch(c + 32 + lane);
    if (c >= 32 && c + 32 <= LB && c + 31 <= s1) {
#pragma unroll 2
      for (int q = 0; q < 32; ++q) step(c + q, std::false_type{});
    } else {
      const int end = s1 - c < 31 ? s1 - c + 1 : 32;
#pragma unroll 1
      for (int q = 0; q < end; ++q) step(c + q, std::true_type{});
    }
  }
}

// The walk.  COOP: the CTA's first warp walks while the others wait in
// walk_help for the steps it wants.  Returns the path's length, 0 on failure.
template <int R, bool SPARSE, bool COOP>
__device__ int64_t walk_path(const WalkJob& J, WalkSmem& sm, const StripShape& h, const uint8_t* slot, uint32_t p) {
  constexpr int SR = 32 * R;
  constexpr int kMask = COOP ? kWalkWarps * kStBlock - 1 : kStBlock - 1;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  uint32_t* nibs = COOP ? sm.nib : sm.nib + wib * kStBlock * 32;
  const int LA = h.LA, LB = h.LB;
  const int64_t limit = (int64_t)LA + LB;
  char* path = J.paths + J.path_off[p];
  int pa = LA, pb = LB;
  char X = (char)J.end_edge[p];
  int64_t n = 0;
  int row0 = LA, s0 = 0, s1 = -1;  // what is in shared memory (nothing yet): first row - 1, steps
  int32_t dev_lo = INT32_MAX, dev_hi = INT32_MIN;
  bool fail = false;
  // X at the cells (pa - l*di, pb - l*dj), l < count (one l per lane)
  auto emit = [&](int l, int count, int di, int dj) {
    if (l >= count) return;
    path[limit - n - 1 - l] = X;
    const int i = pa - l * di;
    if (J.env && i >= 1) {
      const int32_t dv = (pb - l * dj) - (int32_t)((int64_t)i * LB / LA);
      dev_lo = min(dev_lo, dv);
      dev_hi = max(dev_hi, dv);
    }
  };
  auto nibble = [&](int i, int s) -> uint32_t {  // row i of the strip (from 0) at step s
    const int at = (s & kMask) * 32 + i / R;
    const uint32_t word = R == 8 ? nibs[at] : reinterpret_cast<const uint16_t*>(nibs)[at];
    return (word >> (4 * (i % R))) & 15u;
  };
  for (;;) {
    const int di = X != 'I', dj = X != 'D';
    const int i = pa - di * (lane + 1) - 1 - row0, x = pb - dj * (lane + 1) - 1;
    bool valid = false, more = false;
    uint32_t bits = 0;
    if (i >= 0 && x >= 0) {
      const int s = x + i / R;
      if (s >= s0 && s <= s1) {
        valid = true;
        bits = nibble(i, s);
        more = X == 'M' ? (bits & 3u) == 3u : X == 'D' ? !(bits & 4u) : !(bits & 8u);
      }
    }
    const uint32_t stop = ~__ballot_sync(0xffffffffu, more);
    const int run = stop ? __ffs(stop) - 1 : 32;
    const int count = run < 32 ? run + 1 : 32;
    if (n + count > limit) {
      fail = true;
      break;
    }
    emit(lane, count, di, dj);
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
      for (int l = lane; l < rest; l += 32) emit(l, rest, pa > 0, pb > 0);
      n += rest;
      break;
    }
    if (!valid) {
      const int k = (pa - 1) / SR;
      row0 = k * SR;
      s1 = pb - 1 + (pa - 1 - row0) / R;
      s0 = s1 & ~(kStBlock - 1);
      if (COOP) {
        // the steps a path along the problem's slope takes to leave the strip
        const int64_t steps = (int64_t)SR * LB / LA + 31 + 16;
        const int nblk = (int)min((int64_t)kWalkWarps, (int64_t)(s1 / kStBlock) - (s1 - steps < 0 ? 0 : (s1 - steps) / kStBlock) + 1);
        if (lane == 0) {
          sm.want_k = k;
          sm.want_s = s1;
          sm.want_n = nblk;
        }
        __syncthreads();
        walk_block<R, SPARSE>(J, sm.strip[0], sm.nib, kMask, h, slot, p, k, s0, s1);
        __syncthreads();
        s0 -= (nblk - 1) * kStBlock;
      } else {
        __syncwarp();
        const int4* src = reinterpret_cast<const int4*>(slot + strip_rows_bytes(h) + ((int64_t)k * h.S + s0) * (16 * R));
        int4* dst = reinterpret_cast<int4*>(nibs);
        for (int q = lane; q < (s1 - s0 + 1) * R; q += 32) dst[q] = src[q];
        __syncwarp();
      }
      bits = nibble(pa - 1 - row0, s1);
    }
    if (X == 'M')
      X = (bits & 3u) == 3u ? 'M' : (bits & 3u) == 0u ? 'D' : 'I';
    else
      X = (bits & (X == 'D' ? 4u : 8u)) ? 'M' : X;
  }
  if (fail && lane == 0) set_error(J.err, kDevCapacity);
  if (lane == 0) J.path_len[p] = n;
  if (J.env) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      dev_lo = min(dev_lo, __shfl_xor_sync(0xffffffffu, dev_lo, d));
      dev_hi = max(dev_hi, __shfl_xor_sync(0xffffffffu, dev_hi, d));
    }
    if (lane == 0) {
      J.env[2 * p] = dev_lo;
      J.env[2 * p + 1] = dev_hi;
    }
  }
  return n;
}

// The CTA's other warps: warp w computes the block w before the walk's.
template <int R, bool SPARSE>
__device__ void walk_help(const WalkJob& J, WalkSmem& sm, const StripShape& h, const uint8_t* slot, uint32_t p) {
  const int w = threadIdx.x >> 5;
  for (;;) {
    __syncthreads();
    const int k = sm.want_k, s0 = (sm.want_s & ~(kStBlock - 1)) - w * kStBlock;
    if (k < 0) return;
    if (w < sm.want_n)
      walk_block<R, SPARSE>(J, sm.strip[w], sm.nib, kWalkWarps * kStBlock - 1, h, slot, p, k, s0, s0 + kStBlock - 1);
    __syncthreads();
  }
}

// A path written from the end of its slot moves to the slot's head; t of nt
// threads, sync between reading and writing a chunk.
template <class F>
__device__ void walk_compact(char* path, int64_t limit, int64_t n, int t, int nt, F sync) {
  const char* src = path + (limit - n);
  if (src == path) return;
  for (int64_t c = 0; c < n; c += 4 * nt) {
    char v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = c + q * nt + t < n ? src[c + q * nt + t] : 0;
    sync();
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (c + q * nt + t < n) path[c + q * nt + t] = v[q];
    sync();
  }
}

template <bool SPARSE>
__global__ void __launch_bounds__(kWalkWarps * 32) k_strip_walk(WalkJob J) {
  extern __shared__ __align__(16) uint8_t walk_smem[];
  WalkSmem& sm = *reinterpret_cast<WalkSmem*>(walk_smem);
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  if (*(volatile uint32_t*)J.err == kDevWatchdog) return;  // the forward pass stopped early
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) sm.claim = (int)atomicAdd(&J.counter[0], 1u);
    __syncthreads();
    if (sm.claim >= J.nck) break;
    const int w = (int)J.todo[sm.claim];
    const uint32_t p = J.order[w];
    const StripShape h = strip_shape_of<SPARSE>(J, p, w);
    const uint8_t* slot = J.arena + strip_slot_offset(J.slots[w]);
    if (wib == 0) {
      const int64_t n =
          h.R == 8 ? walk_path<8, SPARSE, true>(J, sm, h, slot, p) : walk_path<4, SPARSE, true>(J, sm, h, slot, p);
      if (lane == 0) {
        sm.want_k = -1;
        sm.path_n = n;
      }
      __syncthreads();
    } else if (h.R == 8) {
      walk_help<8, SPARSE>(J, sm, h, slot, p);
    } else {
      walk_help<4, SPARSE>(J, sm, h, slot, p);
    }
    walk_compact(J.paths + J.path_off[p], (int64_t)h.LA + h.LB, sm.path_n, (int)threadIdx.x, kWalkWarps * 32,
                 [] { __syncthreads(); });
  }
  for (;;) {
    int q = 0;
    if (lane == 0) q = J.nck + (int)atomicAdd(&J.counter[1], 1u);
    q = __shfl_sync(0xffffffffu, q, 0);
    if (q >= J.nwork) break;
    const int w = (int)J.todo[q];
    const uint32_t p = J.order[w];
    const StripShape h = strip_shape_of<SPARSE>(J, p, w);
    const uint8_t* slot = J.arena + strip_slot_offset(J.slots[w]);
    const int64_t n =
        h.R == 8 ? walk_path<8, SPARSE, false>(J, sm, h, slot, p) : walk_path<4, SPARSE, false>(J, sm, h, slot, p);
    __syncwarp();
    walk_compact(J.paths + J.path_off[p], (int64_t)h.LA + h.LB, n, lane, 32, [] { __syncwarp(); });
  }
}

}  // namespace mvg
