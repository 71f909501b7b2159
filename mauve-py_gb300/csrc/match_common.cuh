// Device-side pieces of the seed matcher shared by the genome-pair matcher
// (match.cu) and the batched gap anchor search (gapsearch.cu): the hash
// entry, its order, the unique-seed run test and ExtendMatch's walk.
#pragma once
#include "mvg_internal.h"
#include "prim.cuh"

namespace mvg {

constexpr int kTableSize = 40000;  // LM/MemHash.h:30 DEFAULT_MEM_TABLE_SIZE

struct Mhe {
  int64_t s0, s1, len;
};

struct MatchCtx {
  const uint32_t* g[2];
  int64_t n[2];
  SeedDesc s;
};

// The same with the seed elsewhere (one of many).
struct MatchView {
  const uint32_t* g[2];
  int64_t n[2];
  const SeedDesc& s;
};

// ------------------------------------------------------------------ join

// Both genomes' seeds sorted in one array by (seed bits, strand, genome).  A
// seed unique in each genome (counted once in each, strand ignored:
// LM/PairwiseMatchFinder.cpp:37-71 over LM/MatchFinder.cpp:172-340) is a run
// of equal seed bits with exactly two members, one per genome; runs come in
// ascending seed order, the reference's enumeration order.  Key i opens such
// a run when pair_flag(i).
template <typename K>
__device__ __forceinline__ bool pair_flag(const K* __restrict__ keys, int64_t n, int64_t i) {
  const uint64_t k0 = (uint64_t)keys[i], cur = k0 >> 2;
  if (i + 1 >= n || (i > 0 && ((uint64_t)keys[i - 1] >> 2) == cur)) return false;
  const uint64_t k1 = (uint64_t)keys[i + 1];
  return (k1 >> 2) == cur && ((k0 ^ k1) & 1ull) && (i + 2 == n || ((uint64_t)keys[i + 2] >> 2) != cur);
}

// ------------------------------------------------------ hash entries

// LM/MatchHashEntry.cpp:48-67 (strict_start_lessthan_ptr).
__device__ __forceinline__ bool mhe_strict_lt(const Mhe& a, const Mhe& b, int L) {
  int64_t x = a.s0 < 0 ? -a.s0 + a.len - L : a.s0;
  int64_t y = b.s0 < 0 ? -b.s0 + b.len - L : b.s0;
  if (x != y) return x < y;
  x = a.s1 < 0 ? -a.s1 + a.len - L : a.s1;
  y = b.s1 < 0 ? -b.s1 + b.len - L : b.s1;
  if (x != y) return x < y;
  return false;
}

// ExtendMatch (LM/MatchFinder.h:218-374) for two genomes.  The reference cycles
// through four phases (jump left and right by the seed length until the first mismatching window, then try the L
// single-base offsets left and right and move to the furthest matching one)
// and restarts while a single-base phase moves.
//
// Every window pair a phase tests lies on the match's diagonal: in the entry
// orientation S0, the pair tested at step size k from the current left edge
// is the pair at displacement ML + k from the entry left edge (ML = total
// moved in even phases), and in the inverted orientation the pair at MR + k
// from the entry right edge (MR = total moved in odd phases); positive
// starts move by exactly those amounts and negative starts stay.  The room
// a phase has (the genome-end clamp) is likewise C - ML or C' - MR.  So the
// two sides never interact: each side's total is where its own walk stops.
// The match bits come 32 displacements at a time (ext_word), and each pair of
// words is searched for the stop (stop_in_word).  For a same-strand pair a window pair matches iff the
// pattern-selected bases are equal (equal canonical mers with equal strand
// bits); other pairs use the canonical-mer test itself.
// Window start (0-based) in genome q of the pair at displacement u from the
// entry state's edge (st, len), or -1 outside the genome.
__device__ __forceinline__ int64_t ext_start(int64_t st, int64_t len, int64_t u, int L, int64_t n) {
  if (st > 0 && u >= st) return -1;  // a left step past the genome start (the phases never take it)
  const int64_t sq = st > 0 ? st - u : st;
  const int64_t get = sq < 0 ? -sq + len + u - L : sq;
  const int64_t x = get - 1;
  return (x >= 0 && x + L <= n) ? x : -1;
}

// 64 bases (128 bits, big-endian, base p in bits 127:126) from 2-bit words;
// reads words p/16 .. p/16 + 4.
__device__ __forceinline__ void window128(const uint32_t* __restrict__ g, uint64_t p, uint64_t& hi, uint64_t& lo) {
  const uint64_t q = p >> 4;
  const uint32_t sh = (uint32_t)(p & 15) * 2;
  const uint64_t H = ((uint64_t)__ldg(g + q) << 32) | __ldg(g + q + 1);
  const uint64_t M = ((uint64_t)__ldg(g + q + 2) << 32) | __ldg(g + q + 3);
  const uint32_t T = __ldg(g + q + 4);
  if (sh == 0) {
    hi = H;
    lo = M;
  } else {
    hi = (H << sh) | (M >> (64 - sh));
    lo = (M << sh) | (uint64_t)(T >> (32 - sh));
  }
}

// Reverse complement of 32 bases in 64 bits (complement = the 2-bit code
// inverted; base order reversed).
__device__ __forceinline__ uint64_t revcomp64(uint64_t x) {
  const uint64_t r = __brevll(~x);  // groups reversed, bits inside groups swapped
  return ((r >> 1) & 0x5555555555555555ull) | ((r & 0x5555555555555555ull) << 1);
}

// The top 64 bits of the 128-bit value hi:lo shifted left by s (0 <= s < 128).
__device__ __forceinline__ uint64_t top64(uint64_t hi, uint64_t lo, int s) {
  if (s == 0) return hi;
  if (s < 64) return (hi << s) | (lo >> (64 - s));
  return lo << (s - 64);
}

// The even bits of x, packed (bit 2k to bit k).
__device__ __forceinline__ uint32_t even_bits(uint64_t x) {
  x &= 0x5555555555555555ull;
  x = (x | (x >> 1)) & 0x3333333333333333ull;
  x = (x | (x >> 2)) & 0x0f0f0f0f0f0f0f0full;
  x = (x | (x >> 4)) & 0x00ff00ff00ff00ffull;
  x = (x | (x >> 8)) & 0x0000ffff0000ffffull;
  return (uint32_t)(x | (x >> 16));
}

// Match bits of displacements U .. U + 31.  Same-strand windows, and with a
// symmetric pattern opposite-strand ones, are read as one 64-base stretch of
// each genome: one exclusive or gives the differing bases, and an or of that
// mask shifted by each selected base of the pattern tells for 32 windows at
// once whether a selected base differs (about 150 instructions; 32 masked
// 64-bit comparisons took 400).
template <class C>  // MatchCtx or MatchView
__device__ __forceinline__ uint32_t ext_word(const C& c, int64_t st0, int64_t st1, int64_t len, int64_t U) {
  const int L = c.s.L;
  const uint64_t pmask = c.s.base_mask;
  const bool same = (st0 > 0) == (st1 > 0);
  uint32_t word = 0;
  if (same || c.s.sym) {
    // Opposite strands with a symmetric pattern: the reference's test is
    // "canonical mers equal and strands opposite", which for a mer set
    // {f, rc(f)} means: B's forward mer is the reverse complement of A's, and
    // A's mer is not its own reverse complement (then both canonical forms
    // are the forward one).  With a symmetric pattern rc(mer(x)) =
    // mer(rc(x)), so both are masked window comparisons: A's window against
    // the reverse complement of B's (which moves the same way as A's, at a
    // fixed offset), and, where that holds, A's window against its own
    // reverse complement.
    const int64_t a0 = ext_start(st0, len, U, L, c.n[0]), a31 = ext_start(st0, len, U + 31, L, c.n[0]);
    const int64_t b0 = ext_start(st1, len, U, L, c.n[1]), b31 = ext_start(st1, len, U + 31, L, c.n[1]);
    const bool adown = st0 > 0, bdown = st1 > 0;  // window starts decrease with u
    const int64_t amin = adown ? a31 : a0, bmin = bdown ? b31 : b0;
    if (a0 >= 0 && a31 >= 0 && b0 >= 0 && b31 >= 0 && amin + 80 <= c.n[0] && bmin + 80 <= c.n[1]) {
      uint64_t ah, al, bh, bl;
      window128(c.g[0], (uint64_t)amin, ah, al);
      window128(c.g[1], (uint64_t)bmin, bh, bl);
      uint64_t oh = bh, ol = bl;  // what A's bases are compared with
      if (!same) {
        // reverse complement of B's stretch; A's window at j meets its window at j + 33 - L
        const uint64_t rh = revcomp64(bl), rl = revcomp64(bh);
        const int sh = 2 * (33 - L);
        oh = top64(rh, rl, sh);
        ol = sh < 64 ? rl << sh : 0ull;
      }
      const uint64_t dh = ah ^ oh, dl = al ^ ol;
      // bit 63 - k: base k differs
      const uint64_t diff = (uint64_t)even_bits(dh | dh >> 1) << 32 | even_bits(dl | dl >> 1);
      const uint32_t d1 = (uint32_t)(diff >> 32), d0 = (uint32_t)diff;
      uint32_t bad = 0;  // bit 31 - j: window j has a selected base that differs
      for (uint32_t p = __brev((uint32_t)c.s.pattern) >> (32 - L); p; p &= p - 1)
        bad |= __funnelshift_l(d0, d1, __ffs(p) - 1);
      word = adown ? ~bad : __brev(~bad);
      if (!same) {
        const uint64_t rah = revcomp64(al), ral = revcomp64(ah);
        for (uint32_t todo = word; todo; todo &= todo - 1) {
          const int t = __ffs(todo) - 1, ja = adown ? 31 - t : t;
          if (((top64(ah, al, 2 * ja) ^ top64(rah, ral, 2 * (64 - L - ja))) & pmask) == 0) word &= ~(1u << t);
        }
      }
      if (U == 0) word &= ~1u;  // displacement 0 is not a step
      return word;
    }
  }
  for (int t = 0; t < 32; ++t) {
    const int64_t u = U + t;
    const int64_t xa = ext_start(st0, len, u, L, c.n[0]);
    const int64_t xb = ext_start(st1, len, u, L, c.n[1]);
    bool b = false;
    if (u >= 1 && xa >= 0 && xb >= 0) {
      if (same) {
        b = ((window64(c.g[0], (uint64_t)xa) ^ window64(c.g[1], (uint64_t)xb)) & pmask) == 0;
      } else {
        const uint64_t ca = canonical_mer(c.g[0], (uint64_t)xa, c.s);
        const uint64_t cb = canonical_mer(c.g[1], (uint64_t)xb, c.s);
        const bool pa = st0 > 0 ? !(ca & 1ull) : (bool)(ca & 1ull);
        const bool pb = st1 > 0 ? !(cb & 1ull) : (bool)(cb & 1ull);
        b = (ca & c.s.seed_mask) == (cb & c.s.seed_mask) && pa == pb;
      }
    }
    word |= (uint32_t)b << t;
  }
  return word;
}

// Where a side's walk stops.  On one side of the entry the walk starts at
// displacement 0 and, with bit(u) = "the window pair at displacement u
// matches" (0 beyond the genome ends), jumps by L while the window L further
// matches, then moves to the furthest matching window within L, and repeats.
// Every position it reaches is 0 or a matching window, every move is at most
// L, and it moves on from q exactly when one of bits q+1 .. q+L is set.  So
// it can never pass a run of L clear bits, and it stops at the first
// position q in {0} or the set bits whose next L bits are all clear.  Here
// that q is found word by word: for the 64 bits of words i, i+1, the clear
// runs of length L are the bits of y = AND of L shifts of ~x, and the
// candidates of word i whose next L bits are clear are its set bits (and
// the start) at positions r with bit r+1 of y set.
__device__ __forceinline__ uint32_t stop_in_word(uint32_t w, uint32_t w_next, bool first, int L) {
  uint64_t y = ~(((uint64_t)w_next << 32) | w);
  for (int have = 1; have < L;) {  // y bit j: clear bits j .. j+have-1
    const int sh = have < L - have ? have : L - have;
    y &= y >> sh;
    have += sh;
  }
  return (w | (first ? 1u : 0u)) & (uint32_t)(y >> 1);
}

}  // namespace mvg
