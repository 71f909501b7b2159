// Both gapped-alignment passes of a two-genome progressiveMauve run over
// many LCBs in one call: doGappedAlignment (LM/ProgressiveAligner.cpp:
// 1242-1290) with refineAlignment (:1119-1230), first with profile_aln =
// true (step 8 of alignProfileToProfile, :2560-2565), then with profile_aln
// = false (the final iterative refinement, :3750-3755).
//
// Pass 1: every window of every LCB (lcb_windows) that is not a gap window
// and holds bases of both genomes is cut at MUSCLE's anchor columns
// (anchor_columns) as ProfileAlignFast(anchored) does
// (LM/MuscleInterface.cpp:1053-1109, MU/anchoredpp.cpp:429-552); each range
// of at least one column with bases of both genomes is one gap-DP problem, a
// range with bases of one genome becomes those bases against gaps.  Pass 2:
// RefineFast's column windows (500 or 200 columns of windows of density
// class 1 or 2; MU/refinew.cpp:75-184) with bases of both genomes are one
// problem each, everything else keeps its columns.
//
// Each pass plans on the host (pieces as column ranges, LCBs on host
// threads), compacts the problems' characters straight into the pinned upload
// buffer, runs every problem of every LCB in one batched gap-DP call, rebuilds
// the rows of every problem on the GPU (k_path_rows) and splices them into
// the LCBs' rows, the last pass's into the caller's buffers.  What bounds it
// is this host work: 120 LCBs, 1.44 million columns, take 3.8 ms, of which
// the gap-DP calls are 1.3 (the plans' literal rows, the characters and their
// codes as vectors of their own, grown byte by byte, merged and spliced by way
// of further vectors: 10.3).
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <functional>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

#include "lcb_host.h"
#include "mauve_gb300.h"
#include "mvg_internal.h"

namespace mvg {
namespace {

// 0..3 for A/C/G/T in either case, 4 for a gap character, 8 otherwise.
struct Classes {
  uint8_t of[256];
  Classes() {
    for (int c = 0; c < 256; ++c) of[c] = 8;
    for (int k = 0; k < 4; ++k) of["ACGT"[k] + 0u] = of["acgt"[k] + 0u] = (uint8_t)k;
    of[(int)'-'] = of[(int)'.'] = 4;
  }
};
const Classes kClass;

// A piece of an LCB's new rows, from the columns [lo, hi) of its old ones.
enum PieceKind : uint8_t { kLiteral, kProblem, kOnlyA, kOnlyB };
struct Piece {
  uint64_t lo, hi;
  uint64_t n[2];  // bases of each genome in the range (kLiteral: not set)
  PieceKind kind;
};

// The plan of one LCB: its pieces in column order.
struct Plan {
  std::vector<Piece> pieces;
  uint64_t nprob = 0;
  uint64_t chars[2] = {0, 0};  // its problems' bases

  void add(PieceKind kind, uint64_t lo, uint64_t hi, uint64_t na, uint64_t nb) {
    if (kind == kProblem) {
      ++nprob;
      chars[0] += na;
      chars[1] += nb;
    }
    pieces.push_back(Piece{lo, hi, {na, nb}, kind});
  }
  void add_literal(uint64_t lo, uint64_t hi) {
    if (hi > lo) add(kLiteral, lo, hi, 0, 0);
  }
};

// One LCB's rows and its bases before every column.  The windows' counts
// take any character but '-' for a base; '.' is a gap here as well.
struct Rows {
  const uint8_t *a, *b;
  uint64_t n;
  LcbCounts& pre;
  LcbCounts& dots;  // '.' before every column, empty where a row has none

  Rows(const uint8_t* ra, const uint8_t* rb, uint64_t n_, LcbCounts& p, LcbCounts& d)
      : a(ra), b(rb), n(n_), pre(p), dots(d) {
    for (int q = 0; q < 2; ++q) {
      const uint8_t* r = q ? b : a;
      d[q].clear();
      if (!n || !memchr(r, '.', n)) continue;
      d[q].resize(n + 1);
      uint64_t k = 0;
      for (uint64_t c = 0; c < n; ++c) {
        d[q][c] = k;
        k += r[c] == '.';
      }
      d[q][n] = k;
    }
  }
  uint64_t bases(int q, uint64_t lo, uint64_t hi) const {
    return pre[q][hi] - pre[q][lo] - (dots[q].empty() ? 0 : dots[q][hi] - dots[q][lo]);
  }
};

// A thread's buffers for one call.
struct Scratch {
  LcbCounts pre, dots;
  AnchorScratch anchors;
  std::vector<unsigned> cols;
};

// Pass 1 plan for one LCB.
void plan_anchored(Plan& p, const Rows& r, double maxw, Scratch& s) {
  std::vector<unsigned>& cols = s.cols;
  for (const LcbWindow& w : lcb_windows(r.a, r.b, r.n, maxw, r.pre)) {
    if (w.gap || !r.bases(0, w.lo, w.hi) || !r.bases(1, w.lo, w.hi)) {
      p.add_literal(w.lo, w.hi);
      continue;
    }
    anchor_columns(r.a + w.lo, r.b + w.lo, (unsigned)(w.hi - w.lo), cols, s.anchors);
    uint64_t lo = w.lo;
    for (size_t k = 0; k <= cols.size(); ++k) {
      const uint64_t hi = k < cols.size() ? w.lo + cols[k] : w.hi;
      if (hi <= lo) continue;
      const uint64_t na = r.bases(0, lo, hi), nb = r.bases(1, lo, hi);
      if (na && nb)
        p.add(kProblem, lo, hi, na, nb);
      else if (na || nb)  // the other genome's bases against gaps
        p.add(na ? kOnlyA : kOnlyB, lo, hi, na, nb);
      lo = hi;
    }
  }
}

// Pass 2 plan for one LCB.
void plan_refine(Plan& p, const Rows& r, double maxw) {
  uint64_t at = 0;
  for (const LcbWindow& w : lcb_windows(r.a, r.b, r.n, maxw, r.pre)) {
    const uint64_t width = refine_width(w.density);
    if (w.gap || width == 0) continue;
    for (uint64_t lo = w.lo; lo < w.hi; lo += width) {
      const uint64_t hi = lo + width < w.hi ? lo + width : w.hi;
      p.add_literal(at, lo);
      const uint64_t na = r.bases(0, lo, hi), nb = r.bases(1, lo, hi);
      if (na && nb)
        p.add(kProblem, lo, hi, na, nb);
      else
        p.add_literal(lo, hi);
      at = hi;
    }
  }
  p.add_literal(at, r.n);
}

// The bases of the range, compacted to out (which is written one character past
// them when the range ends in a gap); all classes met, or-ed together.
uint8_t compact(const uint8_t* r, uint64_t lo, uint64_t hi, uint8_t* out) {
  uint8_t seen = 0;
  for (uint64_t c = lo; c < hi; ++c) {
    const uint8_t ch = r[c], cl = kClass.of[ch];
    *out = ch;
    out += cl != 4;
    seen |= cl;
  }
  return seen;
}

// Up to 16 host threads for the length of one call.  run(n, fn) runs
// fn(k, thread) for k in [0, n), threads claiming one index at a time (LCBs
// differ in size), and returns when all are done; it throws bad_alloc when a
// call of fn threw.
class Team {
 public:
  explicit Team(size_t n) {
    const size_t hw = std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
    try {
      pool_.reserve(hw);
      for (size_t t = 1; t < std::min(hw, n); ++t) pool_.emplace_back([this, t] { worker(t); });
    } catch (...) {  // fewer threads, and none to leave behind
    }
  }
  ~Team() {
    {
      std::lock_guard<std::mutex> lk(mu_);
      stop_ = true;
    }
    wake_.notify_all();
    for (std::thread& t : pool_) t.join();
  }
  size_t threads() const { return pool_.size() + 1; }
  using Fn = std::function<void(size_t, size_t)>;
  void run(size_t n, const Fn& fn) {
    {
      std::lock_guard<std::mutex> lk(mu_);
      fn_ = &fn;
      n_ = n;
      next_ = 0;
      busy_ = pool_.size();
      ++round_;
    }
    wake_.notify_all();
    claim(0);
    std::unique_lock<std::mutex> lk(mu_);
    done_.wait(lk, [this] { return busy_ == 0; });
    if (failed_) throw std::bad_alloc();
  }

 private:
  void claim(size_t t) {
    try {
      for (size_t k; (k = next_.fetch_add(1)) < n_;) (*fn_)(k, t);
    } catch (...) {
      failed_ = true;
    }
  }
  void worker(size_t t) {
    uint64_t seen = 0;
    for (;;) {
      {
        std::unique_lock<std::mutex> lk(mu_);
        wake_.wait(lk, [&] { return stop_ || round_ != seen; });
        if (stop_) return;
        seen = round_;
      }
      claim(t);
      std::lock_guard<std::mutex> lk(mu_);
      if (--busy_ == 0) done_.notify_one();
    }
  }
  std::vector<std::thread> pool_;
  std::mutex mu_;
  std::condition_variable wake_, done_;
  const Fn* fn_ = nullptr;
  size_t n_ = 0, busy_ = 0;
  std::atomic<size_t> next_{0};
  std::atomic<bool> failed_{false};
  uint64_t round_ = 0;
  bool stop_ = false;
};

__global__ void k_base_codes(const uint8_t* __restrict__ chars, uint64_t n, uint8_t* __restrict__ codes) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t c = chars[i];  // A, C, G, T in either case -> 0 .. 3
    codes[i] = (uint8_t)((c >> 1 & 3) ^ (c >> 2 & 1));
  }
}

// One pass over all LCBs: plan, solve, splice.  Rows of LCB k: columns
// [off[k], off[k + 1]) of in[0] and in[1].  `out` gives the buffers for that
// many columns of new rows (or null rows and an error), off becomes the new
// rows' offsets.
int run_pass(Ctx* c, Team& team, std::vector<Scratch>& scratch, bool anchored, double maxw, const uint8_t* const in[2], std::vector<uint64_t>& off,
             const std::function<int(uint64_t, uint8_t* (&)[2])>& out) {
  const size_t nlcb = off.size() - 1;
  std::vector<Plan> plans(nlcb);
  team.run(nlcb, [&](size_t k, size_t t) {
    const Rows r(in[0] + off[k], in[1] + off[k], off[k + 1] - off[k], scratch[t].pre, scratch[t].dots);
    if (anchored)
      plan_anchored(plans[k], r, maxw, scratch[t]);
    else
      plan_refine(plans[k], r, maxw);
  });
  // where each LCB's problems, and their bases, begin
  std::vector<uint64_t> first(nlcb + 1, 0), chars[2];
  for (int q = 0; q < 2; ++q) chars[q].assign(nlcb + 1, 0);
  for (size_t k = 0; k < nlcb; ++k) {
    first[k + 1] = first[k] + plans[k].nprob;
    for (int q = 0; q < 2; ++q) chars[q][k + 1] = chars[q][k] + plans[k].chars[q];
  }
  const uint64_t np = first[nlcb], na = chars[0][nlcb], nb = chars[1][nlcb], nr = na + nb;
  // pinned: the three offset arrays and both genomes' bases; then the path
  // lengths and the problems' rows over the bases
  const uint64_t tab = 3 * (np + 1) * 8, b_at = (na + 255) & ~(uint64_t)255, nc = b_at + nb, down = np * 8 + 2 * nr;
  uint64_t* const h_oa = (uint64_t*)pinned_buf(c, 0, tab + std::max(nc, down) + 16);
  if (!h_oa) return report_error(MVG_ERR_NOMEM, "pinned allocation failed");
  uint64_t *const h_ob = h_oa + (np + 1), *const h_po = h_ob + (np + 1);
  uint8_t *const h_ca = (uint8_t*)h_oa + tab, *const h_cb = h_ca + b_at;
  std::atomic<bool> bad{false};
  team.run(nlcb, [&](size_t k, size_t) {
    uint64_t p = first[k], at[2] = {chars[0][k], chars[1][k]};
    uint8_t seen = 0;
    for (const Piece& x : plans[k].pieces) {
      if (x.kind != kProblem) continue;
      h_oa[p] = at[0];
      h_ob[p] = at[1];
      h_po[p] = at[0] + at[1];
      ++p;
      for (int q = 0; q < 2; ++q) {
        uint8_t* const to = (q ? h_cb : h_ca) + at[q];
        const uint8_t* const r = in[q] + off[k];
        // the range's last base is its last write: nothing past it is touched
        uint64_t hi = x.hi;
        while (hi > x.lo && kClass.of[r[hi - 1]] == 4) --hi;
        seen |= compact(r, x.lo, hi, to);
        at[q] += x.n[q];
      }
    }
    if (seen & 8) bad = true;
  });
  if (bad) return report_error(MVG_ERR_BAD_BASE, "the gap DP takes A, C, G and T only");
  h_oa[np] = na;
  h_ob[np] = nb;
  h_po[np] = nr;
  const int64_t* plen = nullptr;
  const uint8_t* rows[2] = {nullptr, nullptr};
  if (np) {
    Workspace& ws = c->ws;
    uint8_t* d_chars = (uint8_t*)ws.get(c, 86, nc + 16);
    uint8_t* d_codes = (uint8_t*)ws.get(c, 84, nc + 16);
    uint64_t* d_off = (uint64_t*)ws.get(c, 88, tab);
    int32_t* d_scores = (int32_t*)ws.get(c, 89, np * 4 + 16);
    char* d_paths = (char*)ws.get(c, 90, nr + 16);
    uint8_t* d_down = (uint8_t*)ws.get(c, 92, down + 16);  // path lengths, rows of A, rows of B
    if (!d_codes || !d_chars || !d_off || !d_scores || !d_paths || !d_down)
      return report_error(MVG_ERR_NOMEM, "workspace allocation failed");
    uint64_t *const d_oa = d_off, *const d_ob = d_off + (np + 1), *const d_po = d_ob + (np + 1);
    uint8_t *const d_ra = d_down + np * 8, *const d_rb = d_ra + nr;
    cudaStream_t s = c->stream;
    MVG_CUDA_TRY(cudaMemcpyAsync(d_off, h_oa, tab, cudaMemcpyHostToDevice, s));
    MVG_CUDA_TRY(cudaMemcpyAsync(d_chars, h_ca, nc, cudaMemcpyHostToDevice, s));
    k_base_codes<<<grid_for(nc, 256), 256, 0, s>>>(d_chars, nc, d_codes);
    c->launches++;
    MVG_CUDA_TRY(cudaGetLastError());
    if (int rc = gapdp_batch_dev(c, d_codes, d_oa, d_codes + b_at, d_ob, (int64_t)np, d_scores, d_paths, d_po,
                                 (int64_t*)d_down, h_oa, h_ob))
      return rc;
    if (int rc = mvg_path_rows_dev(reinterpret_cast<mvg_handle>(c), d_chars, d_oa, d_chars + b_at, d_ob, (int64_t)np,
                                   d_paths, d_po, (const int64_t*)d_down, d_ra, d_rb))
      return rc;
    uint8_t* const h_down = (uint8_t*)h_oa + tab;
    MVG_CUDA_TRY(cudaMemcpyAsync(h_down, d_down, down, cudaMemcpyDeviceToHost, s));
    MVG_CUDA_TRY(cudaStreamSynchronize(s));
    plen = (const int64_t*)h_down;
    rows[0] = h_down + np * 8;
    rows[1] = rows[0] + nr;
  }
  // each LCB's new length, then the splice into place
  auto length = [&](const Piece& x, uint64_t& p) -> uint64_t {
    switch (x.kind) {
      case kLiteral: return x.hi - x.lo;
      case kProblem: return (uint64_t)plen[p++];  // one column per edge of the path
      default: return x.n[0] + x.n[1];
    }
  };
  std::vector<uint64_t> noff(nlcb + 1, 0);
  for (size_t k = 0; k < nlcb; ++k) {
    uint64_t len = 0, p = first[k];
    for (const Piece& x : plans[k].pieces) len += length(x, p);
    noff[k + 1] = noff[k] + len;
  }
  const std::vector<uint64_t> old(off);
  off = noff;
  uint8_t* to[2];
  if (int rc = out(noff[nlcb], to)) return rc;
  team.run(nlcb, [&](size_t k, size_t) {
    uint64_t at = noff[k], p = first[k];
    for (const Piece& x : plans[k].pieces) {
      const uint64_t g = p, len = length(x, p);
      for (int q = 0; q < 2; ++q) {
        const uint8_t* const r = in[q] + old[k];
        if (x.kind == kLiteral) {
          std::memcpy(to[q] + at, r + x.lo, len);
        } else if (x.kind == kProblem) {
          std::memcpy(to[q] + at, rows[q] + h_po[g], len);
        } else if ((x.kind == kOnlyA) == (q == 0)) {
          uint8_t* t = to[q] + at;
          for (uint64_t c2 = x.lo; c2 < x.hi; ++c2)
            if (kClass.of[r[c2]] != 4) *t++ = r[c2];
        } else {
          std::memset(to[q] + at, '-', len);
        }
      }
      at += len;
    }
  });
  return 0;
}

}  // namespace
}  // namespace mvg

using namespace mvg;

extern "C" int mvg_gapped_alignment(mvg_handle hd, const uint8_t* rows_a, const uint8_t* rows_b,
                                    const uint64_t* col_off, int64_t nlcb, double max_window_size, int passes,
                                    uint8_t* out_a, uint8_t* out_b, uint64_t* out_off, uint64_t cap) {
  Ctx* c = reinterpret_cast<Ctx*>(hd);
  if (!c || nlcb < 0 || !col_off || !out_off || (passes & ~3) || !(max_window_size > 200.0))
    return report_error(MVG_ERR_ARG, "bad argument");
  const uint64_t ncols = col_off[nlcb];
  if ((ncols && (!rows_a || !rows_b)) || (cap && (!out_a || !out_b))) return report_error(MVG_ERR_ARG, "null argument");
  for (int64_t k = 0; k < nlcb; ++k)
    if (col_off[k + 1] < col_off[k]) return report_error(MVG_ERR_ARG, "column offsets must not decrease");
  MVG_CUDA_TRY(cudaSetDevice(c->device));
  try {
    std::vector<uint64_t> off(col_off, col_off + nlcb + 1);
    const uint64_t base = off[0];
    for (uint64_t& o : off) o -= base;
    const uint8_t* rows[2] = {rows_a, rows_b};
    uint64_t total = ncols;
    std::vector<uint8_t> copy[2];  // of the rows, where the output may overwrite them
    for (int q = 0; q < 2; ++q) {
      const uint8_t* const r = rows[q];
      for (const uint8_t* o : {out_a, out_b})
        if (copy[q].empty() && ncols && cap && r < o + cap && o < r + ncols) copy[q].assign(r, r + ncols);
      if (!copy[q].empty()) rows[q] = copy[q].data();
    }
    Team team((size_t)nlcb);
    std::vector<Scratch> scratch(team.threads());
    // new rows: the caller's buffers after the last pass, pinned memory before
    for (int pass = 1; pass <= 2; ++pass) {
      if (!(passes & pass)) continue;
      const bool last = (passes >> pass) == 0;
      uint8_t* made[2] = {nullptr, nullptr};
      const int rc = run_pass(c, team, scratch, pass == 1, max_window_size, rows, off, [&](uint64_t n, uint8_t* (&to)[2]) {
        total = n;
        if (last) {
          for (int64_t k = 0; k <= nlcb; ++k) out_off[k] = off[k];
          if (n > cap) return report_error(MVG_ERR_CAPACITY, "row buffer too small");
          to[0] = out_a;
          to[1] = out_b;
        } else {
          to[0] = pinned_buf(c, 1, 2 * n + 16);
          if (!to[0]) return report_error(MVG_ERR_NOMEM, "pinned allocation failed");
          to[1] = to[0] + n;
        }
        made[0] = to[0];
        made[1] = to[1];
        return 0;
      });
      if (rc) return rc;
      rows[0] = made[0];
      rows[1] = made[1];
    }
    if (!passes) {
      for (int64_t k = 0; k <= nlcb; ++k) out_off[k] = off[k];
      if (total > cap) return report_error(MVG_ERR_CAPACITY, "row buffer too small");
      if (total) {
        std::memcpy(out_a, rows[0], total);
        std::memcpy(out_b, rows[1], total);
      }
    }
  } catch (const std::bad_alloc&) {
    return report_error(MVG_ERR_NOMEM, "host allocation failed");
  }
  return 0;
}
