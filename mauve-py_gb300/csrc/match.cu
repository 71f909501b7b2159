// Pairwise seed matching and maximal-match extension (two genomes).
//
// The reference (PairwiseMatchFinder over MemHash) walks the two sorted mer
// lists in key order, hashes every seed that is unique in both genomes into
// one of 40,000 buckets by its generalised offset, skips a seed whose bucket
// already holds a match containing it, and otherwise extends the seed to a
// maximal spaced-seed match and inserts it in sorted position.  Here:
//
//   pair_buckets (or pair_sort)          the seeds unique in each genome
//                                       (strand ignored): B's position and
//                                       the strand relation by A's position
//   k_seg_*                              chains of seeds of one diagonal, by
//                                       bucket
//   k_seg_walk                           ExtendMatch from the chains' ends
//   k_comp_*                             matches: buckets in order, each
//                                       bucket's matches in order (GetMatchList)
//   k_flag_*                             buckets where matches overlap: the
//                                       seeds whose test depends on what the
//                                       bisection happens to probe
//
// match_components.cuh says why this is the reference's match list.
#include <algorithm>

#include "match_components.cuh"

namespace mvg {

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

// The buckets k_comp_out flagged, exactly, and the match list again.
static int flagged_matches(Ctx* c, const MatchCtx& mc, const uint32_t* tab, const Components& C, uint32_t ncomp,
                           const uint32_t* bflag, const uint32_t* flagged, uint32_t nflagged, int64_t* d_out, uint64_t cap,
                           uint64_t* matches) {
  const int L = mc.s.L;
  Workspace& ws = c->ws;
  // work and seed counts, sums, the flagged buckets' numbers, all components' output slots, scan scratch
  uint32_t* w = (uint32_t*)ws.get(c, 37, ((size_t)kTableSize + ncomp + scan_scratch_words(ncomp) + 16) * 4);
  if (!w) return report_error(MVG_ERR_NOMEM, "workspace allocation failed");
  uint32_t *count = w, *bnumber = w + 16, *cat = bnumber + kTableSize, *scratch = cat + ncomp;
  MVG_CUDA_TRY(cudaMemsetAsync(count, 0, 64, c->stream));
  k_flag_sort<<<nflagged, 256, 0, c->stream>>>(C, ncomp, L, flagged);
  k_flag_numbers<<<div_up(nflagged, 256), 256, 0, c->stream>>>(flagged, nflagged, bnumber);
  FlagWork W{count, nullptr, nullptr};
  k_flag_plan<<<grid_for(ncomp, 256), 256, 0, c->stream>>>(C, ncomp, bflag, W);
  c->launches += 3;
  MVG_CUDA_TRY(cudaMemcpyAsync(c->h_scalars, count, 8, cudaMemcpyDeviceToHost, c->stream));
  MVG_CUDA_TRY(cudaStreamSynchronize(c->stream));
  const uint32_t whole = ((const uint32_t*)c->h_scalars)[0], behind = ((const uint32_t*)c->h_scalars)[1];
  // the pieces, and room for every position of the seeds' pieces
  const size_t room = (size_t)behind * kFlagPiece;
  W.whole = (uint2*)ws.get(c, 39, ((size_t)whole + behind) * 8 + 16);
  uint64_t* t0 = (uint64_t*)ws.get(c, 40, room * 8 + 16);
  uint64_t* t1 = (uint64_t*)ws.get(c, 41, room * 8 + 16);
  uint32_t* u = (uint32_t*)ws.get(c, 42, room * 4 * 4 + 16);
  uint32_t* sscr = (uint32_t*)ws.get(c, 43, sort_scratch_words((int64_t)room, 64) * 4);
  if (!W.whole || !t0 || !t1 || !u || !sscr) return report_error(MVG_ERR_NOMEM, "workspace allocation failed");
  W.behind = W.whole + whole;
  W.count = count + 2;
  FlagSeeds S{t0, u, u + room, u + 2 * room, count + 4};
  k_flag_plan<<<grid_for(ncomp, 256), 256, 0, c->stream>>>(C, ncomp, bflag, W);
  k_flag_time<<<div_up((int64_t)whole * 32, 256), 256, 0, c->stream>>>(mc, tab, C, W.whole, whole);
  k_flag_collect<<<div_up((int64_t)behind * 32, 256), 256, 0, c->stream>>>(mc, tab, C, W.behind, behind, S);
  c->launches += 3;
  MVG_CUDA_TRY(cudaMemcpyAsync(c->h_scalars, count + 4, 4, cudaMemcpyDeviceToHost, c->stream));
  MVG_CUDA_TRY(cudaStreamSynchronize(c->stream));
  const uint32_t nseeds = ((const uint32_t*)c->h_scalars)[0];
  if (nseeds) {
    // by mer, then stably by bucket; the mers stay where they are for the tests
    uint64_t* keys = (uint64_t*)ws.get(c, 48, (size_t)nseeds * 8);
    if (!keys) return report_error(MVG_ERR_NOMEM, "workspace allocation failed");
    MVG_CUDA_TRY(cudaMemcpyAsync(keys, t0, (size_t)nseeds * 8, cudaMemcpyDeviceToDevice, c->stream));
    uint32_t *id = S.id, *id_alt = u + 3 * room;
    if (sort_pairs<uint64_t>(keys, id, t1, id_alt, nseeds, 2 * mc.s.w, sscr, c->stream, &c->launches, c->d_err))
      std::swap(id, id_alt);
    uint32_t *number = (uint32_t*)keys, *number_alt = (uint32_t*)t1;
    k_flag_bucket<<<div_up(nseeds, 256), 256, 0, c->stream>>>(C, S.e, id, nseeds, bnumber, number);
    int bits = 1;
    while ((1u << bits) < nflagged) ++bits;
    if (sort_pairs<uint32_t>(number, id, number_alt, id_alt, nseeds, bits, sscr, c->stream, &c->launches, c->d_err)) {
      std::swap(number, number_alt);
      std::swap(id, id_alt);
    }
    k_flag_test<<<nflagged, 1024, 0, c->stream>>>(C, ncomp, L, flagged, number, id, nseeds, S);
    c->launches += 2;
  }
  exclusive_scan(C.copies, cat, ncomp, scratch, count + 5, c->stream, &c->launches);
  k_comp_out_copies<<<grid_for(ncomp, 256), 256, 0, c->stream>>>(C, ncomp, cat, L, d_out, cap);
  c->launches++;
  MVG_CUDA_TRY(cudaMemcpyAsync(c->h_scalars, count + 5, 4, cudaMemcpyDeviceToHost, c->stream));
  MVG_CUDA_TRY(cudaStreamSynchronize(c->stream));
  MVG_CUDA_TRY(cudaGetLastError());
  *matches = (uint32_t)c->h_scalars[0];
  return 0;
}

int pairwise_matches_dev(Ctx* c, const uint8_t* d_a, uint64_t na, const uint8_t* d_b, uint64_t nb, uint64_t seed,
                         int64_t* d_out, uint64_t cap, uint64_t* count) {
  const SeedDesc s = make_seed_desc(seed);
  if (s.L == 0 || s.L > 31) return report_error(MVG_ERR_ARG, "invalid seed pattern");
  if (na >= 0x7fffffffull || nb >= 0x7fffffffull) return report_error(MVG_ERR_ARG, "genome longer than 2^31-1");
  c->stats = MatchStats();
  *count = 0;
  stage_begin_call(c);
  stage_mark(c, "pack");
  Workspace& ws = c->ws;
  uint32_t* ga = (uint32_t*)ws.get(c, 20, packed_words(na) * 4);
  uint32_t* gb = (uint32_t*)ws.get(c, 21, packed_words(nb) * 4);
  if (!ga || !gb) return report_error(MVG_ERR_NOMEM, "workspace allocation failed");
  MVG_CUDA_TRY(cudaMemsetAsync(c->d_err, 0, sizeof(uint32_t), c->stream));
  int rc;
  if ((rc = pack_sequence(c, d_a, na, ga))) return rc;
  if ((rc = pack_sequence(c, d_b, nb, gb))) return rc;
  const uint64_t ca = na >= (uint64_t)s.L ? na - s.L + 1 : 0;
  const uint64_t cb = nb >= (uint64_t)s.L ? nb - s.L + 1 : 0;
  if (ca == 0 || cb == 0) return check_device_error(c);
  // weights up to 22 and up to 2^25 seeds: the bucketed join; otherwise one
  // sort of both genomes' keys and a join over its runs
  const bool bucketed = s.w <= kPairBucketMaxWeight && ca + cb <= kPairBucketMaxKeys;
  const int64_t ntiles = div_up((int64_t)na, kSegTile);
  uint32_t* tab = (uint32_t*)ws.get(c, 38, na * 4);
  uint32_t* masks = (uint32_t*)ws.get(c, 39, (size_t)ntiles * (kSegTile / 32) * 2 * 4);
  // head and tail counts per tile, their offsets, scan scratch, sums
  uint32_t* tcount = (uint32_t*)ws.get(c, 44, ((size_t)ntiles * 4 + scan_scratch_words(2 * ntiles) + 16) * 4);
  uint32_t* scal = (uint32_t*)ws.get(c, 34, 64);  // segment ends, pairs, components, flagged buckets
  if (!tab || !masks || !tcount || !scal) return report_error(MVG_ERR_NOMEM, "workspace allocation failed");
  uint32_t *headw = masks, *tailw = masks + ntiles * (kSegTile / 32);
  uint32_t *toff = tcount + 2 * ntiles, *tscr = toff + 2 * ntiles;
  MVG_CUDA_TRY(cudaMemsetAsync(tab, 0xff, na * 4, c->stream));
  MVG_CUDA_TRY(cudaMemsetAsync(scal, 0, 64, c->stream));
  stage_mark(c, "sml_sort");
  if (bucketed) {
    if ((rc = pair_buckets(c, ga, ca, gb, cb, s, tab))) return rc;
  } else {
    SmlKeys sk;
    if ((rc = pair_sort(c, ga, ca, gb, cb, s, &sk))) return rc;
    stage_mark(c, "unique_join");
    const int64_t nk = (int64_t)sk.count;
    if (sk.wide)
      k_tab_runs<uint64_t><<<div_up(nk, 256), 256, 0, c->stream>>>((const uint64_t*)sk.keys, sk.pos, nk, tab);
    else
      k_tab_runs<uint32_t><<<div_up(nk, 256), 256, 0, c->stream>>>((const uint32_t*)sk.keys, sk.pos, nk, tab);
    c->launches++;
  }
  stage_mark(c, "segments");
  k_seg_bits<<<(unsigned)ntiles, 256, 0, c->stream>>>(tab, (int64_t)na, s.L, headw, tailw, tcount, ntiles, scal + 1);
  c->launches++;
  scan_counts(tcount, 2 * ntiles, toff, tscr, scal, c->stream, &c->launches);
  MVG_CUDA_TRY(cudaMemcpyAsync(c->h_scalars, scal, 8, cudaMemcpyDeviceToHost, c->stream));
  if ((rc = check_device_error(c))) return rc;
  const int64_t ends = ((const uint32_t*)c->h_scalars)[0], nseg = ends / 2;
  const uint64_t npairs = ((const uint32_t*)c->h_scalars)[1];
  c->stats.pairs = npairs;
  if (npairs == 0) return 0;

  uint32_t* k0 = (uint32_t*)ws.get(c, 40, ends * 4);
  uint32_t* v0 = (uint32_t*)ws.get(c, 41, ends * 4);
  uint32_t* k1 = (uint32_t*)ws.get(c, 42, ends * 4);
  uint32_t* v1 = (uint32_t*)ws.get(c, 48, ends * 4);
  uint32_t* sscr = (uint32_t*)ws.get(c, 43, sort_scratch_words(ends, 17) * 4);
  // per segment: last position, two walks, the join with the next one; its
  // tiles' component counts and offsets; per component (at most one per
  // segment) its fields; the buckets' flags and the list of flagged ones
  const int64_t ctiles = div_up(nseg, kSegTile);
  uint64_t* blk = (uint64_t*)ws.get(c, 45, (size_t)nseg * (8 * 2 + 4 * 5 + 4 * 3 + 1) + (2 * ctiles + 2 * kTableSize + scan_scratch_words(ctiles)) * 4 + 256);
  if (!k0 || !v0 || !k1 || !v1 || !sscr || !blk) return report_error(MVG_ERR_NOMEM, "workspace allocation failed");
  Components C;
  C.diag = blk;
  C.time = blk + nseg;
  uint32_t* w = (uint32_t*)(blk + 2 * nseg);
  auto take = [&](int64_t n) {
    uint32_t* p = w;
    w += n;
    return p;
  };
  C.lo = take(nseg);
  C.hi = take(nseg);
  C.seed = take(nseg);
  C.bucket = take(nseg);
  C.copies = take(nseg);
  uint32_t *last = take(nseg), *moved = take(2 * nseg);
  uint32_t *ccount = take(ctiles), *coff = take(ctiles), *cscr = take(scan_scratch_words(ctiles));
  uint32_t *bflag = take(kTableSize), *flagged = take(kTableSize);
  uint8_t* joined = (uint8_t*)w;
  MatchCtx mc;
  mc.g[0] = ga;
  mc.g[1] = gb;
  mc.n[0] = (int64_t)na;
  mc.n[1] = (int64_t)nb;
  mc.s = s;
  k_seg_emit<<<(unsigned)ntiles, 128, 0, c->stream>>>(tab, s.L, headw, tailw, toff, ntiles, k0, v0);
  stage_mark(c, "segment_sort");
  const bool alt = sort_pairs<uint32_t>(k0, v0, k1, v1, ends, 17, sscr, c->stream, &c->launches, c->d_err) != 0;
  const uint32_t *key = alt ? k1 : k0, *head = alt ? v1 : v0, *tail = head + nseg;
  stage_mark(c, "walks");
  k_seg_pair<<<div_up(nseg, 256), 256, 0, c->stream>>>(tab, head, key, tail, nseg, last);
  k_seg_walk<<<div_up(2 * nseg * 8, 256), 256, 0, c->stream>>>(mc, tab, key, head, last, nseg, moved, joined);
  stage_mark(c, "components");
  MVG_CUDA_TRY(cudaMemsetAsync(bflag, 0, kTableSize * 4, c->stream));
  k_comp_count<<<(unsigned)ctiles, 256, 0, c->stream>>>(joined, nseg, ccount);
  scan_counts(ccount, ctiles, coff, cscr, scal + 2, c->stream, &c->launches);
  k_comp_emit<<<(unsigned)ctiles, 256, 0, c->stream>>>(tab, key, head, last, moved, joined, nseg, coff, C);
  k_comp_out<<<grid_for(nseg, 256), 256, 0, c->stream>>>(C, scal + 2, s.L, d_out, cap, bflag, flagged, scal + 3);
  c->launches += 6;
  stage_end(c);
  MVG_CUDA_TRY(cudaMemcpyAsync(c->h_scalars, scal + 2, 8, cudaMemcpyDeviceToHost, c->stream));
  if ((rc = check_device_error(c))) return rc;
  uint64_t nm = ((const uint32_t*)c->h_scalars)[0];
  const uint32_t nflagged = ((const uint32_t*)c->h_scalars)[1];
  if (nflagged && (rc = flagged_matches(c, mc, tab, C, (uint32_t)nm, bflag, flagged, nflagged, d_out, cap, &nm))) return rc;
  c->stats.matches = nm;
  c->stats.collisions = npairs - nm;
  *count = nm;
  if (nm > cap) return report_error(MVG_ERR_CAPACITY, "match output buffer too small");
  return 0;
}

}  // namespace mvg
