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
#include "match_components.cuh"

namespace mvg {

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
  const bool bucketed = 2 * s.w <= kPairMaxBits && ca + cb <= kPairBucketMaxKeys;
  uint32_t* tab = (uint32_t*)ws.get(c, 38, na * 4);
  if (!tab) return report_error(MVG_ERR_NOMEM, "workspace allocation failed");
  MVG_CUDA_TRY(cudaMemsetAsync(tab, 0xff, na * 4, c->stream));
  stage_mark(c, "sml_sort");
  PairBucketBufs join;
  if (bucketed) {
    if ((rc = pair_buckets(c, ga, ca, gb, cb, s, tab, &join))) return rc;
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
  OnePair prob;
  prob.c.g[0] = ga;
  prob.c.g[1] = gb;
  prob.c.n[0] = (int64_t)na;
  prob.c.n[1] = (int64_t)nb;
  prob.c.s = s;
  prob.out = d_out;
  prob.cap = cap;
  ComponentResult r;
  if ((rc = match_components(c, prob, tab, bucketed ? &join : nullptr, (int64_t)na, 16, [](uint64_t) { return 0; }, &r))) return rc;
  stage_end(c);
  MVG_CUDA_TRY(cudaStreamSynchronize(c->stream));
  c->stats.pairs = r.pairs;
  c->stats.matches = r.rows;
  c->stats.collisions = r.pairs - r.rows;
  *count = r.rows;
  if (r.rows > cap) return report_error(MVG_ERR_CAPACITY, "match output buffer too small");
  return 0;
}

}  // namespace mvg
