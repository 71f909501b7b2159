"""The seed join's buckets of repeated mers: runs of N and tandem repeats put
thousands of equal keys into one bucket, beside mers that are unique.  Buckets
through the table of their mers, in one piece and in several, and sorted (small
caps, which few mers fill)."""
import numpy as np
import pytest

import mvg
import oracle as O
import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = mvg.Context(0)
    yield c
    c.close()


def _pair(kind, n, run, rng):
    """Two genomes of n bases, 3% apart, with a stretch of `run` bases each."""
    b = synth.random_bases(rng, n)
    a = synth._substitute(rng, b, rng.random(n) < 0.03)
    if kind == "N":
        s = [np.full(run, ord("N"), np.uint8)] * 2
    else:  # a tandem repeat of `kind` bases, exact or 1% substituted
        t = np.resize(synth.random_bases(rng, abs(kind)), run)
        s = [t, t] if kind < 0 else [synth._substitute(rng, t, rng.random(run) < 0.01) for _ in range(2)]
    i, j = n // 3, n // 2
    return np.concatenate([a[:i], s[0], a[i:]]), np.concatenate([b[:j], s[1], b[j:]])


# below and above the 3,072 keys of a bucket's shared memory and the 8,192 of a piece
@pytest.mark.parametrize("cap", [3072, 200, 32])
@pytest.mark.parametrize("weight", [11, 15, 17, 21])
@pytest.mark.parametrize("kind,n,run", [("N", 30000, 700), ("N", 30000, 1600), ("N", 30000, 4000), ("N", 200000, 9000),
                                        ("N", 300000, 60000), (1, 20000, 30000), (-1, 3000, 50000), (3, 50000, 40000),
                                        (-7, 50000, 40000), (61, 20000, 60000)])
def test_pairwise(ctx, kind, n, run, weight, cap):
    a, b = _pair(kind, n, run, np.random.default_rng(run + weight))
    seed = mvg.get_seed(weight, 3 if weight != 21 else 0)
    ctx.set_pair_bucket_cap(cap)
    try:
        got = ctx.pairwise_matches(a, b, seed)
    finally:
        ctx.set_pair_bucket_cap(3072)
    np.testing.assert_array_equal(got, O.pairwise_matches(a, b, seed))


def test_one_genome_repeats(ctx):
    """Mers of every small count in either genome, most of them in one bucket's pieces."""
    rng = np.random.default_rng(11)
    words = [synth.random_bases(rng, 40) for _ in range(60)]
    n_run = np.full(20000, ord("A"), np.uint8)

    def genome(counts):
        parts = [w for w, c in zip(words, counts) for _ in range(c)]
        rng.shuffle(parts)
        return np.concatenate([x for p in parts for x in (p, synth.random_bases(rng, 30))] + [n_run])

    for _ in range(4):
        a, b = genome(rng.integers(0, 4, 60)), genome(rng.integers(0, 4, 60))
        for weight in (9, 15, 19):
            seed = mvg.get_seed(weight, 0)
            np.testing.assert_array_equal(ctx.pairwise_matches(a, b, seed), O.pairwise_matches(a, b, seed))


@pytest.mark.parametrize("kind,run", [("N", 1500), ("N", 5000), ("N", 15000), (1, 15000), (2, 30000), (-3, 12000),
                                      (37, 30000)])
def test_gap_search(ctx, kind, run):
    """Several gaps with a stretch each, one without, one that is nothing else."""
    rng = np.random.default_rng(run)
    pieces = [_pair(kind, n, run, rng) for n in (4000, 20000)]
    plain = synth.random_bases(rng, 6000)
    pieces.append((synth._substitute(rng, plain, rng.random(6000) < 0.05), plain))
    pieces.append(tuple(np.full(run, ord("N"), np.uint8) for _ in range(2)))
    gaps, at = [], [0, 0]
    for p in pieces:
        gaps.append((at[0], len(p[0]), at[1], len(p[1])))
        at = [at[q] + len(p[q]) for q in (0, 1)]
    a, b = (np.concatenate([p[q] for p in pieces]) for q in (0, 1))
    got, off = ctx.gap_anchor_search(a, b, gaps)
    for k, (x, y) in enumerate(pieces):
        _, want = O.gap_anchor_search(x, y)
        want = np.zeros((0, 3), np.int64) if want is None else want
        mine = got[off[k]:off[k + 1]].copy()
        for q, s in ((0, gaps[k][0]), (1, gaps[k][2])):
            mine[:, q] -= np.sign(mine[:, q]) * s
        np.testing.assert_array_equal(mine, want)
