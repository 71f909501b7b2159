"""Match lists where matches of one hash bucket overlap: two copies of a
stretch of A lie 40,000 bases apart in B (the hash table's size), each with
its own substitutions, so that seeds of two diagonals of one bucket interleave
and the reference's bisection (its comparator is no strict order there) finds
or misses entries by what it happens to probe.  Also segment edges: genome
ends, seeds exactly L and L + 1 apart, and lone seeds."""
import numpy as np
import pytest

import mvg
import oracle as O
import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import build as pkg_build
    pkg_build.build()
    c = mvg.Context(0)
    yield c
    c.close()


def interleaved_pair(seed, rate, flip, n):
    """B holds copies of A's first n bases at 0 and 40,000 (flip bit k: copy k
    reverse-complemented, placed so that its diagonals hash like the other's)."""
    rng = np.random.default_rng(seed)
    x = synth.random_bases(rng, n)
    b = synth.random_bases(rng, 90_000)
    for k in range(2):
        y = synth._substitute(rng, x, rng.random(n) < rate)
        at = 40_000 * k
        if flip == 2 and k == 1:
            # one forward copy at 0, one reverse: offsets y - x = 0 and
            # -(y + x) - 2 - L must agree modulo 40,000 (windows of L = 21 bases)
            at = 80_000 - n - 2
        b[at:at + n] = synth.revcomp(y) if flip == 1 or (flip == 2 and k == 1) else y
    return np.concatenate([x, synth.random_bases(rng, 3000)]), b


@pytest.mark.parametrize("flip", [0, 1, 2])
@pytest.mark.parametrize("rate,n", [(0.02, 2000), (0.08, 6000), (0.2, 3000)])
def test_interleaved_diagonals_of_one_bucket(ctx, rate, n, flip):
    a, b = interleaved_pair(int(1000 * rate) + 7 * flip + n, rate, flip, n)
    seed = mvg.get_seed(15, 3)
    want = O.pairwise_matches(a, b, seed)
    if rate < 0.2:  # the case is what it is meant to be: the reference inserts some entries twice
        assert len(want) > len(np.unique(want, axis=0))
    np.testing.assert_array_equal(ctx.pairwise_matches(a, b, seed), want)
    st = ctx.pairwise_stats()
    assert st["matches"] == len(want) and st["pairs"] == st["matches"] + st["collisions"]


@pytest.mark.parametrize("weight", [5, 11, 15, 17])
def test_segment_edges(ctx, weight):
    """Matches that reach both genomes' ends, and pairs of substitutions that
    leave seeds 1 to 2 L apart."""
    rng = np.random.default_rng(weight)
    a = synth.random_bases(rng, 5000 if weight > 5 else 300)
    b = a.copy()
    seed = mvg.get_seed(weight, 0)
    L = mvg.seed_length(seed)
    for k, p in enumerate(range(4 * L, len(a) - 8 * L, 6 * L)):
        for q in (p, p + 1 + k % (2 * L)):
            b[q] = ord("ACGT"["ACGT".index(chr(b[q])) - 1])
    for x, y in ((a, b), (a, synth.revcomp(b)), (b[L // 2:], a[:-3]), (a[:2048], b), (a[:2049], synth.revcomp(b))):
        np.testing.assert_array_equal(ctx.pairwise_matches(x, y, seed), O.pairwise_matches(x, y, seed))


@pytest.mark.parametrize("gap", [20, 40, 63, 64, 65, 96, 200, 255, 256, 288, 289, 320, 1000, 1290, 1330, 4000])
@pytest.mark.parametrize("flip", [False, True])
def test_walks_across_repeats(ctx, gap, flip):
    """Segments of one diagonal with a repeat of `gap` bases between them,
    whose seeds match but are not unique: walks of every length, some of which
    end on a substitution in the repeat."""
    rng = np.random.default_rng(gap)
    a, b = [], []
    for k in range(12):
        u, v, r = (synth.random_bases(rng, n) for n in (150, 170, gap))
        rb = r.copy()
        if k % 3:
            rb[int(rng.integers(0, gap))::max(1, gap // (k % 3))] = ord("A")
        a += [u, r, v, r, synth.random_bases(rng, 60)]
        b += [u, rb, v, synth.random_bases(rng, 80), rb]
    a, b = np.concatenate(a), np.concatenate(b)
    if flip:
        b = synth.revcomp(b)
    seed = mvg.get_seed(15, 0)
    np.testing.assert_array_equal(ctx.pairwise_matches(a, b, seed), O.pairwise_matches(a, b, seed))


@pytest.mark.parametrize("n", [2_000, 60_000, 230_000, 262_000, 300_000])
@pytest.mark.parametrize("weight", [15, 17])
def test_segment_order_around_one_cta_s_sort(ctx, n, weight):
    """From a few segment ends to twice as many as one CTA sorts."""
    rng = np.random.default_rng(n + weight)
    a = synth.random_bases(rng, n)
    b = synth._substitute(rng, a, rng.random(n) < 0.06)
    b[n // 3:n // 2] = synth.revcomp(b[n // 3:n // 2])
    seed = mvg.get_seed(weight, 0)
    got = ctx.pairwise_matches(a, b, seed)
    np.testing.assert_array_equal(got, O.pairwise_matches(a, b, seed))


@pytest.mark.parametrize("seed", [0b1, 0b11, 0b101, 0b1101, 0b10111])
def test_fewest_buckets(ctx, seed):
    """Seeds of so few bases that the join has four to sixteen buckets."""
    rng = np.random.default_rng(seed)
    for n in (3, 9, 40, 200):
        a, b = synth.random_bases(rng, n), synth.random_bases(rng, n + 2)
        np.testing.assert_array_equal(ctx.pairwise_matches(a, b, seed), O.pairwise_matches(a, b, seed))
    same = np.frombuffer(b"ACGTTGCAAC", np.uint8)
    np.testing.assert_array_equal(ctx.pairwise_matches(same, same, seed), O.pairwise_matches(same, same, seed))


@pytest.mark.parametrize("weight", [16, 21, 22, 23, 25, 31])
def test_join_and_sort_on_both_sides_of_their_line(ctx, weight):
    """Seeds of up to 22 bases go through the bucketed join, longer ones through
    the sort of both genomes' keys."""
    rng = np.random.default_rng(weight)
    a = synth.random_bases(rng, 30_000)
    b = synth._substitute(rng, a, rng.random(len(a)) < 0.01)
    b = np.concatenate([b[:12_000], synth.revcomp(b[12_000:20_000]), b[500:1500], b[20_000:]])
    seed = (1 << weight) - 1  # solid: any weight up to 31
    np.testing.assert_array_equal(ctx.pairwise_matches(a, b, seed), O.pairwise_matches(a, b, seed))
