"""Gap search where its filter changes hands: gaps whose matches have equal
left ends in A or in B (repeats with substitutions on either side), gaps of
more matches than one CTA sorts, gaps of a handful, and more gaps than one
chunk takes; every gap against the oracle's pairwiseAnchorSearch."""
import numpy as np
import pytest

import mvg
import oracle as O
import synth
from test_gpu_gapsearch import embed, shift

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import build as pkg_build
    pkg_build.build()
    c = mvg.Context(0)
    yield c
    c.close()


def check(ctx, rng, pairs, every=1):
    ga, gb, rows = embed(rng, pairs)
    anchors, off = ctx.gap_anchor_search(ga, gb, rows)
    wants = []
    for k in range(0, len(pairs), every):
        anc = O.gap_anchor_search(*pairs[k])[1]
        want = np.zeros((0, 3), np.int64) if anc is None else shift(anc, rows[k, 0], rows[k, 2])
        np.testing.assert_array_equal(anchors[off[k]:off[k + 1]], want, err_msg="gap %d" % k)
        wants.append(len(want))
    return wants


@pytest.mark.parametrize("copies", [2, 5])
@pytest.mark.parametrize("side", [0, 1])
def test_equal_left_ends(ctx, side, copies):
    """Each copy of a repeat starts a match at the same place of the other
    genome; one gap, and forty (above and below one copy per gap)."""
    rng = np.random.default_rng(10 * copies + side)
    pairs = []
    for k in range(40):
        x = synth.random_bases(rng, int(rng.integers(60, 4000)))
        y = np.concatenate([np.concatenate([x, synth.random_bases(rng, 50)]) for _ in range(copies)])
        y = synth._substitute(rng, y, rng.random(len(y)) < 0.04)
        pairs.append((y, x) if side else (x, y))
    check(ctx, rng, pairs)
    check(ctx, rng, pairs[:1])


@pytest.mark.parametrize("rate", [0.06, 0.15])
def test_gaps_around_one_cta_s_sort(ctx, rate):
    """From a few matches to more per gap than one CTA sorts."""
    rng = np.random.default_rng(5)
    pairs = []
    for n in (30, 100, 400, 8_000, 20_000, 40_000, 160_000):
        b = synth.random_bases(rng, n)
        pairs.append((synth._substitute(rng, b, rng.random(n) < rate), b))
    wants = check(ctx, rng, pairs)
    assert rate < 0.15 or wants[-1] > 1536


def test_more_gaps_than_a_chunk(ctx):
    rng = np.random.default_rng(6)
    pairs = []
    for k in range(16_500):
        b = synth.random_bases(rng, 40 + k % 90)
        pairs.append((synth._substitute(rng, b, rng.random(len(b)) < 0.05), b))
    check(ctx, rng, pairs, every=23)
