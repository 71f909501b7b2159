"""Full gap DP under a tight arena bound: slots that do not fit in the shape
chosen for speed are checkpointed in taller strips, with states some blocks
apart, and give the same scores and paths."""
import numpy as np
import pytest

import mvg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = mvg.Context(0)
    yield c
    c.close()


def _pair(rng, la, lb):
    a = rng.integers(0, 4, la, dtype=np.uint8)
    b = np.resize(a, lb)
    hit = rng.random(lb) < 0.15
    b[hit] = rng.integers(0, 4, int(hit.sum()), dtype=np.uint8)
    cut = lb // 3
    return a, np.concatenate([b[cut // 2:cut], b[:cut // 2], b[cut:]])  # a move: gaps on both sides


def _batch(rng, shapes):
    pairs = [_pair(rng, la, lb) for la, lb in shapes]
    off = [np.concatenate([[0], np.cumsum([len(p[q]) for p in pairs])]) for q in (0, 1)]
    return np.concatenate([p[0] for p in pairs]), off[0], np.concatenate([p[1] for p in pairs]), off[1]


# stored bits; half-height strips; one strip, states two blocks apart; one that
# fits; a mix; many strips with one state each, with none (twice); bits by
# request; a batch that fits in waves
@pytest.mark.parametrize("shapes,bound,checkpoints", [
    ([(5900, 700)], 1 << 20, True),
    ([(5000, 1500)], 1357 << 10, True),
    ([(200, 40000)], 1278 << 10, True),
    ([(100, 32767)], 1 << 20, True),
    ([(257, 10000), (255, 29999), (129, 700)], 1 << 20, True),
    ([(100000, 180)], 2726 << 10, True),
    ([(200000, 120)], 1500032, True),
    ([(139000, 120)], 1048576, True),
    ([(5900, 690)], 2215424, False),
    ([(3000, 1000), (31, 33), (1, 5000), (5000, 1), (700, 700)], 1 << 20, True)])
def test_tight_bound(ctx, shapes, bound, checkpoints):
    rng = np.random.default_rng(len(shapes) + bound)
    batch = _batch(rng, shapes)
    ctx.set_dp_checkpoint(checkpoints)
    try:
        want = ctx.gap_align_batch(*batch)
        ctx.set_tb_arena(bound)
        got = ctx.gap_align_batch(*batch)
    finally:
        ctx.set_tb_arena(2**64 - 1)
        ctx.set_dp_checkpoint(True)
    np.testing.assert_array_equal(got[0], want[0])
    assert got[1] == want[1]


def test_tight_bound_many(ctx):
    """A mixed batch in many waves, and the banded entry point's fallback."""
    rng = np.random.default_rng(5)
    shapes = [(int(rng.integers(1, 2500)), int(rng.integers(1, 2500))) for _ in range(60)]
    batch = _batch(rng, shapes)
    want = ctx.gap_align_batch(*batch)
    half = np.full(len(shapes), 12, np.int32)
    delta = np.zeros(len(shapes), np.int32)
    ctx.set_tb_arena(2 << 20)
    try:
        got = ctx.gap_align_batch(*batch)
        banded = ctx.gap_align_banded(*batch, delta, half)
    finally:
        ctx.set_tb_arena(2**64 - 1)
    for r in (got, banded):
        np.testing.assert_array_equal(r[0], want[0])
        assert r[1] == want[1]
