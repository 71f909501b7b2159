"""Bands that no ring height takes, few and many (more than two thirds of the
device's warps): each on a CTA, or on a warp up to 2,048 columns, with the full
DP's scores and paths."""
import numpy as np
import pytest

import mvg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = mvg.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("count", [30, 1800])
def test_equal_to_full(ctx, count):
    rng = np.random.default_rng(count)
    la = rng.integers(4000, 4400, count)
    lb = la + rng.integers(-60, 60, count)
    oa, ob = (np.concatenate([[0], np.cumsum(x)]) for x in (la, lb))
    a = rng.integers(0, 4, int(oa[-1]), dtype=np.uint8)
    b = np.concatenate([np.resize(a[oa[k]:oa[k + 1]], lb[k]) for k in range(count)])
    hit = rng.random(len(b)) < 0.04
    b[hit] = rng.integers(0, 4, int(hit.sum()), dtype=np.uint8)
    half = np.full(count, 560, np.int32)
    half[::7] = 1030  # wide enough for a CTA in either case
    half[5::50] = 3  # a narrow one, some rejected
    delta = np.where(np.arange(count) % 11 == 3, 700, 0).astype(np.int32)
    want = ctx.gap_align_batch(a, oa, b, ob)
    ctx.set_band_whole_fraction(0.9)
    try:
        scores, paths, status, _ = ctx.gap_align_banded(a, oa, b, ob, delta, half)
    finally:
        ctx.set_band_whole_fraction(0.5)
    np.testing.assert_array_equal(scores, want[0])
    assert paths == want[1]
    assert set(status) == {0, 1}
