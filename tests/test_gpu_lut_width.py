"""Gaps of every width around the steps in which the fill looks for a partner
(8 entries per thread, then 32, then 256 at a time), across tile edges, in LUTs
where it is there, one entry out of reach, or missing."""
import numpy as np
import pytest

import indexutils as IU
import mvg
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = mvg.Context(0)
    yield c
    c.close()


WIDTHS = [1, 7, 8, 9, 39, 40, 41, 42, 295, 296, 297, 298, 551, 552, 553, 554, 2000]


@pytest.mark.parametrize("reach", [-1, 0, 1, 5000])
@pytest.mark.parametrize("mode", ["fill", "smooth"])
def test_partner_at(ctx, mode, reach):
    rng = np.random.default_rng(3 + reach)
    for width in WIDTHS:
        n = 6 * width + 30_000
        lut = np.arange(n, dtype=np.int32) + 1000
        holes = np.arange(50, n - width - 10, width + 37)
        for k in holes:
            end = k + width
            lut[k:end] = -1 if mode == "fill" else rng.integers(0, 10**6, width)
            if k % 5 == 0:  # no partner: the rest lies elsewhere
                lut[end:] += 17
        got, want = lut.copy(), lut.copy()
        radius = max(1, width + reach)
        if mode == "fill":
            IU.fillGaps(got, radius, ctx=ctx)
            O.fill_gaps(want, radius)
        else:
            IU.smoothEdges(got, radius, ctx=ctx)
            O.smooth_edges(want, radius)
        np.testing.assert_array_equal(got, want, err_msg="width %d" % width)


def test_no_partner_for_most(ctx):
    rng = np.random.default_rng(8)
    lut = rng.integers(0, 9000, 9000).astype(np.int32)
    lut[rng.random(9000) < 0.5] = -1
    for width in (300, 3000, 2**31 - 1):
        got, want = lut.copy(), lut.copy()
        IU.fillGaps(got, width, ctx=ctx)
        O.fill_gaps(want, width)
        np.testing.assert_array_equal(got, want)
