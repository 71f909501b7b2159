"""Index LUT at the edges of its tiles of 4,096 columns and entries: blocks
that begin, end or are empty at and beside a tile's edge, rows that start off
a 16-byte boundary and at a column above 0, blocks that overwrite each other,
and gaps that run from one tile into the next, against the oracle."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import build as pkg_build
    pkg_build.build()
    import mvg
    c = mvg.Context(0)
    yield c
    c.close()


@pytest.fixture(scope="module")
def iu():
    import indexutils
    return indexutils


def rows(rng, n, gaps):
    g = rng.choice(np.frombuffer(b"ACGT", np.uint8), n)
    r = np.where(rng.random(n) < 0.1, rng.choice(np.frombuffer(b"ACGT", np.uint8), n), g)
    for row in (g, r):
        row[rng.random(n) < gaps] = ord("-")
    both = rng.random(n) < 0.02
    g[both] = r[both] = ord("-")
    return g, r


@pytest.mark.parametrize("widths", [
    [1], [16], [4095], [4096], [4097], [4096, 4096], [4095, 0, 1, 0, 0, 4096, 3], [5, 4091, 1, 4095],
    [1] * 300 + [0] * 40 + [7] * 900, [20_000, 15, 17, 8192, 31], [3, 70_000, 1]])
@pytest.mark.parametrize("skip", [0, 3, 16])
def test_blocks_at_tile_edges(ctx, iu, widths, skip):
    import torch
    rng = np.random.default_rng(len(widths) + sum(widths) + skip)
    off = np.concatenate([[skip], skip + np.cumsum(widths)]).astype(np.uint64)
    g, r = rows(rng, int(off[-1]), 0.05)
    # overlapping genome ranges; a block that starts at 0 wraps to the last entry
    gs = rng.integers(0, max(2, sum(widths) // 2), len(widths)).astype(np.int64)
    gs[0] = 0
    rs = rng.integers(1, 5000, len(widths)).astype(np.int64)
    n = int(sum(widths) * 3 // 4 + 12)
    want = np.empty(n, np.int32)
    assert O.lib().mo_lut_from_blocks(O._p(gs), O._p(rs), O._p(off), O._p(g), O._p(r), len(gs), O._p(want), n) == 0
    np.testing.assert_array_equal(iu.lutFromBlocks(iu.Blocks(gs, rs, off, g, r), n, ctx=ctx), want)
    genome, ref = rng.choice(np.frombuffer(b"ACGT", np.uint8), n), rng.choice(np.frombuffer(b"ACGT", np.uint8), 9000)
    # the rows one byte off a boundary, and each its own way
    pad_g, pad_r = torch.zeros(len(g) + 1, dtype=torch.uint8), torch.zeros(len(r) + 3, dtype=torch.uint8)
    pad_g[1:] = torch.from_numpy(g)
    pad_r[3:] = torch.from_numpy(r)
    t = [x.cuda() for x in (torch.from_numpy(gs), torch.from_numpy(rs), torch.from_numpy(off.view(np.int64)), pad_g,
                            pad_r, torch.from_numpy(genome), torch.from_numpy(ref))]
    lut = torch.empty(n, dtype=torch.int32, device="cuda")
    iu.buildIndexLutDev(t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), t[3].data_ptr() + 1, t[4].data_ptr() + 3,
                        len(gs), t[5].data_ptr(), n, t[6].data_ptr(), len(ref), lut.data_ptr(), n, fill_gaps=False,
                        smooth_edges=True, smoothing_radius=20, ctx=ctx)
    O.smooth_edges(want, 20)
    np.testing.assert_array_equal(lut.cpu().numpy(), want)


@pytest.mark.parametrize("n", [2, 4095, 4096, 4097, 8193, 30_000])
@pytest.mark.parametrize("width", [1, 9, 40, 300, 6000])
def test_fills_across_tiles(ctx, iu, n, width):
    """Runs of gaps of every length up to a tile and more, some closed by a
    partner and some not, with clusters that cross a tile's edge."""
    rng = np.random.default_rng(n + width)
    for trial in range(6):
        lut = np.arange(n, dtype=np.int32) + 50
        at = 1
        while at < n:
            run = int(np.exp(rng.uniform(0, np.log(min(n, 5000 if trial % 2 else 40)))))
            lut[at:at + run] = -1
            if rng.random() < 0.3:
                lut[at + run:] += int(rng.integers(-3, 4))
            at += run + int(rng.integers(1, 60 if trial < 4 else 4000))
        lut[rng.random(n) < 0.02] = 7
        for fn_o, fn_g in ((O.fill_gaps, iu.fillGaps), (O.smooth_edges, iu.smoothEdges)):
            a, b = lut.copy(), lut.copy()
            fn_o(a, width)
            fn_g(b, width, ctx=ctx)
            np.testing.assert_array_equal(a, b, err_msg="trial %d" % trial)
    a, b = lut.copy(), lut.copy()
    np.testing.assert_array_equal(iu.findGaps(b, ctx=ctx), O.find_gaps(a))
    np.testing.assert_array_equal(a, b)
