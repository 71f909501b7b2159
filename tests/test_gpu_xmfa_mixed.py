"""XMFA text of short alignments whose blocks differ much in width: one wide
block among many small ones, on both sides of the number of CTAs above which
the text is spread by its bytes."""
import numpy as np
import pytest

import mvg
import synth
from test_gpu_xmfa_lines import text_of

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = mvg.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("wide,small,count", [(100_000, 1, 40), (100_000, 1, 700), (60_000, 2, 1500), (900, 1, 3300),
                                              (1100, 1, 1700), (30, 30, 3000)])
def test_text_of_mixed_blocks(ctx, wide, small, count):
    rng = np.random.default_rng(wide + count)
    widths = np.full(count + 1, small)
    widths[count // 2] = wide
    off = np.concatenate([[0], np.cumsum(widths)]).astype(np.uint64)
    rows = [synth.random_bases(rng, int(off[-1])) for _ in range(2)]
    starts = rng.integers(1, 10**6, 2 * len(widths)).astype(np.int64)
    lengths = rng.integers(1, 10**6, 2 * len(widths)).astype(np.int64)
    names = ("a.fasta", "dir/b")
    assert ctx.xmfa_write(*names, starts, lengths, rows[0], rows[1], off) == text_of(names, starts, lengths, rows, off)
