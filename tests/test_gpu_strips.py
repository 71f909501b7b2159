"""The full gap DP's strips and block-wise traceback at the sizes where they
change: strip and lane edges in rows, the staging chunks, the state interval
and the direct-bits limit in columns; checkpointed and stored-bits passes,
strips on one warp or pipelined.  Scores and paths equal the oracle's."""
import numpy as np
import pytest

import mvg
import oracle as O
import synth

pytestmark = pytest.mark.gpu

ROWS = [1, 7, 8, 9, 127, 128, 129, 255, 256, 257, 513, 769]
COLS = [1, 31, 32, 33, 63, 64, 65, 96, 97, 98, 127, 225, 226, 699, 700, 701, 1033]


@pytest.fixture(scope="module")
def ctx():
    import build as pkg_build
    pkg_build.build()
    c = mvg.Context(0)
    yield c
    c.close()


@pytest.fixture(scope="module")
def batch():
    rng = np.random.default_rng(412)
    a, b = [], []
    for la in ROWS:
        for lb in COLS:
            x = rng.integers(0, 4, la).astype(np.uint8)
            y = synth.mutate_codes(rng, x, 0.1, la // 60, 3.0)  # homologous where the lengths allow it
            y = np.concatenate([y, rng.integers(0, 4, lb).astype(np.uint8)])[:lb]
            a.append(x)
            b.append(y)
    for la, lb in ((1500, 1400), (3000, 900), (600, 2600)):  # unrelated: long runs of gaps
        a.append(rng.integers(0, 4, la).astype(np.uint8))
        b.append(rng.integers(0, 4, lb).astype(np.uint8))
    oa = np.concatenate([[0], np.cumsum([len(x) for x in a])]).astype(np.uint64)
    ob = np.concatenate([[0], np.cumsum([len(x) for x in b])]).astype(np.uint64)
    sa, sb = np.concatenate(a), np.concatenate(b)
    scores, plen, paths, poff = O.nw_batch(sa, oa, sb, ob)
    raw = paths.tobytes()
    return sa, oa, sb, ob, scores, [raw[int(poff[k]):int(poff[k]) + int(plen[k])].decode() for k in range(len(a))]


@pytest.mark.parametrize("rows,ckpt,piped", [(8, True, 2), (8, True, 1000), (8, False, 2), (4, True, 3)])
def test_strip_edges_vs_oracle(ctx, batch, rows, ckpt, piped):
    sa, oa, sb, ob, want, want_paths = batch
    full, band = ctx.full_rows, ctx.band_rows
    try:
        ctx.set_dp_rows(rows, band)
        ctx.set_dp_checkpoint(ckpt)
        ctx.set_dp_coop_strips(piped)
        scores, paths = ctx.gap_align_batch(sa, oa, sb, ob)
        ctx.set_tb_arena(4 << 20)  # many waves
        again, paths_again = ctx.gap_align_batch(sa, oa, sb, ob)
    finally:
        ctx.set_tb_arena(1 << 62)
        ctx.set_dp_rows(full, band)
        ctx.set_dp_checkpoint(True)
        ctx.set_dp_coop_strips(8)
    np.testing.assert_array_equal(scores, want)
    assert paths == want_paths
    np.testing.assert_array_equal(again, want)
    assert paths_again == want_paths
