"""Sorted mer lists at the edges of the sort's tiles of 2,048 keys, from one
8-bit pass (seeds of weight 3) to six (64-bit keys), and with only positions
or only mers asked for, against the oracle."""
import ctypes

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


@pytest.mark.parametrize("seed", [0b111, 0b1101, 0b11011, mvg.get_seed(15, 0), mvg.get_seed(16, 0),
                                  mvg.get_seed(21, 0)])
@pytest.mark.parametrize("count", [1, 31, 2047, 2048, 2049, 6145, 140_000])
def test_sml_at_tile_edges(ctx, seed, count):
    import torch
    rng = np.random.default_rng(count + bin(seed).count("1"))
    n = count + mvg.seed_length(seed) - 1
    seq = synth.random_bases(rng, n, 0.4)
    if count > 5000:
        seq = synth.insert_repeats(rng, seq, 300, 8)[:n]
    want_pos, want_mer = O.sml_build(seq, seed)
    pos, mer = ctx.sml_build(seq, seed)
    np.testing.assert_array_equal(pos, want_pos)
    np.testing.assert_array_equal(mer, want_mer)
    d_seq = torch.from_numpy(seq.copy()).cuda()
    d_pos = torch.full((count,), -1, dtype=torch.int32, device="cuda")
    d_mer = torch.full((count,), -1, dtype=torch.int64, device="cuda")
    got = ctypes.c_uint64(0)
    torch.cuda.synchronize()
    build = mvg.load_library().mvg_sml_build_dev
    mvg._check(build(ctx.handle, d_seq.data_ptr(), n, seed, d_pos.data_ptr(), None, count, ctypes.byref(got)))
    mvg._check(build(ctx.handle, d_seq.data_ptr(), n, seed, None, d_mer.data_ptr(), count, ctypes.byref(got)))
    np.testing.assert_array_equal(d_pos.cpu().numpy().view(np.uint32), want_pos)
    np.testing.assert_array_equal(d_mer.cpu().numpy().view(np.uint64), want_mer)
