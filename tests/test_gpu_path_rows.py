"""Rows from paths at the edges of a warp's step and of a CTA's shares, on both
sides of the number of problems from which a problem has one warp, and paths
that do not consume their sequences anywhere along them."""
import numpy as np
import pytest

import mvg
import synth

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 31, 32, 33, 127, 128, 129, 1023, 1024, 1025, 4095, 4097, 9001]


@pytest.fixture(scope="module")
def ctx():
    import build as pkg_build
    pkg_build.build()
    c = mvg.Context(0)
    yield c
    c.close()


def batch(rng, lengths, kinds):
    paths = ["".join(rng.choice(list(kinds), n)) for n in lengths]
    la = [p.count("M") + p.count("D") for p in paths]
    lb = [p.count("M") + p.count("I") for p in paths]
    oa, ob = (np.concatenate([[0], np.cumsum(x)]).astype(np.uint64) for x in (la, lb))
    return paths, synth.random_bases(rng, int(oa[-1])), oa, synth.random_bases(rng, int(ob[-1])), ob


def row(seq, path, skip):
    at = np.frombuffer(path.encode(), np.uint8) != ord(skip)
    out = np.full(len(path), ord("-"), np.uint8)
    out[at] = seq
    return out.tobytes()


@pytest.mark.parametrize("kinds", ["M", "MDI", "MMMMMMMMDI", "DI"])
@pytest.mark.parametrize("nprob", [1, 14, 608, 609])
def test_rows_equal_paths(ctx, nprob, kinds):
    rng = np.random.default_rng(nprob + len(kinds))
    sizes = [9001] if nprob == 1 else [LENGTHS[k % 14] if k % 14 < 8 or k < 42 else k % 90 for k in range(nprob)]
    paths, sa, oa, sb, ob = batch(rng, sizes, kinds)
    for k, (ra, rb) in enumerate(ctx.path_rows(sa, oa, sb, ob, paths)):
        assert ra == row(sa[oa[k]:oa[k + 1]], paths[k], "I"), k
        assert rb == row(sb[ob[k]:ob[k + 1]], paths[k], "D"), k


@pytest.mark.parametrize("nprob", [1, 609])
@pytest.mark.parametrize("at", [0, 40, 2500, 4999])
def test_bad_paths_are_refused(ctx, nprob, at):
    rng = np.random.default_rng(at)
    paths, sa, oa, sb, ob = batch(rng, [5000] + [10] * (nprob - 1), "MMDI")
    ctx.path_rows(sa, oa, sb, ob, paths)
    p = paths[0]
    for bad in (p[:at] + "x" + p[at + 1:], p[:at] + "M" + p[at:], p[:at] + p[at + 1:]):
        with pytest.raises(ValueError):
            ctx.path_rows(sa, oa, sb, ob, [bad] + paths[1:])
