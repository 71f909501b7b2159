"""Pairs of which both sequences are longer than the scaled scores allow
(200,000 for the ring schedule, 400,000 for stored bits): the full DP and the
banded strip kernel, two recurrences of their own, agree in score and path, and
the score is the path's."""
import numpy as np
import pytest

import mvg

pytestmark = pytest.mark.gpu

SP = np.array([[91, -114, -31, -123], [-114, 100, -125, -31], [-31, -125, 100, -114], [-123, -31, -114, 91]]) + 60


@pytest.fixture(scope="module")
def ctx():
    c = mvg.Context(0)
    yield c
    c.close()


def _path_score(a, b, path):
    """Substitution scores, and -400 per run of gaps, -200 where it touches an end."""
    p = np.frombuffer(path.encode(), np.uint8)
    m, d, i = (p == ord(x) for x in "MDI")
    ia, ib = np.cumsum(m | d) - 1, np.cumsum(m | i) - 1
    assert ia[-1] == len(a) - 1 and ib[-1] == len(b) - 1
    score = int(SP[a[ia[m]], b[ib[m]]].sum())
    for g in (d, i):
        starts = np.flatnonzero(g & ~np.concatenate([[False], g[:-1]]))
        ends = np.flatnonzero(g & ~np.concatenate([g[1:], [False]]))
        for s, e in zip(starts, ends):
            score -= 200 * int(s > 0) + 200 * int(e < len(p) - 1)
    return score


# A path that leaves a band of half-width 400 gives up some 57,000 (380 bases of
# 151 or more), a substitution costs 225 at most, the gaps below 12,000: 60
# substitutions keep the band, 3% do not, and the full DP runs again.
@pytest.mark.parametrize("rate,kept", [(0.03, 0), (60, 1)])
@pytest.mark.parametrize("n", [200_500, 400_500])
def test_full_and_banded_agree(ctx, n, rate, kept):
    rng = np.random.default_rng(n)
    a = rng.integers(0, 4, n, dtype=np.uint8)
    b = a.copy()
    hit = rng.random(n) < (rate if rate < 1 else 0)
    if rate > 1:
        hit[rng.integers(0, n, rate)] = True
    b[hit] = rng.integers(0, 4, int(hit.sum()), dtype=np.uint8)
    b = np.concatenate([b[:n // 5], b[n // 5 + 90:n // 2], rng.integers(0, 4, 60, dtype=np.uint8), b[n // 2:]])
    oa, ob = np.array([0, len(a)]), np.array([0, len(b)])
    assert min(len(a), len(b)) > (400_000 if n > 400_000 else 200_000)
    scores, paths = ctx.gap_align_batch(a, oa, b, ob)
    assert _path_score(a, b, paths[0]) == scores[0]
    banded = ctx.gap_align_banded(a, oa, b, ob, np.array([-20], np.int32), np.array([400], np.int32))
    assert banded[2][0] == kept
    assert banded[0][0] == scores[0] and banded[1] == paths
    if n > 400_000:  # bits are not stored there, asked for or not
        ctx.set_dp_checkpoint(False)
        try:
            again = ctx.gap_align_batch(a, oa, b, ob)
        finally:
            ctx.set_dp_checkpoint(True)
        assert again[0][0] == scores[0] and again[1] == paths
