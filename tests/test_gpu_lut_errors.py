"""LUT calls that end in an error which some of a launch's CTAs raise while
others have yet to start: the error is reported, the handle stays usable and
the next call's result is right."""
import numpy as np
import pytest

import mvg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = mvg.Context(0)
    yield c
    c.close()


def _blocks(n, g_start=1, r_start=1):
    rows = np.frombuffer(b"ACGT", np.uint8)[np.arange(n) % 4].copy()
    return np.array([g_start], np.int64), np.array([r_start], np.int64), np.array([0, n], np.uint64), rows


def _build(ctx, n, glen, gs, rs, off, rows, fill=1):
    lut = np.full(glen, 7, np.int32)
    genome = np.frombuffer(b"ACGT", np.uint8)[np.arange(glen) % 4].copy()
    rc = mvg.load_library().mvg_build_index_lut(
        ctx.handle, mvg._ptr(gs), mvg._ptr(rs), mvg._ptr(off), mvg._ptr(rows), mvg._ptr(rows), 1, mvg._ptr(genome), glen,
        mvg._ptr(genome), glen, fill, 300, fill, 20, mvg._ptr(lut), glen)
    return rc, lut


@pytest.mark.parametrize("n", [5000, 3_000_000])
def test_errors_of_many_ctas(ctx, n):
    want = np.arange(n, dtype=np.int32)
    for kind in ("overflow", "range", "zero"):
        for _ in range(5):
            if kind == "overflow":  # reference indices past int32 from the second half on
                gs, rs, off, rows = _blocks(n, 1, 2**31 - n // 2)
                rc, _ = _build(ctx, n, n, gs, rs, off, rows)
                assert rc == 9  # MVG_ERR_OVERFLOW
            elif kind == "range":  # genome indices below -n
                gs, rs, off, rows = _blocks(n, -3 * n, 1)
                rc, _ = _build(ctx, n, n, gs, rs, off, rows)
                assert rc == 8  # MVG_ERR_RANGE
            else:  # fixZeroIdx finds no entry: the block lies outside the genome
                gs, rs, off, rows = _blocks(n, n + 1, 1)
                rc, _ = _build(ctx, n, n, gs, rs, off, rows)
                assert rc == 8
            gs, rs, off, rows = _blocks(n)
            rc, lut = _build(ctx, n, n, gs, rs, off, rows)
            assert rc == 0, mvg.load_library().mvg_last_error()
            np.testing.assert_array_equal(lut, want)
