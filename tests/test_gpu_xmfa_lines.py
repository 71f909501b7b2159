"""XMFA text where its pieces meet, short and long enough for either kernel: rows of one to a few columns, of whole
lines and one more or less, empty blocks, absent sequences, and rows that
start off a word boundary, against the text put together line by line."""
import numpy as np
import pytest

import mvg
import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import build as pkg_build
    pkg_build.build()
    c = mvg.Context(0)
    yield c
    c.close()


def text_of(names, starts, lengths, rows, off):
    out = ["#FormatVersion Mauve1\n"]
    for q in range(2):
        out.append("#Sequence%dFile\t%s\n#Sequence%dFormat\tFastA\n" % (q + 1, names[q], q + 1))
    for b in range(len(off) - 1):
        lo, hi = int(off[b]), int(off[b + 1])
        if lo == hi:
            continue
        for q in range(2):
            s, n = int(starts[2 * b + q]), int(lengths[2 * b + q])
            if s == 0 and b > 0:
                continue
            where = "0-0 +" if s == 0 else "%d-%d %s" % (abs(s), abs(s) + n - 1, "+" if s > 0 else "-")
            out.append("> %d:%s %s\n" % (q + 1, where, names[q]))
            row = rows[q][lo:hi].tobytes().decode()
            out += [row[c:c + 80] + "\n" for c in range(0, len(row), 80)]
        out.append("=\n")
    return "".join(out).encode()


@pytest.mark.parametrize("shift", [(0, 0), (1, 2), (3, 16)])
@pytest.mark.parametrize("widths", [[1], [79], [80], [81], [1, 2, 3, 4, 5, 0, 1, 1], [160, 161, 159, 0, 80],
                                    [4, 76, 77, 78, 400], [5000, 1, 12_345], [3] * 300, [180_000, 7],
                                    [196_000], [300_001, 1, 80, 79, 5]])
def test_text_of_uneven_blocks(ctx, widths, shift):
    import torch
    rng = np.random.default_rng(sum(widths) + len(widths))
    off = np.concatenate([[0], np.cumsum(widths)]).astype(np.uint64)
    n = int(off[-1])
    rows = [synth.random_bases(rng, n) for _ in range(2)]
    starts = rng.integers(-10 ** 6, 10 ** 6, 2 * len(widths)).astype(np.int64)
    starts[rng.random(len(starts)) < 0.2] = 0
    lengths = rng.integers(1, 10 ** 6, 2 * len(widths)).astype(np.int64)
    names = ("a.fasta", "dir/b")
    want = text_of(names, starts, lengths, rows, off)
    assert ctx.xmfa_write(*names, starts, lengths, rows[0], rows[1], off) == want
    dev = []
    for row, k in zip(rows, shift):
        t = torch.zeros(n + k, dtype=torch.uint8, device="cuda")
        t[k:] = torch.from_numpy(row).cuda()
        dev.append(t)
    out = torch.zeros(len(want) + 64, dtype=torch.uint8).pin_memory()
    got = ctx.xmfa_write_dev(*names, starts, lengths, dev[0].data_ptr() + shift[0], dev[1].data_ptr() + shift[1], off,
                             out.data_ptr(), len(want))
    assert got == len(want) and out[:got].numpy().tobytes() == want and not out[got:].any()
