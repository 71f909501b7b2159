"""Performance cases of the pairwise anchoring and gap-alignment path.

Each case is one call (or the pair of calls a program makes together) of the
library's public entry points on seeded synthetic data with the sizes and
mutation spectra of the repository's workloads.  Inputs are drawn on the GPU;
a program that aligns many genome pairs keeps one handle, so all states of a
process share one.  Outputs are the caller's own buffers, sized by the case,
with the counts that say how much of them is filled.
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "mauve-py_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import bandnet  # noqa: E402
import indexutils  # noqa: E402
import mvg  # noqa: E402

DEV = "cuda"
WEIGHTS = os.path.join(PKG, "bandnet_weights.npz")
DIMS = [(256, 528), (256, 256), (256, 256), (2, 256)]


def listed():
    return [
        # one inter-anchor gap by itself: what a caller without a batch pays (latency, launches)
        {"name": "gapdp_one", "path": "gapdp", "gaps": 1, "shortest": 300, "longest": 320, "divergence": 0.1},
        # the batched full gap DP: lengths log-uniform 10-20,000, divergence U(0, 30%), a handful of gaps of tens of kbp
        {"name": "gapdp_batch", "path": "gapdp", "gaps": 4000, "shortest": 10, "longest": 20000, "divergence": 0.3},
        # the gaps of a recoded genome pair with the learned band: proposal by the network, banded DP, exact fallback
        {"name": "gapdp_learned_band", "path": "band", "gaps": 30011, "shortest": 20, "longest": 5000},
        # anchoring two plain 1 Mbp genomes that lie in host memory (FASTA just read)
        {"name": "anchor_plain_host", "path": "anchor", "kind": "plain", "bases": 1000000, "host": True},
        # anchoring the 4.6 Mbp recoded pair (repeats, codon substitutions, rearrangements), genomes resident
        {"name": "anchor_recoded", "path": "anchor", "kind": "recoded", "bases": 4600000, "host": False},
        # anchoring a 12 Mbp many-contig pair, 8% diverged, 1,000 rearrangements (weight 17: 64-bit keys)
        {"name": "anchor_large", "path": "anchor", "kind": "large", "bases": 12000000, "host": False},
        # one genome's sorted mer list with its mers (what the .sslist cache holds), an odd length
        {"name": "sorted_mers", "path": "sml", "bases": 3981477},
        # a recursion round's gap anchor search: gaps of 200-20,000 bp in one call, the overlap filter included
        {"name": "gap_search", "path": "search", "gaps": 5003, "shortest": 200, "longest": 20000},
        # both gapped-alignment passes over the LCBs of a genome pair (host rows in, host rows out)
        {"name": "refine_lcbs", "path": "refine", "lcbs": 120, "shortest": 6000, "longest": 18000},
        # buildIndex's LUT of a bacterial genome from its aligned blocks
        {"name": "index_lut", "path": "lut", "bases": 4600000, "blocks": 64},
        # the XMFA text of the same alignment, rows on the device, text into pinned memory
        {"name": "xmfa_text", "path": "xmfa", "bases": 4600000, "blocks": 64},
        # loss and gradients of one training minibatch of the band network (forward and backward)
        {"name": "band_net_gradient", "path": "gradient", "gaps": 4096},
    ]


def _between(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    path = rng.choice(["gapdp", "gapdp", "band", "anchor", "anchor", "sml", "search", "refine", "lut", "xmfa",
                       "gradient"])
    if path == "gapdp":
        longest = _between(rng, 64, 20000)
        return {"path": path, "gaps": _between(rng, 1, 4000), "shortest": _between(rng, 1, min(longest, 400)),
                "longest": longest, "divergence": round(rng.uniform(0.02, 0.3), 3)}
    if path == "band":
        return {"path": path, "gaps": _between(rng, 100, 30011), "shortest": 20, "longest": _between(rng, 300, 5000)}
    if path == "anchor":
        kind = rng.choice(["plain", "recoded", "large"])
        lo, hi = {"plain": (20000, 1000000), "recoded": (200000, 4600000), "large": (1000000, 12000000)}[kind]
        return {"path": path, "kind": kind, "bases": _between(rng, lo, hi), "host": rng.random() < 0.3}
    if path == "sml":
        return {"path": path, "bases": _between(rng, 5000, 4600000)}
    if path == "search":
        return {"path": path, "gaps": _between(rng, 1, 5003), "shortest": 200, "longest": _between(rng, 1000, 20000)}
    if path == "refine":
        shortest = _between(rng, 300, 6000)
        return {"path": path, "lcbs": _between(rng, 1, 120), "shortest": shortest, "longest": 3 * shortest}
    if path in ("lut", "xmfa"):
        return {"path": path, "bases": _between(rng, 20000, 4600000), "blocks": _between(rng, 1, 200)}
    return {"path": path, "gaps": _between(rng, 64, 4096)}


# ------------------------------------------------------------- random data

def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _rand(g, n):
    return torch.rand(n, generator=g, device=DEV)


def _codes(g, n, gc=0.5):
    """n base codes (A, C, G, T = 0..3) at the given GC content."""
    u = _rand(g, n)
    code = (u >= (1 - gc) / 2).to(torch.uint8)
    code += u >= 0.5
    code += u >= (1 + gc) / 2
    return code


def _ascii(codes):
    return torch.tensor(list(b"ACGT"), dtype=torch.uint8, device=DEV)[codes.long()]


def _geometric(g, n, mean):
    u = _rand(g, n).clamp_(1e-7, 1 - 1e-7)
    return (torch.log(u) / math.log(1 - 1 / mean)).floor_().long() + 1


def _offsets(lens):
    off = torch.zeros(len(lens) + 1, dtype=torch.int64, device=DEV)
    off[1:] = torch.cumsum(lens, 0)
    return off


def _mutate(g, seq, off, sub, indel, mean):
    """A copy of every sequence seq[off[k]:off[k+1]] with substitutions at
    rate sub (per base, or one rate per base) and insertions and deletions
    starting at rate indel, lengths geometric.  No copy is empty."""
    n = len(seq)
    other = (seq + torch.randint(1, 4, (n,), generator=g, device=DEV, dtype=torch.uint8)) % 4
    b = torch.where(_rand(g, n) < sub, other, seq)
    event = torch.nonzero(_rand(g, n) < indel).view(-1)
    length = _geometric(g, len(event), mean)
    ins = _rand(g, len(event)) < 0.5
    end = off[torch.searchsorted(off, event, right=True)]
    edge = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    edge.scatter_add_(0, event[~ins], torch.ones_like(event[~ins]))
    edge.scatter_add_(0, torch.minimum(event + length, end)[~ins], -torch.ones_like(event[~ins]))
    count = (torch.cumsum(edge[:-1], 0) <= 0).long()
    count[event[ins]] += length[ins] * count[event[ins]]
    total = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(count, 0, out=total[1:])
    empty = total[off[1:]] == total[off[:-1]]
    count[off[:-1][empty]] = 1
    torch.cumsum(count, 0, out=total[1:])
    out = torch.repeat_interleave(b, count)
    copied = torch.zeros(len(out), dtype=torch.bool, device=DEV)
    copied[total[:-1][count > 0]] = True
    fresh = torch.randint(0, 4, (len(out),), generator=g, device=DEV, dtype=torch.uint8)
    return torch.where(copied, out, fresh), total[off]


def _lengths(g, case):
    """Lengths spread evenly over the logarithm of the case's range, in random order."""
    n = case["gaps"]
    lo, hi = math.log(case["shortest"]), math.log(case["longest"])
    at = (torch.arange(n, device=DEV, dtype=torch.float64) + 0.5) / n
    la = torch.exp(lo + (hi - lo) * at).round().long().clamp_(case["shortest"], case["longest"])
    return la[torch.randperm(n, generator=g, device=DEV)]


def _gaps(g, case, max_divergence):
    """Inter-anchor gaps: lengths log-uniform, the second sequence derived
    from the first (substitutions to indels 9:1, indel lengths of mean 3)."""
    n, la = case["gaps"], _lengths(g, case)
    oa = _offsets(la)
    sa = _codes(g, int(oa[-1]))
    div = torch.repeat_interleave(_rand(g, n) * max_divergence, la)
    sb, ob = _mutate(g, sa, oa, 0.9 * div, 0.1 * div / 3, 3.0)
    return sa, oa, sb, ob


def _recoded_gaps(g, case):
    """Gaps as a recoded genome pair has them: 90% with 0.5-3% substitutions
    and few indels, 10% divergent (25-40%)."""
    n, la = case["gaps"], _lengths(g, case)
    oa = _offsets(la)
    sa = _codes(g, int(oa[-1]))
    far, u = _rand(g, n) < 0.1, _rand(g, n)
    div = 0.25 + 0.15 * u
    sub = torch.where(far, 0.9 * div, 0.005 + 0.025 * u)
    indel = torch.where(far, 0.1 * div / 3, torch.full_like(u, 0.0005))
    sb, ob = _mutate(g, sa, oa, torch.repeat_interleave(sub, la), torch.repeat_interleave(indel, la), 4.0)
    return sa, oa, sb, ob


def _rearrange(r, s, n, lo, hi):
    """n inversions and translocations of segments of lo..hi bases."""
    for _ in range(n):
        size = r.randint(lo, hi)
        if size >= len(s) // 2:
            continue
        p = r.randrange(0, len(s) - size)
        if r.random() < 0.5:
            s[p:p + size] = 3 - s[p:p + size].flip(0)
        else:
            rest = torch.cat([s[:p], s[p + size:]])
            q = r.randrange(0, len(rest))
            s = torch.cat([rest[:q], s[p:p + size], rest[q:]])
    return s


def _repeats(g, r, s, families, copies, gc):
    """Copies of repeat families written over random places of s."""
    fams = [_codes(g, size, gc) for size in families]
    for k in range(copies):
        f = fams[k % len(fams)]
        if len(f) < len(s) // 4:
            p = r.randrange(0, len(s) - len(f))
            s[p:p + len(f)] = f
    return s


def _genomes(g, r, kind, n):
    """A pair of genomes (base codes): A is a mutated, rearranged B."""
    off = torch.tensor([0, n], dtype=torch.int64, device=DEV)
    if kind == "plain":  # 0.5% substitutions, 50 indels and two 10 kbp inversions per Mbp
        b = _codes(g, n)
        a, _ = _mutate(g, b, off, 0.005, 50e-6, 5.0)
        for _ in range(2):
            size = min(10000, n // 10)
            p = r.randrange(0, len(a) - size)
            a[p:p + size] = 3 - a[p:p + size].flip(0)
        return a, b
    if kind == "recoded":  # 3% of codon third positions in ORFs, 0.05% elsewhere, repeats of 1.3 kbp
        b = _repeats(g, r, _codes(g, n, 0.508), [1300], max(1, 40 * n // 4600000), 0.508)
        norf = max(1, 4300 * n // 4600000)
        orf = (torch.clamp(950 + 250 * torch.randn(norf, generator=g, device=DEV), min=90).long() // 3) * 3
        slack = torch.sort(torch.randint(0, max(1, n - int(orf.sum())), (norf,), generator=g, device=DEV))[0]
        start = slack + torch.cumsum(orf, 0) - orf
        at = torch.arange(n, device=DEV)
        k = torch.searchsorted(start, at, right=True) - 1
        into = at - start[k.clamp(min=0)]
        third = (k >= 0) & (into < orf[k.clamp(min=0)]) & (into % 3 == 2)
        sub = torch.where(third, torch.tensor(0.03, device=DEV), torch.tensor(0.0005, device=DEV))
        a, _ = _mutate(g, b, off, sub, 200 / 4.6e6, 4.0)
        return _rearrange(r, a, 5, 5000, 50000), b
    # many contigs at GC 0.38, five repeat families, 8% substitutions, many rearrangements
    b = _repeats(g, r, _codes(g, n, 0.38), [r.randint(300, 6000) for _ in range(5)], max(5, 300 * n // 12000000), 0.38)
    a, _ = _mutate(g, b, off, 0.08, 2000 / 12e6, 6.0)
    return _rearrange(r, a, max(1, 1000 * n // 12000000), 1000, 100000), b


def _alignment(g, r, case):
    """Aligned rows of a genome against a reference (2% substitutions, 0.05%
    indels) cut into shuffled blocks: (genome starts, reference starts,
    column offsets, genome rows, reference rows, genome, reference)."""
    n, nblocks = case["bases"], case["blocks"]
    ref = _codes(g, n)
    other = (ref + torch.randint(1, 4, (n,), generator=g, device=DEV, dtype=torch.uint8)) % 4
    gen = _ascii(torch.where(_rand(g, n) < 0.02, other, ref))
    ref = _ascii(ref)
    event = torch.nonzero(_rand(g, n) < 0.0005).view(-1)
    length = _geometric(g, len(event), 3.3)
    ins = _rand(g, len(event)) < 0.5
    edge = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    edge.scatter_add_(0, event[~ins], torch.ones_like(event[~ins]))
    edge.scatter_add_(0, (event + length).clamp(max=n)[~ins], -torch.ones_like(event[~ins]))
    gen[torch.cumsum(edge[:-1], 0) > 0] = ord("-")
    count = torch.ones(n, dtype=torch.int64, device=DEV)
    count[event[ins]] += length[ins]
    first = torch.cumsum(count, 0) - count
    cols = int(count.sum())
    rows_g, rows_r = _ascii(_codes(g, cols)), torch.full((cols,), ord("-"), dtype=torch.uint8, device=DEV)
    rows_g[first], rows_r[first] = gen, ref
    cuts = sorted(r.sample(range(1, cols), nblocks - 1))
    bounds = [0] + cuts + [cols]
    order = list(range(nblocks))
    r.shuffle(order)
    zero = torch.zeros(1, dtype=torch.int64, device=DEV)
    before = [torch.cat([zero, torch.cumsum((x != ord("-")).long(), 0)]) for x in (rows_g, rows_r)]
    at = torch.tensor([bounds[b] for b in order], device=DEV)
    to = torch.tensor([bounds[b + 1] for b in order], device=DEV)
    starts = [x[at] + 1 for x in before]
    lengths = [x[to] - x[at] for x in before]
    genome = rows_g[rows_g != ord("-")]
    pick = [torch.cat([x[bounds[b]:bounds[b + 1]] for b in order]) for x in (rows_g, rows_r)]
    return starts, lengths, _offsets(to - at), pick[0], pick[1], genome, ref


def _lcbs(g, r, case):
    """LCBs as two gapped rows each: a random sequence and a copy with 2-25%
    substitutions, one-sided gap runs at 1% of the columns."""
    out, count = [], case["lcbs"]
    order = r.sample(range(count), count)
    for k in order:
        n = case["shortest"] + (case["longest"] - case["shortest"]) * (2 * k + 1) // (2 * count)
        a = _codes(g, n)
        other = (a + torch.randint(1, 4, (n,), generator=g, device=DEV, dtype=torch.uint8)) % 4
        b = torch.where(_rand(g, n) < r.uniform(0.02, 0.25), other, a)
        rows = [_ascii(a), _ascii(b)]
        event = torch.nonzero(_rand(g, n) < 0.01).view(-1)
        length, side = _geometric(g, len(event), 4.0), _rand(g, len(event)) < 0.5
        for row, mine in zip(rows, (side, ~side)):
            edge = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
            edge.scatter_add_(0, event[mine], torch.ones_like(event[mine]))
            edge.scatter_add_(0, (event + length).clamp(max=n)[mine], -torch.ones_like(event[mine]))
            row[torch.cumsum(edge[:-1], 0) > 0] = ord("-")
        keep = (rows[0] != ord("-")) | (rows[1] != ord("-"))
        out.append(tuple(row[keep].cpu().numpy() for row in rows))
    return out


def _features(g, n):
    """Band-network inputs (two 4-mer spectra and log lengths, bf16) and
    targets (diagonal offset / 100, log(1 + half-width)) of n gaps."""
    la = torch.exp(math.log(20) + math.log(250) * _rand(g, n)).floor_()
    lb = (la * (1 + 0.02 * torch.randn(n, generator=g, device=DEV))).floor_().clamp_(min=10)
    mean = ((la - 3) / 256).unsqueeze(1).expand(n, 256).contiguous()
    shared = torch.poisson(mean, generator=g)
    lost = torch.poisson(0.05 * mean, generator=g)
    x = torch.zeros(n, 528, device=DEV)
    x[:, :256] = shared * (256 / (la - 3)).unsqueeze(1)
    x[:, 256:512] = (shared + lost) * (256 / (lb - 3)).unsqueeze(1)
    x[:, 512], x[:, 513] = torch.log(la) / 5, torch.log(lb) / 5
    half = torch.exp(math.log(16) + math.log(20) * _rand(g, n))
    target = torch.stack([0.1 * torch.randn(n, generator=g, device=DEV), torch.log1p(half)], 1)
    return x.to(torch.bfloat16).contiguous(), target.contiguous()


# ------------------------------------------------------------------- cases

_kept = {}


def _handle():
    """The handle and the trained band network that a program keeps."""
    if not _kept:
        ctx = mvg.Context(torch.cuda.current_device())
        w = np.load(WEIGHTS)
        ctx.set_band_whole_fraction(float(w["whole"]))
        ctx.set_band_gate(int(w["gate"]))
        _kept.update(ctx=ctx, net=bandnet.BandNet(ctx, params=w["params"]), alpha=float(w["alpha"]),
                     beta=float(w["beta"]))
    return _kept


def _gap_state(s, sa, oa, sb, ob):
    n = len(oa) - 1
    path_off = _offsets(oa[1:] - oa[:-1] + ob[1:] - ob[:-1])
    slots = 2 * len(sa) + len(sa) // 4 + 64 * n + 1024  # room for the sum of both lengths of every gap
    assert int(path_off[-1]) <= slots
    s.update(n=n, sa=sa, oa=oa, sb=sb, ob=ob, path_off=path_off, chars_a=_ascii(sa), chars_b=_ascii(sb),
             scores=torch.zeros(n, dtype=torch.int32, device=DEV),
             paths=torch.zeros(slots, dtype=torch.uint8, device=DEV),
             path_len=torch.zeros(n, dtype=torch.int64, device=DEV),
             rows_a=torch.zeros(slots, dtype=torch.uint8, device=DEV),
             rows_b=torch.zeros(slots, dtype=torch.uint8, device=DEV))


def prepare(case, seed):
    g, r = _generator(seed), random.Random(int(seed))
    s = {"path": case["path"], **_handle()}
    path = case["path"]
    if path == "gapdp":
        _gap_state(s, *_gaps(g, case, case["divergence"]))
    elif path == "band":
        _gap_state(s, *_recoded_gaps(g, case))
    elif path in ("anchor", "sml"):
        if path == "anchor":
            a, b = (_ascii(x) for x in _genomes(g, r, case["kind"], case["bases"]))
        else:
            a = b = _ascii(_codes(g, case["bases"], 0.508))
        s["seed"] = mvg.get_seed(mvg.default_seed_weight((len(a) + len(b)) // 2), mvg.CODING_SEED)
        if path == "sml":
            s.update(seq=a, pos=torch.zeros(len(a), dtype=torch.int32, device=DEV),
                     mer=torch.zeros(len(a), dtype=torch.int64, device=DEV))
        else:
            s.update(host=case["host"], cap=case["bases"] // 4 + 1024)
            if case["host"]:
                s.update(a=a.cpu().numpy(), b=b.cpu().numpy(), out=np.zeros((s["cap"], 3), np.int64))
            else:
                s.update(a=a, b=b, out=torch.zeros(s["cap"], 3, dtype=torch.int64, device=DEV))
    elif path == "search":
        sa, oa, sb, ob = _gaps(g, case, 0.3)
        genomes, rows = [], []
        for seq, off in ((sa, oa), (sb, ob)):
            lens = off[1:] - off[:-1]
            start = off[:-1] + 100 * (torch.arange(len(lens), device=DEV) + 1)  # 100 bases between gaps
            genome = _codes(g, int(off[-1]) + 100 * (len(lens) + 1))
            genome[torch.arange(len(seq), device=DEV) + torch.repeat_interleave(start - off[:-1], lens)] = seq
            genomes.append(_ascii(genome))
            rows += [start, lens]
        s.update(a=genomes[0], b=genomes[1], gaps=torch.stack(rows, 1).cpu().numpy(), cap=len(sa) // 8 + 1024)
        s.update(out=np.zeros((s["cap"], 3), np.int64), off=np.zeros(case["gaps"] + 1, np.uint64))
    elif path == "refine":
        lcbs = _lcbs(g, r, case)
        off = np.zeros(len(lcbs) + 1, np.uint64)
        off[1:] = np.cumsum([len(a) for a, _ in lcbs])
        cap = int(1.3 * case["lcbs"] * (case["shortest"] + case["longest"]) / 2) + 1024
        s.update(n=len(lcbs), off=off, rows_a=np.concatenate([a for a, _ in lcbs]), cap=cap,
                 rows_b=np.concatenate([b for _, b in lcbs]), out_a=np.zeros(cap, np.uint8),
                 out_b=np.zeros(cap, np.uint8), out_off=np.zeros(len(off), np.uint64))
    elif path in ("lut", "xmfa"):
        starts, lengths, off, rows_g, rows_r, genome, ref = _alignment(g, r, case)
        s.update(off=off, rows_g=rows_g, rows_r=rows_r, genome=genome, ref=ref, nblocks=case["blocks"])
        if path == "lut":
            room = case["bases"] + case["bases"] // 50 + 4096
            s.update(starts=starts, lut=torch.zeros(room, dtype=torch.int32, device=DEV))
        else:
            flip = torch.where(torch.arange(case["blocks"], device=DEV) % 2 == 1, -1, 1)  # strands
            s.update(starts=torch.stack([starts[0], starts[1] * flip], 1).view(-1).cpu().numpy(),
                     lengths=torch.stack(lengths, 1).view(-1).cpu().numpy(), off=off.cpu().numpy().astype(np.uint64))
            s["cap"] = 2 * case["bases"] + case["bases"] // 10 + 8192 + 300 * case["blocks"]
            s["text"] = torch.zeros(s["cap"], dtype=torch.uint8, pin_memory=True)
    else:
        s["x"], s["target"] = _features(g, case["gaps"])
    torch.cuda.synchronize()
    return s


def run(s):
    ctx, path = s["ctx"], s["path"]
    if path in ("gapdp", "band"):
        seqs = [s[k].data_ptr() for k in ("sa", "oa", "sb", "ob")]
        outs = [s[k].data_ptr() for k in ("scores", "paths", "path_off", "path_len")]
        bands = ()
        if path == "gapdp":
            ctx.gap_align_batch_dev(*seqs, s["n"], *outs)
        else:
            # which gaps the band was kept for is no part of the alignment and is not returned
            bands = s["net"].propose_dev(*seqs, s["n"], s["alpha"], s["beta"])
            ctx.gap_align_banded_dev(*seqs, s["n"], *bands, *outs)
        # the aligned rows (the paths fill only the heads of their slots)
        mvg._check(mvg.load_library().mvg_path_rows_dev(
            ctx.handle, s["chars_a"].data_ptr(), seqs[1], s["chars_b"].data_ptr(), seqs[3], s["n"], outs[1], outs[2],
            outs[3], s["rows_a"].data_ptr(), s["rows_b"].data_ptr()))
        return [s["scores"], s["path_len"], s["rows_a"], s["rows_b"], *bands]
    if path == "anchor":
        if s["host"]:
            n = ctypes.c_uint64(0)
            mvg._check(mvg.load_library().mvg_pairwise_matches(
                ctx.handle, s["a"].ctypes.data, len(s["a"]), s["b"].ctypes.data, len(s["b"]), s["seed"],
                s["out"].ctypes.data, s["cap"], ctypes.byref(n)))
            return int(n.value), s["out"]
        n = ctx.pairwise_matches_dev(s["a"].data_ptr(), len(s["a"]), s["b"].data_ptr(), len(s["b"]), s["seed"],
                                     s["out"].data_ptr(), s["cap"])
        return n, s["out"]
    if path == "sml":
        n = ctx.sml_build_dev(s["seq"].data_ptr(), len(s["seq"]), s["seed"], s["pos"].data_ptr(), s["mer"].data_ptr(),
                              len(s["seq"]))
        return s["pos"][:n], s["mer"][:n]
    if path == "search":
        n = ctypes.c_uint64(0)
        mvg._check(mvg.load_library().mvg_gap_anchor_search_dev(
            ctx.handle, s["a"].data_ptr(), len(s["a"]), s["b"].data_ptr(), len(s["b"]), s["gaps"].ctypes.data,
            len(s["gaps"]), s["out"].ctypes.data, s["cap"], s["off"].ctypes.data, ctypes.byref(n)))
        return int(n.value), s["out"], s["off"].view(np.int64)
    if path == "refine":
        mvg._check(mvg.load_library().mvg_gapped_alignment(
            ctx.handle, s["rows_a"].ctypes.data, s["rows_b"].ctypes.data, s["off"].ctypes.data, s["n"], 20000.0, 3,
            s["out_a"].ctypes.data, s["out_b"].ctypes.data, s["out_off"].ctypes.data, s["cap"]))
        return s["out_off"].view(np.int64), s["out_a"], s["out_b"]
    if path == "lut":
        indexutils.buildIndexLutDev(s["starts"][0].data_ptr(), s["starts"][1].data_ptr(), s["off"].data_ptr(),
                                    s["rows_g"].data_ptr(), s["rows_r"].data_ptr(), s["nblocks"],
                                    s["genome"].data_ptr(), len(s["genome"]), s["ref"].data_ptr(), len(s["ref"]),
                                    s["lut"].data_ptr(), len(s["genome"]), ctx=ctx)
        return s["lut"]
    if path == "xmfa":
        n = ctx.xmfa_write_dev("genome.fasta", "reference.fasta", s["starts"], s["lengths"], s["rows_g"].data_ptr(),
                               s["rows_r"].data_ptr(), s["off"], s["text"].data_ptr(), s["cap"])
        return n, s["text"]
    return list(s["net"].grad_dev(s["x"].data_ptr(), s["target"].data_ptr(), len(s["x"])))


def work(case):
    path = case["path"]
    if path in ("gapdp", "band", "search"):
        lo, hi = math.log(case["shortest"]), math.log(case["longest"])
        mean = (case["longest"] - case["shortest"]) / (hi - lo) if hi > lo else case["longest"]
        square = (case["longest"] ** 2 - case["shortest"] ** 2) / (2 * (hi - lo)) if hi > lo else mean * mean
        bases = 2 * case["gaps"] * mean
        if path == "search":
            return {"bytes": bases, "flops": 0}
        # codes and letters read, two rows written; ten integer operations a cell of the matrix (a
        # band's cells are counted as a tenth of it)
        return {"bytes": 4 * bases, "flops": case["gaps"] * square * (10 if path == "gapdp" else 1)}
    if path == "anchor":
        return {"bytes": 2 * case["bases"], "flops": 0}
    if path == "sml":
        return {"bytes": 13 * case["bases"], "flops": 0}
    if path == "refine":
        # four rows read and written; windows of a few hundred columns are aligned twice
        cols = case["lcbs"] * (case["shortest"] + case["longest"]) / 2
        return {"bytes": 4 * cols, "flops": 2 * 10 * 200 * cols}
    if path == "lut":
        return {"bytes": 8 * case["bases"], "flops": 0}
    if path == "xmfa":
        return {"bytes": 4 * case["bases"], "flops": 0}
    weights = [o * i for o, i in DIMS]
    return {"bytes": case["gaps"] * (2 * 528 + 8) + 8 * sum(weights),
            "flops": 2 * case["gaps"] * (2 * sum(weights) + sum(weights[1:]))}


def exact(case, seed):
    """Loss and gradients of the band network in 64 bits; the other paths
    return whole numbers and bytes."""
    if case["path"] != "gradient":
        return None
    x, target = _features(_generator(seed), case["gaps"])
    flat = torch.from_numpy(np.load(WEIGHTS)["params"]).to(DEV).double().requires_grad_(True)
    h, at = x.double(), 0
    for k, (o, i) in enumerate(DIMS):
        w, b = flat[at:at + o * i].view(o, i), flat[at + o * i:at + o * i + o]
        at += o * i + o
        h = h @ w.T + b
        if k < 3:
            h = torch.nn.functional.gelu(h)
    loss = ((h - target.double()) ** 2).sum() / len(x)
    loss.backward()
    return [flat.grad, float(loss.detach())]
