"""Performance cases: what a program that uses genomics_b200 has it do.

Sequences are seeded and synthetic, with the shapes and divergence of the
generator's workloads (genomics_b200/synth.py): reads against the window they
came from, and pairs whose query is the target with substitutions and indels.
Everything random is drawn on the GPU from the seed alone.

A case is a flat dict.  `op` says which entry point a pass calls:

  sw_call     align.smith_waterman_banded, one pair per call
  wfa_call    align.wfa_affine_cpu, one pair per call
  sw          GenomicsDevice.sw_banded on batches resident on the device
  sw_host     GenomicsDevice.sw_banded from page-locked host SequenceBatches
  nw          GenomicsDevice.nw_banded on resident batches
  wfa         GenomicsDevice.wfa_affine on resident batches
  wfa_cigar   GenomicsDevice.wfa_cigar (costs and CIGAR runs) on resident batches

`n` pairs; template lengths are log-uniform in [lo, hi]; `pad` extra target
bases on both sides of the template (0: global alignment of the whole target);
`div` the largest per-pair divergence (smallest: a tenth of it), 70%
substitutions, 15% insertions, 15% deletions.  `bands` is one band for all
pairs, or several to draw from per pair; `scores` are match, mismatch,
gap_open, gap_extend.  WFA cases take x4 o6 e2; max_error 0 means the bound
that no pair passes.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "computational-genomics-mojo_b200"))
from genomics_b200 import align, synth  # noqa: E402
from genomics_b200.align import AlignConfig, WFAConfig  # noqa: E402
from genomics_b200.core import SequenceBatch, get_view  # noqa: E402
from genomics_b200.device import SW_RESULT_DTYPE  # noqa: E402

READ_SCORES = "2,-4,-4,-2"     # the benchmark's scoring
DEFAULT_SCORES = "2,-3,-5,-2"  # align.default_config()


def listed():
    return [
        # the reference's per-pair function called in a loop: one read, default config
        dict(name="sw_call_read", op="sw_call", n=1, lo=150, hi=150, pad=25, div=0.05,
             bands="32", scores=DEFAULT_SCORES),
        # one amplicon-sized pair per call
        dict(name="wfa_call_1kbp", op="wfa_call", n=1, lo=1000, hi=1000, pad=0, div=0.04,
             max_error=0),
        # the benchmark: a million 150 bp reads against their 200 bp windows
        dict(name="sw_reads_1m", op="sw", n=1_000_000, lo=150, hi=150, pad=25, div=0.03,
             bands="32", scores=READ_SCORES, pinned=True),
        # trimmed reads straight from host memory, copies inside the call
        dict(name="sw_host_reads_300k", op="sw_host", n=300_000, lo=75, hi=150, pad=25,
             div=0.05, bands="32", scores=DEFAULT_SCORES, pinned=True),
        # mixed-length batch with a band per pair
        dict(name="sw_mixed_50k", op="sw", n=50_000, lo=100, hi=2000, pad=10, div=0.08,
             bands="16,32,64,128", scores=READ_SCORES, pinned=True),
        # a band width between the powers of two, ragged lengths, results into a new array
        dict(name="sw_band40_100k", op="sw", n=100_000, lo=100, hi=300, pad=20, div=0.06,
             bands="40", scores=READ_SCORES, pinned=False),
        # long reads against their locus, wide band
        dict(name="sw_long_4k", op="sw", n=4_000, lo=2000, hi=10_000, pad=20, div=0.05,
             bands="128", scores=DEFAULT_SCORES, pinned=False),
        # global alignment of reads to their origin windows
        dict(name="nw_reads_500k", op="nw", n=500_000, lo=150, hi=150, pad=0, div=0.04,
             bands="32", scores=READ_SCORES),
        # global alignment of ragged amplicons, wider band
        dict(name="nw_band64_20k", op="nw", n=20_000, lo=100, hi=1000, pad=0, div=0.08,
             bands="64", scores=DEFAULT_SCORES),
        # edit-cost filter over short reads, default max_error
        dict(name="wfa_reads_500k", op="wfa", n=500_000, lo=150, hi=150, pad=0, div=0.06,
             max_error=200),
        # the long-pair workload: 100-10,000 bp
        dict(name="wfa_long_20k", op="wfa", n=20_000, lo=100, hi=10_000, pad=0, div=0.10,
             max_error=0),
        # alignments with their CIGARs
        dict(name="wfa_cigar_5k", op="wfa_cigar", n=5_000, lo=100, hi=3000, pad=0, div=0.08,
             max_error=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["sw", "sw", "sw", "sw_host", "nw", "nw", "wfa", "wfa", "wfa_cigar",
                     "sw_call", "wfa_call"])
    top = {"sw": 10_000, "sw_host": 600, "nw": 1_000, "wfa": 10_000, "wfa_cigar": 3_000,
           "sw_call": 2_000, "wfa_call": 4_000}[op]
    hi = _log_int(rng, 60, top)
    lo = hi if rng.random() < 0.3 else max(40, int(hi * rng.uniform(0.1, 1.0)))
    hi = max(lo, hi)
    c = dict(op=op, n=1, lo=lo, hi=hi, pad=0, div=round(rng.uniform(0.02, 0.10), 3))
    mean = (lo + hi) / 2
    if op in ("sw", "sw_host", "sw_call", "nw"):
        c["pad"] = 0 if op == "nw" else rng.randint(0, 25)
        c["scores"] = rng.choice([READ_SCORES, DEFAULT_SCORES])
        kind = rng.random()
        if op == "sw" and kind < 0.3:
            bands = [16, 32, 64, 128]
        elif op == "sw" and kind < 0.4:
            bands = sorted(rng.sample(range(10, 129), 4))
        elif kind < 0.7:
            bands = [rng.choice([16, 32, 64, 128])]
        else:
            bands = [rng.randint(10, 128)]
        c["bands"] = ",".join(map(str, bands))
        cells = mean * (2 * sum(bands) / len(bands) + 1)
        most = {"sw_call": 1, "sw_host": 3e9 / cells, "nw": 2e9 / cells, "sw": 3e9 / cells}[op]
        if op == "sw_host":
            most = min(most, 300_000)
        c["pinned"] = rng.random() < 0.5
    else:
        c["max_error"] = 200 if rng.random() < 0.3 else 0
        steps = (c["div"] * mean * 2.6) ** 2 + 200
        most = {"wfa_call": 1, "wfa": 5e9 / steps, "wfa_cigar": 4e8 / steps}[op]
        most = min(most, 40_000_000 / mean)
    most = max(1, min(500_000, int(most)))
    c["n"] = 1 if op.endswith("_call") else _log_int(rng, min(300, most), most)
    return c


# ---- inputs -----------------------------------------------------------------------

def _ints(text):
    return [int(v) for v in text.split(",")]


def _codes(c, seed):
    """(query codes [n, *], query lengths, target codes [n, *], target lengths), on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    dev = torch.device("cuda")
    n, lo, hi, pad = c["n"], c["lo"], c["hi"], c["pad"]
    u = torch.rand(n, generator=g, device=dev, dtype=torch.float64)
    lens = (lo * torch.exp(u * math.log(hi / lo))).round().long().clamp_(lo, hi)
    div = c["div"] * (0.1 + 0.9 * torch.rand(n, generator=g, device=dev))
    parts = []
    step = max(1, (1 << 26) // hi)
    for i in range(0, n, step):
        ln, d = lens[i:i + step, None], div[i:i + step, None]
        m = ln.shape[0]
        target = torch.randint(0, 4, (m, hi + 2 * pad), generator=g, device=dev, dtype=torch.uint8)
        t = target[:, pad:pad + hi]
        e = torch.rand((m, hi), generator=g, device=dev)
        other = torch.randint(1, 4, (m, hi), generator=g, device=dev, dtype=torch.uint8)
        inside = torch.arange(hi, device=dev)[None] < ln
        dele, ins, sub = e < 0.15 * d, (e >= 0.15 * d) & (e < 0.3 * d), (e >= 0.3 * d) & (e < d)
        count = torch.where(dele, 0, torch.where(ins, 2, 1)) * inside
        end = count.cumsum(1)
        base = torch.where(sub, (t + other) & 3, t)
        q = torch.zeros((m, int(end[:, -1].max()) + 1), dtype=torch.uint8, device=dev)
        trash = q.shape[1] - 1
        q.scatter_(1, torch.where(count > 0, end - count, trash), base)
        q.scatter_(1, torch.where(count == 2, end - 1, trash), other)
        parts.append((q[:, :-1], end[:, -1], target, ln[:, 0] + 2 * pad))
    width = max(p[0].shape[1] for p in parts)
    q = torch.cat([torch.nn.functional.pad(p[0], (0, width - p[0].shape[1])) for p in parts])
    return q, torch.cat([p[1] for p in parts]), torch.cat([p[2] for p in parts]), \
        torch.cat([p[3] for p in parts])


def _batch(codes, lens, pinned=False):
    """SequenceBatch of the given 2-bit codes, sequences one after another."""
    n, width = codes.shape
    nw = (width + 31) // 32
    at = torch.arange(nw * 32, device=codes.device)
    shift = (62 - 2 * (at % 32)).view(nw, 32)
    words_of = (lens + 31) // 32
    words = []
    step = max(1, (1 << 26) // (nw * 32))
    for i in range(0, n, step):
        part = torch.nn.functional.pad(codes[i:i + step], (0, nw * 32 - width)).long()
        part *= at[None] < lens[i:i + step, None]
        w = (part.view(-1, nw, 32) << shift).sum(2)
        words.append(w[torch.arange(nw, device=w.device)[None] < words_of[i:i + step, None]])
    packed = torch.cat(words).cpu().numpy().view(np.uint64)
    offsets = (words_of.cumsum(0) - words_of).cpu().numpy()
    return SequenceBatch.from_arrays(packed, np.zeros_like(packed), offsets, lens.cpu().numpy(),
                                     pinned=pinned)


def _bands(c, seed):
    """The band of every pair, when they differ."""
    b = _ints(c["bands"])
    if len(b) == 1:
        return None
    return np.random.default_rng(seed).choice(np.array(b, np.int32), c["n"]).astype(np.int32)


def _pinned(n, dtype):
    """A page-locked array that lives as long as any view of it."""
    return torch.zeros(n * dtype.itemsize, dtype=torch.uint8, pin_memory=True).numpy().view(dtype)


def prepare(case, seed):
    c = dict(case)
    op = c["op"]
    q, ql, t, tl = _codes(c, seed)
    dev = align.default_device()
    qb = _batch(q, ql, pinned=op == "sw_host")
    tb = _batch(t, tl, pinned=op == "sw_host")
    s = dict(op=op, dev=dev)
    if "scores" in c:
        bands = _ints(c["bands"])
        s["cfg"] = AlignConfig(*_ints(c["scores"]), bands[0])
        s["bands"] = _bands(c, seed)
        s["out"] = None
        if c.get("pinned") and op in ("sw", "sw_host"):
            s["out"] = _pinned(c["n"], SW_RESULT_DTYPE)
            if s["bands"] is not None:
                b = _pinned(c["n"], np.dtype(np.int32))
                b[:] = s["bands"]
                s["bands"] = b
    else:
        me = c["max_error"] or synth.wfa_max_error_cover(qb, tb, 4, 6, 2)
        s["cfg"] = WFAConfig(4, 6, 2, int(me))
    if op == "wfa_cigar":
        # twice the expected number of runs (an edit in the middle of matches starts two)
        s["room"] = c["n"] * int(2.2 * c["div"] * _means(c["lo"], c["hi"])[0] + 16)
    if op.endswith("_call"):
        s["q"], s["t"] = get_view(qb, 0), get_view(tb, 0)
    elif op == "sw_host":
        s["q"], s["t"] = qb, tb
    else:
        s["q"] = dev.upload_batch(qb, with_nmask=False)
        s["t"] = dev.upload_batch(tb, with_nmask=False)
    return s


# ---- one pass ---------------------------------------------------------------------

def _columns(res):
    """score, query_end, ref_end of every pair as the columns of one int32 array."""
    return res.view(np.int32).reshape(-1, 3)


def run(s):
    op, dev = s["op"], s["dev"]
    if op == "sw_call":
        a = align.smith_waterman_banded(s["q"], s["t"], s["cfg"])
        return a.score, a.query_end, a.ref_end
    if op == "wfa_call":
        return align.wfa_affine_cpu(s["q"], s["t"], s["cfg"])
    if op in ("sw", "sw_host"):
        return _columns(dev.sw_banded(s["q"], s["t"], s["cfg"], bands=s["bands"], out=s["out"]))
    if op == "nw":
        return _columns(dev.nw_banded(s["q"], s["t"], s["cfg"], bands=s["bands"]))
    if op == "wfa":
        return dev.wfa_affine(s["q"], s["t"], s["cfg"])
    cost, runs, offsets = dev.wfa_cigar(s["q"], s["t"], s["cfg"], raw=True)
    held = np.zeros(s["room"], np.uint32)  # the program's own array, the same size for any input
    held[:len(runs)] = runs
    return cost, held, offsets


def _means(lo, hi):
    """E[L] and E[L^2] of a log-uniform length."""
    if lo == hi:
        return lo, lo * lo
    span = math.log(hi / lo)
    return (hi - lo) / span, (hi * hi - lo * lo) / (2 * span)


def work(case):
    """Packed words, offsets and lengths read once and results written once; the integer
    operations of the recurrences as the reference writes them (11 per Smith-Waterman cell,
    6 per Needleman-Wunsch cell, 13 per wavefront cell) over the cells that they visit."""
    c = dict(case)
    n = c["n"]
    mean, square = _means(c["lo"], c["hi"])
    read = n * (2 * mean / 4 + 2 * c["pad"] / 4 + 32)
    if "scores" in c:
        b = _ints(c["bands"])
        cells = n * mean * (2 * sum(b) / len(b) + 1)
        return {"bytes": read + 12 * n, "flops": cells * (6 if c["op"] == "nw" else 11)}
    # an edit costs 0.7 * 4 + 0.3 * 8; scores go in steps of 2, a step is as wide as its number
    d2 = c["div"] ** 2 * (1 + 0.1 + 0.01) / 3
    cells = n * d2 * square * 2.6 ** 2
    if c["max_error"]:
        cells = min(cells, n * (c["max_error"] / 2) ** 2)
    runs = n * mean * c["div"] * 1.1 * 4 if c["op"] == "wfa_cigar" else 0
    return {"bytes": read + 4 * n + runs, "flops": 13 * (cells + n)}


# ---- the same in 64-bit integers ----------------------------------------------------

def _banded(c, seed, local):
    """smith_waterman_banded (local) or needleman_wunsch_banded, one row of all pairs at a time."""
    q, ql, t, tl = _codes(c, seed)
    match, mis, go, ge = _ints(c["scores"])
    goe, neg = go + ge, -1_000_000
    per_pair = _bands(c, seed)
    n = c["n"]
    out = torch.zeros((n, 3), dtype=torch.int64, device=q.device)
    groups = [(b, None) for b in _ints(c["bands"])] if per_pair is None else \
        [(b, torch.from_numpy(np.nonzero(per_pair == b)[0]).to(q.device)) for b in _ints(c["bands"])]
    for b, rows in groups:
        every = torch.arange(n, device=q.device) if rows is None else rows
        w = 2 * b + 1
        j = torch.arange(w, device=q.device)
        for part in every.split(max(1, (1 << 26) // w)):
            qq, qn, tt, tn = q[part], ql[part], t[part], tl[part, None]
            right = int(qn.max()) + b + 1
            tt = torch.nn.functional.pad(tt, (b, max(0, right - tt.shape[1])), value=9)
            if local:
                h = torch.zeros((len(part), w), dtype=torch.int64, device=q.device)
            else:
                h = torch.where(j < b, neg, torch.where(j == b, 0, go + (j - b) * ge))
                h = h.expand(len(part), w).clone()
            best = torch.zeros(len(part), dtype=torch.int64, device=q.device)
            end = torch.zeros((len(part), 2), dtype=torch.int64, device=q.device)
            for i in range(int(qn.max())):
                ri = i - b + j
                valid = (ri >= 0)[None] & (ri[None] < tn)
                a = h + torch.where(tt[:, i:i + w] == qq[:, i, None], match, mis)
                up = torch.nn.functional.pad(h[:, 1:], (0, 1), value=0 if local else neg) + goe
                if local:  # E extends along the row: a running maximum of up - ge * j
                    up = torch.where(valid, up - ge * j, neg * 4).cummax(1).values + ge * j
                    a = torch.maximum(a, up).clamp_(min=0)
                    a = torch.where(valid, a, 0)
                else:
                    a = torch.where(valid, torch.maximum(a, up), neg)
                new = (a - goe * j).cummax(1).values + goe * j
                new = torch.where(valid, new, 0 if local else neg)
                live = i < qn
                h = torch.where(live[:, None], new, h)
                if local:
                    key = (new * w + (w - 1 - j)).max(1).values
                    better = live & (key // w > best)
                    best = torch.where(better, key // w, best)
                    at = torch.stack((torch.full_like(key, i), i - b + (w - 1 - key % w)), 1)
                    end = torch.where(better[:, None], at, end)
            if not local:
                fin = tn[:, 0] - qn + b
                best = h.gather(1, fin.clamp(0, w - 1)[:, None])[:, 0]
                best = torch.where((fin >= 0) & (fin < w), best, neg)
                end = torch.stack((qn - 1, tn[:, 0] - 1), 1)
            out[part] = torch.cat((best[:, None], end), 1)
    return out.cpu().numpy()


def _affine_cost(c, seed, max_error):
    """Global gap-affine cost (x4 o6 e2) of every pair, -1 past max_error."""
    q, ql, t, tl = _codes(c, seed)
    n = c["n"]
    cost = torch.zeros(n, dtype=torch.int64, device=q.device)
    for part in torch.arange(n, device=q.device).split(max(1, (1 << 26) // (t.shape[1] + 1))):
        qq, tt = q[part], t[part]
        j = torch.arange(tt.shape[1] + 1, device=q.device)
        h = torch.where(j == 0, 0, 6 + 2 * j).expand(len(part), -1).clone()
        f = torch.full_like(h, 1 << 40)
        for i in range(int(ql[part].max()) + 1):
            if i:
                f = torch.minimum(f, h + 6) + 2
                d = h[:, :-1] + torch.where(tt == qq[:, i - 1, None], 0, 4)
                a = torch.minimum(f, torch.nn.functional.pad(d, (1, 0), value=1 << 40))
                e = (a - 2 * j).cummin(1).values + 2 * j + 6
                h = torch.minimum(a, e)
            done = ql[part] == i
            cost[part[done]] = h[done].gather(1, tl[part[done], None])[:, 0]
    return torch.where(cost > max_error, -1, cost).cpu().numpy()


def exact(case, seed):
    c = dict(case)
    mean, _ = _means(c["lo"], c["hi"])
    if "scores" in c:
        width = 2 * max(_ints(c["bands"])) + 1
        if c["n"] * c["hi"] * width > 2e10 or c["hi"] > 3000:
            return None
        v = _banded(c, seed, c["op"] != "nw")
        return tuple(int(x) for x in v[0]) if c["op"] == "sw_call" else v
    if c["n"] * c["hi"] * c["hi"] > 6e10:
        return None
    me = c["max_error"] or 1 << 60
    v = _affine_cost(c, seed, me)
    if c["op"] == "wfa_call":
        return int(v[0])
    return (v, None, None) if c["op"] == "wfa_cigar" else v
