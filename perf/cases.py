"""The workloads by which this package's speed is measured.

Every case is one pass through the public Python interface (marvel_b200), on host data as a
program that compares DB blocks has it: the blocks' decoded bases in host memory, one device
context that the program keeps for all its block comparisons, results back in the program's own
host arrays (whose size is the case's, so that every seed gives outputs of one shape; what lies
past the results stays as it was).

  block     daligner, one block against itself: the unit of every HPCdaligner plan
  pair      daligner, block 1 against block 2, both masked with DBdust's track (-mdust)
  block2    daligner2 (modimizer seeds), one block against itself
  dust      DBdust's track of one block
  check     Compute_Trace_PTS of every record of a block's overlaps (what LAcheck -a does)
  align     Local_Alignment from given seeds (the reference-named entry points' batch)
  score     the triage model over a block's pair groups, as calibration does
  grad      one gradient of the triage model over a mini-batch, as training does

The reads are drawn from a seeded random genome: log-normal lengths, both strands,
insertions, deletions and substitutions at PacBio-like or nanopore-like rates.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import marvel_b200 as mb
from marvel_b200 import dazzdb

PACBIO = dict(p_ins=0.09, p_del=0.045, p_sub=0.015, hp=1.0)
# nanopore-like: fewer errors, deletions three times as likely inside homopolymers
NANOPORE = dict(p_ins=0.03, p_del=0.05, p_sub=0.02, hp=3.0)
# typical sizes of a pair group's features: hits, read lengths, spans, diagonals, densities, fractions
FEATURE_SIZES = np.array([20, 9000, 9000, 4000, 150, 300, 60, 4500, 0.01, 0.8, 0.5, 0.02], np.float32)
DALIGNER = dict(k=14, w=6, h=35, e=0.70, l=1000, s=100)


def _block(name, kind, genome, cov, mean, sd, most, errors, **more):
    c = dict(name=name, kind=kind, genome=genome, cov=cov, mean=mean, sd=sd, most=most, copies=0, spread=0.0,
             tandem=0.0, at=0.5, biased=False)
    c.update(DALIGNER)
    c.update(errors)
    c.update(more)
    return c


def listed():
    return [
        # a handful of reads: what a test, a small amplicon set or the last block of a DB costs
        _block("block_small", "block", 60_000, 12, 4000, 2000, 12000, PACBIO),
        # 1 Mbp at 20x: a BAC pool or small plasmid set, one block
        _block("block_1mbp", "block", 1_000_000, 20, 8000, 4000, 30000, PACBIO),
        # a bacterial genome with its repeat families in one block: the headline workload
        _block("block_bacterial", "block", 4_600_000, 25, 10000, 5000, 60000, PACBIO, copies=40),
        # long uneven reads, lower error rate
        _block("block_long_reads", "block", 2_500_000, 25, 20000, 15000, 150000, NANOPORE),
        # one off-diagonal block pair of a large repeat-rich genome at low depth per block
        _block("pair_repeats_dust", "pair", 25_000_000, 2, 15000, 7500, 100000, PACBIO, spread=0.35, tandem=0.02),
        # other options together: weighted tuples (-b) on an AT-rich genome, 16-bit traces, k = 16
        _block("block_biased_k16_s200", "block", 700_001, 15, 6000, 3000, 20000, PACBIO, at=0.64, biased=True,
               k=16, w=5, s=200, e=0.75),
        _block("block2_2mbp", "block2", 2_000_000, 20, 10000, 5000, 60000, PACBIO, copies=10),
        # the track that -mdust needs, for a whole block
        _block("dust_100mbp", "dust", 5_000_000, 20, 10000, 5000, 60000, PACBIO, tandem=0.02),
        _block("check_traces", "check", 1_000_000, 15, 8000, 4000, 30000, PACBIO, records=45_000),
        _block("align_seeds", "align", 600_000, 12, 8000, 4000, 30000, PACBIO, seeds=4000),
        dict(name="triage_score_1m", kind="score", rows=1_000_000),
        dict(name="triage_grad_8192", kind="grad", rows=8192),
    ]


def draw(rng):
    kind = rng.choice(["block", "block", "block", "pair", "block2", "dust", "check", "align", "score", "grad"])
    if kind == "score":
        return dict(kind=kind, rows=int(math.exp(rng.uniform(math.log(1000), math.log(1_000_000)))))
    if kind == "grad":
        return dict(kind=kind, rows=int(math.exp(rng.uniform(math.log(500), math.log(60_000)))))
    cov = rng.randint(8, 25)
    lo, hi = {"block": (0.5e6, 60e6), "pair": (1e6, 40e6), "block2": (0.5e6, 40e6), "dust": (1e6, 100e6),
              "check": (0.5e6, 20e6), "align": (0.5e6, 8e6)}[kind]
    bases = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    if kind == "pair":
        cov = rng.randint(2, 8)
    mean = rng.randint(3000, 18000)
    c = _block("", kind, max(50_001, int(bases / cov)), cov, mean, int(mean * rng.uniform(0.3, 0.8)),
               rng.choice([20000, 60000, 150000]), rng.choice([PACBIO, PACBIO, NANOPORE]),
               copies=rng.choice([0, 0, 5, 20]) if kind in ("block", "block2") else 0,
               tandem=rng.choice([0.0, 0.02]) if kind in ("pair", "dust") else 0.0,
               spread=rng.choice([0.1, 0.35]) if kind == "pair" else 0.0)
    del c["name"]
    if kind == "block":
        c["k"], c["w"] = rng.choice([(14, 6), (14, 6), (13, 6), (16, 5)])
        c["s"] = rng.choice([50, 100, 100, 126, 200])
        c["e"] = rng.choice([0.70, 0.70, 0.75])
        c["at"] = rng.choice([0.5, 0.6])
        c["biased"] = rng.random() < 0.2
    if kind == "check":
        c["records"] = int(2 * c["genome"] * cov / mean * cov * 0.8)
    if kind == "align":
        c["seeds"] = int(math.exp(rng.uniform(math.log(100), math.log(8000))))
    return c


# ---- inputs --------------------------------------------------------------------------------


def _genome(c, rng):
    n = c["genome"]
    gc = rng.random(n, np.float32) >= c["at"]
    one = rng.random(n, np.float32) < 0.5
    g = np.where(gc, np.where(one, 1, 2), np.where(one, 0, 3)).astype(np.uint8)  # A, C, G, T = 0..3

    def put(unit, div):
        u = unit.copy()
        at = np.nonzero(rng.random(u.size) < div)[0]
        u[at] = (u[at] + rng.integers(1, 4, at.size, dtype=np.uint8)) & 3
        p = int(rng.integers(0, max(n - u.size, 1)))
        g[p:p + u.size] = u[:n - p]

    if c["copies"]:  # one insertion-sequence-like family, nearly identical copies
        unit = rng.integers(0, 4, 5000, dtype=np.uint8)
        for _ in range(c["copies"]):
            put(unit, 0.015)
    if c["spread"] > 0:  # interspersed families of 1-10 kbp at 5-15 % divergence
        families = [rng.integers(0, 4, int(rng.integers(1000, 10001)), dtype=np.uint8)
                    for _ in range(max(1, int(c["spread"] * n) // 200000))]
        left = c["spread"] * n
        while left > 0:
            u = families[int(rng.integers(0, len(families)))]
            put(u, float(rng.uniform(0.05, 0.15)))
            left -= u.size
    if c["tandem"] > 0:  # tandem arrays of period 2-200
        left = c["tandem"] * n
        while left > 0:
            unit = rng.integers(0, 4, int(rng.integers(2, 201)), dtype=np.uint8)
            span = int(rng.integers(500, 5000))
            put(np.tile(unit, span // unit.size + 1)[:span], 0.02)
            left -= span
    return g


def _reads(c, g, rng, gen):
    """One block of reads of genome g (on the GPU), in the layout of a decoded DB block."""
    dev = "cuda"
    n = g.numel()
    mean, sd = float(c["mean"]), float(c["sd"])
    s2 = math.log(1 + (sd * sd) / (mean * mean))
    target = c["cov"] * n
    lens = rng.lognormal(math.log(mean) - s2 / 2, math.sqrt(s2), int(1.5 * target / mean) + 64)
    lens = np.clip(np.round(lens), 1000, min(c["most"], n)).astype(np.int64)
    lens = lens[:int(np.searchsorted(np.cumsum(lens), target)) + 1]
    start = (rng.random(lens.size) * (n - lens + 1)).astype(np.int64)
    strand = rng.random(lens.size) < 0.5
    pdel = None
    if c["hp"] != 1.0:
        change = torch.ones(n, dtype=torch.bool, device=dev)
        change[1:] = g[1:] != g[:-1]
        run = torch.cumsum(change, 0) - 1
        pdel = torch.where(torch.bincount(run)[run] >= 4, min(c["p_del"] * c["hp"], 0.5), c["p_del"])
    parts, rlens = [], []
    cuts = [0]
    while cuts[-1] < lens.size:  # pieces of at most about 32 M bases
        cuts.append(max(cuts[-1] + 1, int(np.searchsorted(np.cumsum(lens), np.cumsum(lens)[cuts[-1]] + 32_000_000))))
    for a, b in zip(cuts, cuts[1:]):
        b = min(b, lens.size)
        L = torch.from_numpy(lens[a:b]).to(dev)
        S = torch.from_numpy(start[a:b]).to(dev)
        rev = torch.from_numpy(strand[a:b]).to(dev)
        off = torch.cumsum(L, 0) - L
        total = int(L.sum())
        read = torch.repeat_interleave(torch.arange(b - a, device=dev), L)
        pos = torch.arange(total, device=dev) - off[read]
        r = rev[read]
        idx = S[read] + torch.where(r, L[read] - 1 - pos, pos)
        base = g[idx]
        base = torch.where(r, 3 - base, base)
        u = torch.rand(total, device=dev, generator=gen)
        pd = pdel[idx] if pdel is not None else c["p_del"]
        keep = u >= pd
        sub = keep & (u < pd + c["p_sub"])
        other = torch.randint(1, 4, (total,), device=dev, generator=gen, dtype=torch.uint8)
        base = torch.where(sub, (base + other) & 3, base)
        ins = torch.rand(total, device=dev, generator=gen).clamp_min(1e-30).log_().div_(math.log(c["p_ins"]))
        count = ins.floor_().to(torch.int64) + keep
        ends = torch.cumsum(count, 0)
        out = torch.randint(0, 4, (int(ends[-1]),), device=dev, generator=gen, dtype=torch.uint8)
        out[ends[keep] - 1] = base[keep]
        tail = ends[off + L - 1]
        rl = torch.diff(tail, prepend=tail.new_zeros(1))
        buf = torch.full((int(tail[-1]) + b - a,), 4, dtype=torch.uint8, device=dev)
        who = torch.repeat_interleave(torch.arange(b - a, device=dev), rl)
        buf[torch.arange(out.numel(), device=dev) + who] = out
        parts.append(buf)
        rlens.append(rl)
    rlen = torch.cat(rlens).to(torch.int32).cpu().numpy()
    body = torch.cat(parts)
    bases = np.full(body.numel() + 1 + 4, 4, np.uint8)
    bases[1:1 + body.numel()] = body.cpu().numpy()
    boff = np.zeros(rlen.size + 1, np.int64)
    boff[1:] = np.cumsum(rlen.astype(np.int64) + 1)
    freq = torch.bincount(body.to(torch.int64), minlength=5)[:4].to(torch.float64)
    freq = (freq / freq.sum()).to(torch.float32).cpu().numpy()
    return dazzdb.Block(bases, boff, rlen, 0, 1, freq, int(rlen.max()), int(rlen.sum()))


_CONTEXT = None


def _context():
    """The one device context that a program keeps for all its block comparisons."""
    global _CONTEXT
    if _CONTEXT is None:
        _CONTEXT = mb.Context()
    return _CONTEXT


def _mask(ctx, blk):
    ctx.set_filter_params()
    ctx.load_block(0, blk)
    anno, data = ctx.dust(0, blk.freq)
    iv = data.reshape(-1, 2).tolist()
    at = (anno // 8).tolist()
    blk.mask = [[tuple(p) for p in iv[a:b]] for a, b in zip(at, at[1:])]


def _zeros(nbytes, pinned):
    return torch.zeros(nbytes, dtype=torch.uint8, pin_memory=pinned).numpy()


def _rows(c):
    """Room for the records of a block: two of each pair of overlapping reads, and of each pair of
    repeat copies that reads hold."""
    reads = c["genome"] * c["cov"] / c["mean"]
    spread = c["genome"] * c["spread"] * c["cov"] / 5000
    pairs = 2.6 * reads * c["cov"] + 2.6 * (c["copies"] * c["cov"]) ** 2 + spread * 100
    return int(pairs * 1.2) + 20_000


def _options(c):
    return {x: c[x] for x in ("k", "w", "h", "e", "l", "s")}


def _model(rng, feat):
    p = np.zeros(mb.TRI_NPARAM, np.float32)
    p[:12], p[12:24] = feat.mean(0), feat.std(0)
    at = 24
    for rows, cols in ((64, 12), (64, 64), (1, 64)):
        p[at:at + rows * cols] = rng.uniform(-1, 1, rows * cols) * math.sqrt((3.0 if rows == 1 else 6.0) / cols)
        at += rows * cols + rows
    return p


def prepare(case, seed):
    c = case
    rng = np.random.Generator(np.random.PCG64(seed))
    if c["kind"] in ("score", "grad"):
        # the features of pair groups: counts, lengths, spans and fractions of very different sizes
        n = c["rows"]
        size = FEATURE_SIZES
        feat = (rng.standard_gamma(2.0, (n, mb.TRI_NF)).astype(np.float32) * size).astype(np.float32)
        label = (feat[:, 0] + 10 * rng.standard_normal(n) > 40).astype(np.float32)
        return dict(case=c, ctx=_context(), params=_model(rng, feat), feat=feat, label=label)
    gen = torch.Generator("cuda").manual_seed(seed)
    g = torch.from_numpy(_genome(c, rng)).to("cuda")
    A = _reads(c, g, rng, gen)
    B = _reads(c, g, rng, gen) if c["kind"] == "pair" else None
    ctx = _context()
    ctx.set_variant(1)
    ctx.set_biased(False)
    st = dict(case=c, ctx=ctx, A=A, B=B)
    if c["kind"] == "pair":
        _mask(ctx, A)
        _mask(ctx, B)
    elif c["kind"] in ("check", "align"):
        recs, trace = mb.daligner_block(ctx, A, **_options(c))
        n = c["records"] if c["kind"] == "check" else 0
        if n:  # a file's worth of records, taken over and over where the block has fewer
            at = np.sort(np.arange(n) % recs.size)
            st["recs"], st["trace"] = recs[at], trace
        if c["kind"] == "align":
            # seeds at the beginnings of forward overlaps, as a first k-mer hit gives them
            fwd = recs[recs["flags"] == 0]
            fwd = fwd[rng.integers(0, fwd.size, c["seeds"])]
            diag = fwd["abpos"] - fwd["bbpos"]
            st["out"] = np.zeros(c["seeds"] * (8 * c["most"] // c["s"] + 64), np.uint16)
            st["seeds"] = (A.boff[fwd["aread"]] + 1, A.rlen[fwd["aread"]], A.boff[fwd["bread"]] + 1,
                           A.rlen[fwd["bread"]], diag, fwd["abpos"] + fwd["bbpos"])
    if c["kind"] in ("block", "pair", "block2"):
        # a program that streams large blocks keeps them, and its result buffers, in pinned memory
        pinned = c["genome"] * c["cov"] > 40_000_000
        if pinned:
            pin = _zeros(A.bases.size, True)
            pin[:] = A.bases
            A.bases = pin
        rows = _rows(c)
        st["out"] = (_zeros(rows * mb.OVL_DTYPE.itemsize, pinned).view(mb.OVL_DTYPE),
                     _zeros(int(rows * (c["mean"] / c["s"] + 40) * (2 if c["s"] > 125 else 1)), pinned))
    elif c["kind"] == "dust":
        n = c["genome"] * c["cov"]
        st["out"] = (np.zeros(n // 1000 + 1000, np.int64), np.zeros(n // 50 + 100_000, np.int32))
    torch.cuda.empty_cache()
    return st


# ---- one pass ------------------------------------------------------------------------------


def run(state):
    c, ctx = state["case"], state["ctx"]
    kind = c["kind"]
    if kind == "score":
        return ctx.mlp_forward(state["params"], state["feat"])
    if kind == "grad":
        return ctx.mlp_grad(state["params"], state["feat"], state["label"], 2.0)
    A, B = state["A"], state.get("B")
    if kind in ("block", "pair", "block2"):
        # the steps of one daligner call (daligner_block / daligner2_block), results in the program's arrays
        ctx.set_variant(2 if kind == "block2" else 1)
        ctx.set_biased(c["biased"])
        ctx.set_filter_params(c["k"], c["w"], 0, c["h"])
        ctx.new_align_spec(c["e"], c["s"], A.freq)
        ctx.set_globals(2 * c["l"], False, 32 * 0x40000000)
        ctx.reset_overlap_buffer()
        ctx.load_block(0, A)
        if B is not None:
            ctx.load_block(1, B)
        (mb.run_loaded2 if kind == "block2" else mb.run_loaded)(ctx, B is None)
        ctx.overlaps(out=state["out"])
        recs, trace = state["out"]
        return recs.view(np.int32).reshape(-1, mb.OVL_DTYPE.itemsize // 4), trace
    ctx.set_variant(1)
    ctx.set_filter_params(c["k"], c["w"], 0, c["h"])
    if kind == "dust":
        ctx.load_block(0, A)
        anno, data = ctx.dust(0, A.freq)
        state["out"][0][:anno.size] = anno
        state["out"][1][:data.size] = data
        return state["out"]
    ctx.new_align_spec(c["e"], c["s"], A.freq)
    if kind == "check":
        ctx.load_block(0, A)
        ctx.complement_block(0, 2)
        return ctx.compute_trace_pts(state["recs"], state["trace"], 0, 0, 2)
    aoff, alen, boff, blen, diag, anti = state["seeds"]
    stride = 2 * (4 * (int(1.2 * c["most"]) // c["s"] + 2) + 16)
    out, trace, cells = ctx.local_alignment_batch(A.bases, aoff, alen, A.bases, boff, blen, diag, anti, 0, stride)
    # the traces back to back, A's and then B's of each seed, as a program keeps them
    tlen = out[:, [5, 11]].ravel()
    first = (np.arange(len(diag))[:, None] * stride + np.array([0, stride // 2])).ravel()
    at = np.arange(tlen.sum()) + np.repeat(first - (np.cumsum(tlen) - tlen), tlen)
    state["out"][:at.size] = trace.ravel()[at]
    return out, state["out"], cells


# ---- what one pass cannot do without -------------------------------------------------------


def work(case):
    c = case
    if c["kind"] in ("score", "grad"):
        macs = 12 * 64 + 64 * 64 + 64
        return dict(bytes=c["rows"] * (mb.TRI_NF + 1) * 4, flops=c["rows"] * macs * (2 if c["kind"] == "score" else 6))
    bases = c["genome"] * c["cov"]
    reads = bases / c["mean"]
    if c["kind"] == "dust":
        return dict(bytes=bases, flops=20 * bases)
    # reads that overlap pairwise (each pair once), half a read long; copies of a repeat meet too
    pairs = reads * c["cov"] + (c["copies"] * c["cov"]) ** 2 / 2
    if c["kind"] == "align":
        pairs = c["seeds"]
    trace = pairs * c["mean"] / 2 / c["s"] * 2
    err = c["p_ins"] + c["p_del"] + c["p_sub"]
    # an alignment's waves: one per difference, about ten diagonals wide, 16 integer operations a cell
    cells = pairs * c["mean"] / 2 * 2 * err * 10
    if c["kind"] == "check":
        cells /= 2
    blocks = 2 if c["kind"] == "pair" else 1
    return dict(bytes=blocks * bases + 2 * pairs * 48 + 2 * trace, flops=16 * cells)


# ---- the numbers that outputs in floating point should have --------------------------------


def exact(case, seed):
    c = case
    if c["kind"] not in ("score", "grad"):
        return None  # whole numbers and bytes
    rng = np.random.Generator(np.random.PCG64(seed))
    n = c["rows"]
    size = FEATURE_SIZES
    feat = (rng.standard_gamma(2.0, (n, 12)).astype(np.float32) * size).astype(np.float32)
    label = (feat[:, 0] + 10 * rng.standard_normal(n) > 40).astype(np.float64)
    p = _model(rng, feat).astype(np.float64)
    scale = p[12:24]
    w1, b1, w2 = p[24:792].reshape(64, 12), p[792:856], p[856:4952].reshape(64, 64)
    b2, w3, b3 = p[4952:5016], p[5016:5080], p[5080]
    x = (feat.astype(np.float64) - p[:12]) / scale
    h1 = np.maximum(x @ w1.T + b1, 0)
    h2 = np.maximum(h1 @ w2.T + b2, 0)
    z = h2 @ w3 + b3
    q = 1 / (1 + np.exp(-z))
    if c["kind"] == "score":
        return q
    w = np.where(label > 0.5, 2.0, 1.0)
    loss = float(np.sum(w * (np.maximum(z, 0) - z * label + np.log1p(np.exp(-np.abs(z))))) / n)
    dz = w * (q - label) / n
    d2 = np.outer(dz, w3) * (h2 > 0)
    d1 = (d2 @ w2) * (h1 > 0)
    grad = np.concatenate([np.zeros(24), (d1.T @ x).ravel(), d1.sum(0), (d2.T @ h1).ravel(), d2.sum(0), h2.T @ dz,
                           [dz.sum()]])
    return grad, loss
