"""Compute_Trace_PTS's segments against the restatement: distances inside and beyond the fast
kernel's bands, length differences of either sign, one- and two-byte traces, no trace points,
and traces that run past their record."""
import numpy as np
import pytest

from marvel_b200 import dazzdb

pytestmark = pytest.mark.gpu


def block(reads):
    rlen = np.array([r.size for r in reads], np.int32)
    bases = np.concatenate([np.array([4], np.uint8)] + [np.append(r, np.uint8(4)) for r in reads] +
                           [np.full(4, 4, np.uint8)])
    boff = np.zeros(rlen.size + 1, np.int64)
    boff[1:] = np.cumsum(rlen.astype(np.int64) + 1)
    return dazzdb.Block(bases, boff, rlen, 0, 1, np.full(4, .25, np.float32), int(rlen.max()), int(rlen.sum()))


def make(rng, ts):
    """Reads and records: the same read, mutated copies at rising rates, unrelated reads."""
    a = rng.integers(0, 4, 40 * ts + 37, dtype=np.uint8)
    reads, recs, traces = [a], [], []
    for rate in (0.0, 0.02, 0.15, 0.3, 0.6, 1.0):
        ab = int(rng.integers(0, 2 * ts))
        ae = a.size - int(rng.integers(0, 2 * ts))
        cuts = [ab] + list(range((ab // ts + 1) * ts, ae, ts)) + [ae]
        pieces, points = [], []
        for i, (s, e) in enumerate(zip(cuts, cuts[1:])):
            p = a[s:e][rng.random(e - s) >= rate / 3].copy()
            m = rng.random(p.size) < rate
            p[m] = rng.integers(0, 4, int(m.sum()), dtype=np.uint8)
            if i % 7 == 3:  # B far shorter or longer than A in this interval, or empty
                p = rng.integers(0, 4, int(rng.choice([0, 1, e - s + 55, min(2 * ts, 250)])), dtype=np.uint8)
            p = p[:250 if ts <= 125 else 4 * ts]
            pieces.append(p)
            points.append(p.size)
        b = np.concatenate([rng.integers(0, 4, 11, dtype=np.uint8)] + pieces + [rng.integers(0, 4, 9, dtype=np.uint8)])
        reads.append(b)
        recs.append((ab, 11, ae, 11 + sum(points), len(reads) - 1))
        traces.append(np.array([v for p in points for v in (0, p)]))
    recs.append(recs[2][:4] + (3,))  # no trace points: one long segment
    traces.append(np.zeros(0, int))
    return reads, recs, traces


@pytest.mark.parametrize("ts", [20, 100, 125, 126, 300])
def test_segment_distances_match_oracle(ts):
    import marvel_b200 as mb
    import oracle
    rng = np.random.default_rng(ts)
    ctx = mb.Context()
    for _ in range(3):
        reads, recs, traces = make(rng, ts)
        blk = block(reads)
        ctx.set_filter_params()
        ctx.new_align_spec(0.70, ts, blk.freq)
        ctx.load_block(0, blk)
        dt = np.uint8 if ts <= 125 else np.uint16
        raw = [t.astype(dt).view(np.uint8) for t in traces]
        r = np.zeros(len(recs), mb.OVL_DTYPE)
        for i, (ab, bb, ae, be, br) in enumerate(recs):
            r[i]["abpos"], r[i]["bbpos"], r[i]["aepos"], r[i]["bepos"], r[i]["bread"] = ab, bb, ae, be, br
            r[i]["tlen"] = traces[i].size
        r["toff"] = np.cumsum([0] + [t.size for t in raw[:-1]])
        got = ctx.compute_trace_pts(r, np.concatenate(raw), 0, 0, 0)
        want = [oracle.trace_pts_diffs(reads[0], reads[x["bread"]], x, t, ts) for x, t in zip(r, traces)]
        assert got.tolist() == want
    # a trace whose B lengths run past the record's end is refused, as before
    bad = np.concatenate(raw)
    r2 = r[:1].copy()
    r2["bepos"] = r2["bbpos"] + 1
    with pytest.raises(mb.GpuError):
        ctx.compute_trace_pts(r2, bad, 0, 0, 0)
    ctx.close()
