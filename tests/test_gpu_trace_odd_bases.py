"""Compute_Trace_PTS of blocks that hold bytes beyond 3 inside their reads: such a byte equals itself only."""
import numpy as np
import pytest

from test_gpu_trace_segments import block, make

pytestmark = pytest.mark.gpu


def records(recs, traces, ts):
    import marvel_b200 as mb
    r = np.zeros(len(recs), mb.OVL_DTYPE)
    for i, (ab, bb, ae, be, br) in enumerate(recs):
        r[i]["abpos"], r[i]["bbpos"], r[i]["aepos"], r[i]["bepos"], r[i]["bread"] = ab, bb, ae, be, br
        r[i]["tlen"] = traces[i].size
    raw = [t.astype(np.uint8 if ts <= 125 else np.uint16).view(np.uint8) for t in traces]
    r["toff"] = np.cumsum([0] + [t.size for t in raw[:-1]])
    return r, np.concatenate(raw)


@pytest.mark.parametrize("ts", [20, 126])
def test_bytes_beyond_3_match_oracle(ts):
    import marvel_b200 as mb
    import oracle
    rng = np.random.default_rng(ts)
    ctx = mb.Context()
    ctx.set_filter_params()
    ctx.new_align_spec(0.70, ts, np.full(4, .25, np.float32))
    plain, recs, traces = make(rng, ts)
    r, tr = records(recs, traces, ts)

    def check(reads):
        want = [oracle.trace_pts_diffs(reads[0], reads[x["bread"]], x, t, ts) for x, t in zip(r, traces)]
        assert ctx.compute_trace_pts(r, tr, 0, 0, 0).tolist() == want

    for where in ("a", "b", "both", "one"):
        reads = [x.copy() for x in plain]
        for i, x in enumerate(reads):
            if where == "both" or (where == "a") == (i == 0) or (where == "one" and i == 3):
                n = 1 if where == "one" else x.size // 9
                x[rng.integers(0, x.size, n)] = rng.choice([4, 5, 7, 8, 255], n)
        ctx.load_block(0, block(reads))
        check(reads)
        ctx.load_block(0, block(plain))  # the slot's next block is looked at anew
        check(plain)
    ctx.close()


def test_complemented_block_with_bytes_beyond_3():
    """A complemented slot of its own origin, plain A and B: its records compare bytes too."""
    import marvel_b200 as mb
    import oracle
    rng = np.random.default_rng(9)
    ts = 100
    ctx = mb.Context()
    ctx.set_filter_params()
    ctx.new_align_spec(0.70, ts, np.full(4, .25, np.float32))
    reads, recs, traces = make(rng, ts)
    r, tr = records(recs, traces, ts)
    r["flags"] = 1
    odd = [x.copy() for x in reads]
    for x in odd:
        x[rng.integers(0, x.size, 50)] += 4
    ctx.load_block(0, block(reads))
    for comp in (odd, reads):
        ctx.load_block(2, block(comp))
        want = [oracle.trace_pts_diffs(reads[0], comp[x["bread"]], x, t, ts) for x, t in zip(r, traces)]
        assert ctx.compute_trace_pts(r, tr, 0, 0, 2).tolist() == want
    # the complement of an odd block is odd, made before and after the block was looked at
    for look in (False, True):
        ctx.load_block(0, block(odd))
        if look:
            ctx.compute_trace_pts(r[:0], tr, 0, 0, 2)
            ctx.load_block(2, block(reads))
            ctx.compute_trace_pts(r[:1], tr, 0, 0, 2)
        ctx.complement_block(0, 2)
        cb = [np.uint8(3) - x[::-1] for x in odd]
        want = [oracle.trace_pts_diffs(odd[0], cb[x["bread"]], x, t, ts) for x, t in zip(r, traces)]
        assert ctx.compute_trace_pts(r, tr, 0, 0, 2).tolist() == want
    ctx.close()
