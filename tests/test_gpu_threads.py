"""Several threads on one context: seed batches, trace checks, block loads and comparisons at the same time
give what they give one after the other."""
import os
import threading

import numpy as np
import pytest

from golden_cases import load
from marvel_b200 import dazzdb

pytestmark = pytest.mark.gpu


def run_all(jobs):
    errors = []

    def guard(f):
        try:
            f()
        except BaseException as e:  # noqa: BLE001 -- reported by the test's thread
            errors.append(e)

    ts = [threading.Thread(target=guard, args=(j,)) for j in jobs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    if errors:
        raise errors[0]


def test_calls_of_several_threads_take_turns():
    import marvel_b200 as mb
    import oracle
    d, _ = load("self_default")
    A = dazzdb.open_block(os.path.join(d, "G.1"))
    ctx = mb.Context()
    recs, tr = mb.daligner_block(ctx, A)
    recs, tr = recs.copy(), tr.copy()
    hits, _ = oracle.match_hits(A, A, oracle.make_params(A.freq), True)
    rng = np.random.default_rng(1)
    cases = []
    for n, stride in ((3000, 1200), (40, None), (900, 3000), (1, None)):  # traces in pieces through the staging, or whole
        rows = hits[rng.choice(len(hits), size=n)]
        diag, apos, ar, br = rows[:, 0], rows[:, 1], rows[:, 2], rows[:, 3]
        cases.append((A.bases, A.boff[ar] + 1, A.rlen[ar], A.bases, A.boff[br] + 1, A.rlen[br], diag, 2 * apos - diag, 0,
                      stride))
    wanted = [ctx.local_alignment_batch(*c) for c in cases]
    part = [np.sort(rng.choice(recs.size, size=k, replace=False)) for k in (recs.size, recs.size // 3, 5)]
    diffs = [ctx.compute_trace_pts(recs[p], tr) for p in part]

    def batch(i):
        def job():
            for _ in range(6):
                for g, w in zip(ctx.local_alignment_batch(*cases[i]), wanted[i]):
                    assert np.array_equal(g, w)
        return job

    def check(i):
        def job():
            for _ in range(6):
                assert np.array_equal(ctx.compute_trace_pts(recs[part[i]], tr), diffs[i])
        return job

    def compare():
        for _ in range(4):
            ctx.reset_overlap_buffer()
            mb.run_loaded(ctx, True)
            r, t = ctx.overlaps()
            assert r.tobytes() == recs.tobytes() and t.tobytes() == tr.tobytes()

    big = np.full(6 << 20, 4, np.uint8)  # a second block through the staging: slot 1, which nothing else uses
    big[1:-1] = rng.integers(0, 4, big.size - 2, dtype=np.uint8)
    blk = dazzdb.Block(big, np.array([0, big.size - 1], np.int64), np.array([big.size - 2], np.int32), 0, 1,
                       np.full(4, .25, np.float32), big.size - 2, big.size - 2)

    def loads():
        want = None
        for _ in range(6):
            ctx.load_block(1, blk)
            got = ctx.dust(1, blk.freq)
            want = want or got
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])

    run_all([batch(i) for i in range(4)])
    run_all([check(i) for i in range(3)])
    run_all([batch(0), batch(2), check(0), check(1), compare, loads])
    ctx.close()
