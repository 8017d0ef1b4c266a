"""Seeds aligned ahead: that the pair kernel takes them, and every way in which one is left to it -- groups
and seeds beyond the capacities, no room for traces, pebbles that run out -- with the output of a run
that aligns none ahead."""
import numpy as np
import pytest

from test_gpu_ahead import block, reads

pytestmark = pytest.mark.gpu

CASES = [(60, 3000, 0.12, False), (45, 2500, 0.12, True), (64, 20000, 0.06, False)]


def output(ctx, blk):
    import marvel_b200 as mb
    recs, tr = mb.daligner_block(ctx, blk)
    st = ctx.stats()
    rows = sorted(tuple(int(r[f]) for f in ("aread", "bread", "flags", "abpos", "aepos", "bbpos", "bepos", "diffs")) +
                  (tr[int(r["toff"]):int(r["toff"]) + int(r["tlen"])].tobytes(),) for r in recs)
    return rows, st["seeds"], st["cells"], st["reruns"]


@pytest.mark.parametrize("period,span,rate,shared", CASES)
def test_seeds_are_taken_and_every_refusal_aligns_them_later(period, span, rate, shared):
    import marvel_b200 as mb
    blk = block(reads(np.random.default_rng(period + span), period, span, 8 if span < 10000 else 6, rate, shared))
    ctx = mb.Context()
    ctx.set_align_schedule([1], [0, 0])  # classes: no seeds are aligned ahead
    want = output(ctx, blk)
    assert ctx.test_ahead() == (0, 0, 0, 0)
    ctx.set_align_schedule()

    def run(**caps):
        ctx.test_ahead(**caps)
        got = output(ctx, blk)
        assert got[:3] == want[:3]
        return ctx.test_ahead()

    listed, aligned, taken, _ = run()
    assert listed >= aligned >= taken > 0
    some = run(groups=1)  # of each orientation the first group
    assert 0 < some[0] < listed and some[2] < taken
    some = run(seeds=max(1, listed // 4))  # the lists of the last groups end without room
    assert some[1] <= 2 * max(1, listed // 4) and some[1] < aligned and some[2] < taken
    some = run(seeds=1)  # room for no list
    assert some[0] > 2 and some[1:3] == (0, 0)
    some = run(traces=1)  # room for no trace
    assert some[0] == listed and some[1:3] == (0, 0)
    some = run(traces=3000)  # for some
    assert 0 < some[1] < aligned
    assert run()[:3] == (listed, aligned, taken)  # the defaults again
    # pebbles that run out: ahead, where the seed is left to the pair kernel, and there, which is run again
    small = mb.Context()
    small.set_capacities(pebbles=64)
    got = output(small, blk)
    assert got[:3] == want[:3] and sum(got[3]) > 0
    again = small.test_ahead()
    assert again[1] < again[0] and again[2] > 0
    small.close()
    ctx.close()


@pytest.mark.parametrize("rate", [0.0, 0.002, 0.01, 0.04])
def test_overlaps_of_accurate_reads_are_not_looked_at(rate):
    """Their groups hold as many hits as a repeat's, on one band or a few."""
    import marvel_b200 as mb
    from test_gpu_accurate_reads import genome_reads
    ctx = mb.Context()
    mb.daligner_block(ctx, block(genome_reads(np.random.default_rng(3), 60000, 9000, 40, rate, 0)))
    st = ctx.stats()
    assert st["hits"][0] > 65536 and st["groups"][0] > 100
    assert ctx.test_ahead() == (0, 0, 0, 0)
    ctx.close()
