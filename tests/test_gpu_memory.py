"""Device memory of a context: what its calls keep, and that all of it returns when it is destroyed."""
import numpy as np
import pytest

from marvel_b200 import dazzdb

pytestmark = pytest.mark.gpu


def random_block(rng, nreads, length):
    """reads of one genome at about 8x"""
    g = rng.integers(0, 4, nreads * length // 8, dtype=np.uint8)
    reads = [g[a:a + length].copy() for a in rng.integers(0, g.size - length, nreads)]
    for r in reads:
        m = rng.random(r.size) < 0.1
        r[m] = rng.integers(0, 4, int(m.sum()), dtype=np.uint8)
    rlen = np.full(nreads, length, np.int32)
    four = np.array([4], np.uint8)
    bases = np.concatenate([four] + [np.append(r, four) for r in reads])
    boff = np.arange(nreads + 1, dtype=np.int64) * (length + 1)
    return dazzdb.Block(bases, boff, rlen, 0, 1, np.full(4, .25, np.float32), length, int(rlen.sum()))


def free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_destroy_frees_everything():
    import marvel_b200 as mb
    blk = random_block(np.random.default_rng(0), 2000, 8000)

    def cycle():
        ctx = mb.Context()
        mb.daligner_block(ctx, blk)
        ctx.set_biased()
        mb.daligner_block(ctx, blk)
        ctx.set_biased(False)
        mb.daligner2_block(ctx, blk, blk)
        ctx.dust(0, blk.freq)
        ctx.close()

    cycle()
    before = free()
    for _ in range(3):
        cycle()
    assert before - free() < 4 << 20


def one_read(n):
    bases = np.full(n + 2, 4, np.uint8)
    bases[1:-1] = np.random.default_rng(n).integers(0, 4, n, dtype=np.uint8)
    return dazzdb.Block(bases, np.array([0, n + 1], np.int64), np.array([n], np.int32), 0, 1, np.full(4, .25, np.float32),
                        n, n)


def big_check(ctx, nrec, blk, ts=2):
    """nrec records of the read against itself, all with the same trace"""
    import marvel_b200 as mb
    n = int(blk.rlen[0])
    r = np.zeros(nrec, mb.OVL_DTYPE)
    r["aepos"] = r["bepos"] = n
    r["tlen"] = 2 * (n // ts)
    tr = np.tile(np.array([0, ts], np.uint8), n // ts)
    assert not ctx.compute_trace_pts(r, tr, 0, 0, 0).any()


def big_batch(ctx, nseeds, stride, blk):
    z = np.zeros(nseeds, np.int32)
    n = np.full(nseeds, blk.rlen[0], np.int32)
    out, _, _ = ctx.local_alignment_batch(blk.bases, z + 1, n, blk.bases.copy(), z + 1, n, z, z, 0, stride)
    assert (out[:, 2] == n[0]).all()


def test_large_calls_return_their_memory():
    """A trace check of 20 M segments (36 bytes each) and a batch with 1 GB of trace rows keep
    less than 300 MB beyond what a small one keeps."""
    import marvel_b200 as mb
    ctx = mb.Context()
    ctx.set_filter_params()
    blk = one_read(20000)
    ctx.new_align_spec(0.70, 2, blk.freq)
    ctx.load_block(0, blk)
    big_check(ctx, 2, blk)
    before = free()
    big_check(ctx, 2000, blk)
    assert before - free() < 300 << 20
    ctx.new_align_spec(0.70, 100, blk.freq)
    big_batch(ctx, 500, 2000, blk)
    before = free()
    big_batch(ctx, 500, 1 << 20, blk)
    assert before - free() < 300 << 20
    ctx.close()


def test_kept_memory_is_freed_for_a_call_that_needs_it():
    """Buffers that a seed batch and a trace check left do not stand in the way of a block, an index or a
    comparison."""
    import marvel_b200 as mb
    small, blk = one_read(20000), random_block(np.random.default_rng(1), 1500, 6000)
    plain = mb.Context()
    want = mb.daligner_block(plain, blk)
    need = plain.test_memory_limit()
    plain.close()
    ctx = mb.Context()
    ctx.set_filter_params()
    ctx.new_align_spec(0.70, 2, small.freq)
    ctx.load_block(0, small)
    big_check(ctx, 300, small)
    ctx.new_align_spec(0.70, 100, small.freq)
    big_batch(ctx, 500, 100000, small)
    kept = ctx.test_memory_limit()
    assert kept > 200 << 20
    ctx.test_memory_limit(need + (8 << 20))
    got = mb.daligner_block(ctx, blk)
    assert got[0].tobytes() == want[0].tobytes() and got[1].tobytes() == want[1].tobytes()
    held = ctx.test_memory_limit(need // 2)  # what does not fit either way is an error, and the context goes on
    assert held <= need + (8 << 20)
    with pytest.raises(mb.GpuError, match="cudaMalloc"):
        big_batch(ctx, 500, 4 << 20, small)
    ctx.test_memory_limit(0)
    big_batch(ctx, 20, 2000, small)
    got = mb.daligner_block(ctx, blk)
    assert got[0].tobytes() == want[0].tobytes() and got[1].tobytes() == want[1].tobytes()
    ctx.close()


def test_comparison_without_room_for_seeds_ahead():
    """A block of tandem repeats, whose seeds are aligned ahead where there is room: without it they are
    not, and the comparison gives the same."""
    import marvel_b200 as mb
    from test_gpu_ahead import block, reads
    blk = block(reads(np.random.default_rng(7), 60, 3000, 8, 0.12, False))
    ctx = mb.Context()
    want = mb.daligner_block(ctx, blk)
    need = ctx.test_memory_limit()
    ctx.close()
    for short in (60 << 20, 125 << 20):  # less than all of the seeds' buffers (136 MB), all but the smallest
        ctx = mb.Context()
        ctx.test_memory_limit(need - short)
        for _ in range(2):
            got = mb.daligner_block(ctx, blk)
            assert got[0].tobytes() == want[0].tobytes() and got[1].tobytes() == want[1].tobytes()
        assert ctx.test_memory_limit() <= need - short
        ctx.close()


def test_failed_load_leaves_the_slot_empty():
    """A block, or a complement, that finds no memory: calls on its slot are errors until one is loaded."""
    import marvel_b200 as mb
    small, big = one_read(20000), one_read(40 << 20)
    ctx = mb.Context()
    ctx.set_filter_params()
    ctx.new_align_spec(0.70, 100, small.freq)
    for slot in (0, 2):
        ctx.load_block(slot, small)
        ctx.sort_kmers(slot)
    ctx.load_block(1, big)
    ctx.test_memory_limit(ctx.test_memory_limit() + (1 << 20))
    with pytest.raises(mb.GpuError, match="cudaMalloc"):
        ctx.load_block(0, big)
    with pytest.raises(mb.GpuError, match="cudaMalloc"):
        ctx.complement_block(1, 2)
    for slot in (0, 2):
        with pytest.raises(mb.GpuError, match="not loaded"):
            ctx.sort_kmers(slot)
        with pytest.raises(mb.GpuError, match="not loaded"):
            ctx.dust(slot, small.freq)
    with pytest.raises(mb.GpuError, match="built before"):
        ctx.match_filter(1, 0, 0)
    ctx.load_block(0, small)
    assert ctx.sort_kmers(0) == 20000 - 13
    ctx.close()
