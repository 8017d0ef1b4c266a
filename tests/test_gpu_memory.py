"""Device memory of a context: all of it returns when it is destroyed."""
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
