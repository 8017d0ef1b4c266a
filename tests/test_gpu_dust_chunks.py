"""The chunked DBdust scan against the restatement where it can go wrong: reads whose lengths end
around a chunk's, low-complexity stretches across the chunk borders and longer than a chunk."""
import numpy as np
import pytest

from marvel_b200 import dazzdb

pytestmark = pytest.mark.gpu

CHUNK = 128  # interval starts per chunk (gd_dust.cu)


def block(rng, window):
    lens = [14, 15, 16 + window, CHUNK, CHUNK + 1, CHUNK + 2, CHUNK + 3, CHUNK + 1 + window, 2 * CHUNK + 1, 2 * CHUNK + 2,
            2 * CHUNK + 3, 5 * CHUNK + 517, 9 * CHUNK]
    reads = []
    for n in lens:
        r = rng.integers(0, 4, n, dtype=np.uint8)
        for at in list(range(CHUNK, n, CHUNK)) + [0, n]:  # repeats over the borders, the start and the end
            unit = rng.integers(0, 4, int(rng.integers(1, 6)), dtype=np.uint8)
            span = int(rng.choice([3, 12, 40, window, 3 * window, CHUNK + 200]))
            a = max(0, at - int(rng.integers(0, span + 1)))
            t = np.tile(unit, span // unit.size + 1)[:max(0, min(span, n - a))]
            r[a:a + t.size] = t
        reads.append(r)
    rlen = np.array([r.size for r in reads], np.int32)
    bases = np.concatenate([np.array([4], np.uint8)] + [np.append(r, np.uint8(4)) for r in reads] +
                           [np.full(4, 4, np.uint8)])
    boff = np.zeros(rlen.size + 1, np.int64)
    boff[1:] = np.cumsum(rlen.astype(np.int64) + 1)
    return dazzdb.Block(bases, boff, rlen, 0, 1, np.full(4, .25, np.float32), int(rlen.max()), int(rlen.sum()))


@pytest.mark.parametrize("window,thresh,mflag", [(64, 2.0, 10), (3, 2.0, 2), (5, 0.4, 2), (16, 1.0, 4), (128, 2.0, 10),
                                                 (128, 3.5, 20), (127, 0.1, 3)])
def test_chunked_scan_matches_oracle(window, thresh, mflag):
    import marvel_b200 as mb
    import oracle
    ctx = mb.Context()
    for seed in range(4):
        blk = block(np.random.default_rng(100 * window + seed), window)
        ctx.load_block(0, blk)
        anno, data = ctx.dust(0, blk.freq, window, thresh, mflag)
        oa, od = oracle.dust(blk, window, thresh, mflag)
        assert np.array_equal(anno, oa) and np.array_equal(data, od)
    ctx.close()
