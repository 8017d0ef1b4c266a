"""Pair groups with thousands of hits, whose likely seeds are aligned ahead of the pair kernel, against
the oracle: reads that share a tandem array (with flanks of their own or of one genome), block
against itself and block pairs, more bands with a seed than are aligned ahead.  Records,
traces, seeds and wave cells."""
import numpy as np
import pytest

from marvel_b200 import dazzdb

pytestmark = pytest.mark.gpu


def block(reads):
    rlen = np.array([r.size for r in reads], np.int32)
    boff = np.zeros(len(reads) + 1, np.int64)
    boff[1:] = np.cumsum(rlen.astype(np.int64) + 1)
    bases = np.full(int(boff[-1]) + 1, 4, np.uint8)
    for i, r in enumerate(reads):
        bases[boff[i] + 1:boff[i] + 1 + r.size] = r
    return dazzdb.Block(bases, boff, rlen, 0, 1, np.full(4, .25, np.float32), int(rlen.max()), int(rlen.sum()))


def noisy(rng, s, rate):
    s = s[rng.random(s.size) >= rate / 3].copy()
    m = rng.random(s.size) < rate / 3
    s[m] = rng.integers(0, 4, int(m.sum()), dtype=np.uint8)
    at = np.nonzero(rng.random(s.size) < rate / 3)[0]
    return np.insert(s, at, rng.integers(0, 4, at.size, dtype=np.uint8))


def reads(rng, period, span, n, rate, shared):
    unit = rng.integers(0, 4, period, dtype=np.uint8)
    array = np.tile(unit, span // period + 1)[:span]
    left, right = rng.integers(0, 4, (2, 4000), dtype=np.uint8)
    out = []
    for _ in range(n):
        if not shared:
            left, right = rng.integers(0, 4, (2, int(rng.integers(500, 4000))), dtype=np.uint8)
        g = np.concatenate([left, array[:int(span * rng.uniform(0.7, 1.0))], right])
        out.append(noisy(rng, g[int(rng.integers(0, 400)):], rate))
    return out


@pytest.mark.parametrize("period,span,rate,shared,pair", [(60, 3000, 0.12, False, False), (45, 2500, 0.12, True, True),
                                                          (130, 9000, 0.10, True, False), (64, 20000, 0.06, False, True)])
def test_repeat_groups_match_oracle(period, span, rate, shared, pair, tmp_path):
    import marvel_b200 as mb
    import oracle
    rng = np.random.default_rng(period + span)
    both = reads(rng, period, span, 8 if span < 10000 else 6, rate, shared)
    A = block(both[:len(both) // 2] if pair else both)
    B = block(both[len(both) // 2:]) if pair else None
    ctx = mb.Context()
    recs, tr = mb.daligner_block(ctx, A, B)
    st = ctx.stats()
    ctx.close()
    assert st["hits"][0] > 65536  # the case reaches the rule that aligns ahead
    Bo = B if B is not None else A
    orecs, otraces, ost = oracle.daligner(A, Bo, dazzdb.complement_block(Bo), oracle.make_params(A.freq), B is None)
    assert recs.size == len(orecs)
    assert st["seeds"] == [ost["seeds_n"], ost["seeds_c"]]
    assert sum(st["cells"]) == ost["cells"]
    mb.write_las(str(tmp_path / "g.las"), recs, tr, 100)
    oracle.write_las(str(tmp_path / "o.las"), orecs, otraces, 100)
    ok, msg = dazzdb.las_equal(str(tmp_path / "g.las"), str(tmp_path / "o.las"))
    assert ok, msg
