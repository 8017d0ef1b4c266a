"""Reads of few errors, whose pair groups hold a hit per base: thousands of candidate seeds of a group, all
but a few covered by the alignments before them.  Records, traces, seeds and wave cells against the oracle."""
import numpy as np
import pytest

from marvel_b200 import dazzdb
from test_gpu_ahead import block, noisy

pytestmark = pytest.mark.gpu


def genome_reads(rng, n, length, count, rate, copies):
    """reads of both strands from a genome with a repeat family, one read longer than a panel of hits"""
    g = rng.integers(0, 4, n, dtype=np.uint8)
    unit = rng.integers(0, 4, 700, dtype=np.uint8)
    for p in rng.integers(0, n - unit.size, copies):
        g[p:p + unit.size] = unit
    spans = [(0, min(n, 70000))] + [(int(a), int(rng.integers(length // 2, length)))
                                    for a in rng.integers(0, n - length, count - 1)]
    out = []
    for a, m in spans:
        r = noisy(rng, g[a:a + m], rate)
        out.append(np.uint8(3) - r[::-1] if rng.random() < 0.5 else r)
    return out


@pytest.mark.parametrize("rate", [0.0, 0.002, 0.01, 0.04])
@pytest.mark.parametrize("copies,d2", [(0, False), (6, False), (6, True)])
def test_accurate_reads_match_oracle(rate, copies, d2, tmp_path):
    import marvel_b200 as mb
    import oracle
    rng = np.random.default_rng(int(1000 * rate) + copies)
    A = block(genome_reads(rng, 90000, 9000, 24, rate, copies))
    ctx = mb.Context()
    recs, tr = (mb.daligner2_block if d2 else mb.daligner_block)(ctx, A)
    st = ctx.stats()
    ctx.close()
    p = oracle.make_params(A.freq, variant=2 if d2 else 1)
    orecs, otraces, ost = oracle.daligner(A, A, dazzdb.complement_block(A), p, True)
    assert recs.size == len(orecs) > 50
    assert st["seeds"] == [ost["seeds_n"], ost["seeds_c"]]
    assert sum(st["cells"]) == ost["cells"]
    mb.write_las(str(tmp_path / "g.las"), recs, tr, 100)
    oracle.write_las(str(tmp_path / "o.las"), orecs, otraces, 100)
    ok, msg = dazzdb.las_equal(str(tmp_path / "g.las"), str(tmp_path / "o.las"))
    assert ok, msg
