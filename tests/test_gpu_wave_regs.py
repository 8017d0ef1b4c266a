"""Local_Alignment's waves in registers (bands of up to 30 diagonals) against the restatement: bands
that widen past 30 diagonals and narrow again, matches over many trace points in one step, trace
spacings of every size, both orientations, seeds in mid-read (forward and reverse waves)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def mutate(rng, s, rate):
    keep = rng.random(s.size) >= rate / 3
    s = s[keep].copy()
    m = rng.random(s.size) < rate / 3
    s[m] = rng.integers(0, 4, int(m.sum()), dtype=np.uint8)
    at = np.nonzero(rng.random(s.size) < rate / 3)[0]
    return np.insert(s, at, rng.integers(0, 4, at.size, dtype=np.uint8))


def pairs(rng):
    """(a, b, position of a shared point in a and in b)"""
    out = []
    for n, rate in ((900, 0.0), (20000, 0.0), (20000, 0.001), (6000, 0.02), (6000, 0.15), (4000, 0.3), (2500, 0.45)):
        s = rng.integers(0, 4, n, dtype=np.uint8)
        out.append((mutate(rng, s, rate), mutate(rng, s, rate), 0, 0))
    for period in (1, 2, 3, 7, 40, 90):  # tandem repeats: every diagonal a period away matches too
        unit = rng.integers(0, 4, period, dtype=np.uint8)
        t = np.tile(unit, 1500 // period + 1)
        u, v = rng.integers(0, 4, (2, 1200), dtype=np.uint8)
        x = np.concatenate([u, t, v])
        out.append((mutate(rng, x, 0.1), mutate(rng, x, 0.1), 0, 0))
    # a shared stretch inside unrelated flanks: the band spreads where the match ends
    for n in (300, 1500):
        s = rng.integers(0, 4, n, dtype=np.uint8)
        f = [rng.integers(0, 4, 1500, dtype=np.uint8) for _ in range(4)]
        out.append((np.concatenate([f[0], s, f[1]]), np.concatenate([f[2], mutate(rng, s, 0.1), f[3]]), 1500 + n // 2,
                    1500 + n // 2))
    # the match begins and ends with the reads
    s = rng.integers(0, 4, 3000, dtype=np.uint8)
    out.append((s[:2000], mutate(rng, s[700:], 0.1), 1200, 500))
    out.append((mutate(rng, s[700:], 0.1), s[:2000], 500, 1200))
    return out


@pytest.mark.parametrize("ts", [2, 16, 25, 100, 126, 500])
@pytest.mark.parametrize("comp", [0, 1])
def test_waves_match_oracle(ts, comp):
    import marvel_b200 as mb
    import oracle
    rng = np.random.default_rng(10 * ts + comp)
    ps = pairs(rng)
    freq = np.full(4, .25, np.float32)
    p = oracle.make_params(freq, s=ts)
    ctx = mb.Context()
    ctx.new_align_spec(0.70, ts, freq)
    ctx.set_capacities(pebbles=1 << 20)  # room for the marks of the smallest spacings
    four = np.array([4], np.uint8)
    abuf = np.concatenate([four] + [np.append(a, four) for a, _, _, _ in ps])
    bbuf = np.concatenate([four] + [np.append(b, four) for _, b, _, _ in ps])
    alen = np.array([a.size for a, _, _, _ in ps], np.int32)
    blen = np.array([b.size for _, b, _, _ in ps], np.int32)
    aoff = 1 + np.concatenate([[0], np.cumsum(alen[:-1].astype(np.int64) + 1)])
    boff = 1 + np.concatenate([[0], np.cumsum(blen[:-1].astype(np.int64) + 1)])
    idx, diag, anti = [], [], []
    for i, (a, b, pa, pb) in enumerate(ps):
        for f in (0.0, 0.3, 0.6):
            x = pa or int(f * min(a.size, b.size))
            y = pb or x
            idx.append(i)
            diag.append(x - y)
            anti.append(x + y)
    diag, anti = np.array(diag, np.int32), np.array(anti, np.int32)
    out, tr, cells = ctx.local_alignment_batch(abuf, aoff[idx], alen[idx], bbuf, boff[idx], blen[idx], diag, anti, comp)
    half = tr.shape[1] // 2
    for n, i in enumerate(idx):
        a = np.concatenate([four, ps[i][0], four])
        b = np.concatenate([four, ps[i][1], four])
        o, at, bt, oc = oracle.local_alignment(a, b, comp, int(diag[n]), int(anti[n]), p)
        assert (out[n] == o).all(), (n, i, out[n], o)
        assert (tr[n, :o[5]] == at).all() and (tr[n, half:half + o[11]] == bt).all()
        assert cells[n] == oc
    ctx.close()


def test_batch_of_a_longer_read_than_its_length_reads_bytes():
    """A length that ends before the read's 4: the byte waves run on to the 4, as they always have."""
    import marvel_b200 as mb
    import oracle
    rng = np.random.default_rng(3)
    s = rng.integers(0, 4, 3000, dtype=np.uint8)
    a, b = mutate(rng, s, 0.1), mutate(rng, s, 0.1)
    freq = np.full(4, .25, np.float32)
    ctx = mb.Context()
    ctx.new_align_spec(0.70, 100, freq)
    four = np.array([4], np.uint8)
    abuf, bbuf = np.concatenate([four, a, four]), np.concatenate([four, b, four])
    one = np.ones(1, np.int64)
    o, at, bt, oc = oracle.local_alignment(abuf, bbuf, 0, 0, 0, oracle.make_params(freq))
    out, tr, cells = ctx.local_alignment_batch(abuf, one, [a.size - 1], bbuf, one, [b.size], [0], [0], 0)
    assert out[0, :7].tolist() == o[:7].tolist() and cells[0] == oc
    assert (tr[0, :o[5]] == at).all()
    ctx.close()
