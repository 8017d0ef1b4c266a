"""Local_Alignment batches outside the block layout: the batch must give what the byte waves give (the
entry point that allocates nothing reads the bytes always), which end at 4s, not at lengths."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PAD = 1024


def noisy(rng, s, rate=0.1):
    s = s[rng.random(s.size) >= rate / 3].copy()
    m = rng.random(s.size) < rate / 3
    s[m] = rng.integers(0, 4, int(m.sum()), dtype=np.uint8)
    at = np.nonzero(rng.random(s.size) < rate / 3)[0]
    return np.insert(s, at, rng.integers(0, 4, at.size, dtype=np.uint8))


def joined(reads):
    """[4, read, 4, read, ..., 4] and the reads' offsets and lengths"""
    four = np.array([4], np.uint8)
    buf = np.concatenate([four] + [np.append(r, four) for r in reads])
    n = np.array([r.size for r in reads], np.int32)
    return buf, 1 + np.concatenate([[0], np.cumsum(n[:-1].astype(np.int64) + 1)]), n


def byte_waves(ctx, abuf, aoff, alen, bbuf, boff, blen, diag, anti, comp, stride):
    import torch
    import marvel_b200 as mb
    bufs = []
    for b in (abuf, bbuf):
        t = torch.full((b.size + 2 * PAD,), 4, dtype=torch.uint8, device="cuda")
        t[PAD:PAD + b.size] = torch.from_numpy(b).cuda()
        bufs.append(t)
    ins = [torch.from_numpy(np.ascontiguousarray(x, t)).cuda() for x, t in
           ((aoff, np.int64), (alen, np.int32), (boff, np.int64), (blen, np.int32), (diag, np.int32), (anti, np.int32))]
    n = len(diag)
    out = torch.zeros((n, 12), dtype=torch.int32, device="cuda")
    tr = torch.zeros((n, stride), dtype=torch.int16, device="cuda")
    cells = torch.zeros(n, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    mb._check(mb.lib().gd_local_alignment_batch_noalloc(
        ctx.h, bufs[0].data_ptr() + PAD, bufs[1].data_ptr() + PAD, *[t.data_ptr() for t in ins], n,
        int(max(np.max(alen), np.max(blen))), comp, out.data_ptr(), tr.data_ptr(), stride, cells.data_ptr(),
        torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return out.cpu().numpy(), tr.cpu().numpy().view(np.uint16), cells.cpu().numpy()


def same_as_bytes(ctx, *call):
    import marvel_b200 as mb
    stride = 2 * (4 * (int(max(np.max(call[2]), np.max(call[5]))) // 100 + 2) + 16)
    try:
        bo, bt, bc = byte_waves(ctx, *call, stride)
    except mb.GpuError as e:  # waves that find no band: the same failure from both
        with pytest.raises(mb.GpuError, match=str(e).split("seed")[1].split("(")[0]):
            ctx.local_alignment_batch(*call)
        return None
    out, tr, cells = ctx.local_alignment_batch(*call)
    assert tr.shape[1] == stride
    assert np.array_equal(out, bo) and np.array_equal(cells, bc)
    half = tr.shape[1] // 2
    for i, o in enumerate(out):
        assert np.array_equal(tr[i, :o[5]], bt[i, :o[5]]) and np.array_equal(tr[i, half:half + o[11]],
                                                                            bt[i, half:half + o[11]])
    return out


@pytest.fixture
def ctx():
    import marvel_b200 as mb
    c = mb.Context()
    c.new_align_spec(0.70, 100, np.full(4, .25, np.float32))
    yield c
    c.close()


@pytest.mark.parametrize("comp", [0, 1])
@pytest.mark.parametrize("over", [2, 17, 700, 5000])
def test_length_past_the_sequences(ctx, over, comp):
    """The last read's length runs past the end of its buffer, in A, in B, in both."""
    rng = np.random.default_rng(over + comp)
    s = rng.integers(0, 4, 3000, dtype=np.uint8)
    abuf, aoff, alen = joined([rng.integers(0, 4, 400, dtype=np.uint8), noisy(rng, s)])
    bbuf, boff, blen = joined([rng.integers(0, 4, 300, dtype=np.uint8), noisy(rng, s)])
    one = np.array([1, 1, 1])
    same_as_bytes(ctx, abuf, aoff[one], alen[one] + [over, 0, over], bbuf, boff[one], blen[one] + [0, over, over],
                  [0, 0, 0], [0, 1600, 3000], comp)


@pytest.mark.parametrize("comp", [0, 1])
@pytest.mark.parametrize("at", [0, 1, 7, 511, 1600, -2, -1])
@pytest.mark.parametrize("value", [4, 5, 255])
def test_byte_beyond_3_inside_a_read(ctx, value, at, comp):
    """A 4 inside a read ends it there; other bytes match nothing but themselves.  In A, in B, in both."""
    rng = np.random.default_rng(at % 97 + comp)
    s = rng.integers(0, 4, 3000, dtype=np.uint8)
    abuf, aoff, alen = joined([noisy(rng, s), noisy(rng, s)])
    bbuf, boff, blen = joined([noisy(rng, s), noisy(rng, s)])
    for buf, off, n in ((abuf, aoff, alen), (bbuf, boff, blen)):
        buf[off[1] + at % n[1]] = value
    i, j = np.array([1, 0, 1, 0]), np.array([0, 1, 1, 0])
    same_as_bytes(ctx, abuf, aoff[i], alen[i], bbuf, boff[j], blen[j], [0, 2, -3, 1], [200, 1400, 2901, 3001], comp)


@pytest.mark.parametrize("comp", [0, 1])
def test_length_over_a_separator(ctx, comp):
    """Lengths that take the 4 behind a read with them, or the read behind that too."""
    rng = np.random.default_rng(40 + comp)
    s = rng.integers(0, 4, 3000, dtype=np.uint8)
    abuf, aoff, alen = joined([noisy(rng, s[:1500]), noisy(rng, s[1500:])])
    bbuf, boff, blen = joined([noisy(rng, s), noisy(rng, s)])
    both = alen[0] + 1 + alen[1]
    same_as_bytes(ctx, abuf, aoff[[0, 0, 1]], np.array([alen[0] + 1, both, alen[1] + 1]), bbuf, boff[[0, 1, 1]],
                  np.array([blen[0], blen[1] + 1, blen[1] + 1]), [0, 0, 0], [400, 400, 800], comp)


def test_seed_outside_its_reads(ctx):
    """Positions beyond a read's ends but within its buffer, whose bytes the waves then read."""
    rng = np.random.default_rng(5)
    s = rng.integers(0, 4, 2000, dtype=np.uint8)
    reads = [s[:900], noisy(rng, s[:1000])]
    buf, off, n = joined(reads)
    for x, y in ((905, 3), (3, 905), (-1, -1), (900, 900), (901, 902)):
        same_as_bytes(ctx, buf, off[:1], n[:1], buf.copy(), off[:1], n[:1], [x - y], [x + y], 0)


def test_seed_outside_the_sequences_is_refused(ctx):
    import marvel_b200 as mb
    buf, off, n = joined([np.zeros(500, np.uint8)])
    for o, x, y in ((1, 600, 0), (1, 0, 600), (1, -90, 0), (1, 0, -90), (-200, 0, 0), (5000, 0, 0), (1, 1 << 29, 0)):
        with pytest.raises(mb.GpuError, match="outside the sequences"):
            ctx.local_alignment_batch(buf, [o], n, buf, [o], n, [x - y], [x + y], 0)


def test_results_do_not_depend_on_earlier_calls(ctx):
    """Whole trace rows, the part behind the trace included."""
    import marvel_b200 as mb
    rng = np.random.default_rng(8)
    s = rng.integers(0, 4, 4000, dtype=np.uint8)
    buf, off, n = joined([noisy(rng, s), noisy(rng, s)])
    first = (buf, off[[0, 0]], n[[0, 0]], buf.copy(), off[[1, 1]], n[[1, 1]], [0, 0], [3000, 5000], 0)
    second = (buf, off[[0, 0]], n[[0, 0]], buf.copy(), off[[1, 1]], n[[1, 1]], [900, -900], [3100, 5000], 0)
    ctx.local_alignment_batch(*first)
    got = ctx.local_alignment_batch(*second)
    fresh = mb.Context()
    fresh.new_align_spec(0.70, 100, np.full(4, .25, np.float32))
    want = fresh.local_alignment_batch(*second)
    fresh.close()
    for g, w in zip(got, want):
        assert np.array_equal(g, w)
    half = got[1].shape[1] // 2
    for o, row in zip(*got[:2]):
        assert not row[o[5]:half].any() and not row[half + o[11]:].any()


@pytest.mark.parametrize("comp", [0, 1])
@pytest.mark.parametrize("length,fits", [(2999, True), (2500, True), (100, False)])
def test_length_far_below_the_read(ctx, length, fits, comp):
    """Byte waves run on to the read's 4, up to a match of the length at a time: where the trace outgrows
    the room that the lengths give it, an error of that seed (code 3), and the context goes on."""
    import marvel_b200 as mb
    rng = np.random.default_rng(60 + comp)
    s = rng.integers(0, 4, 3000, dtype=np.uint8)
    t = s.copy()
    t[80::90] = (t[80::90] + 1) & 3
    abuf, aoff, alen = joined([s])
    bbuf, boff, blen = joined([t])
    n = np.array([length], np.int32)
    for at in (0, min(length, 1400)):
        call = (abuf, aoff, n, bbuf, boff, n, [0], [2 * at], comp)
        out = same_as_bytes(ctx, *call)
        assert (out is not None) == fits
        if not fits:
            with pytest.raises(mb.GpuError, match="code 3"):
                ctx.local_alignment_batch(*call)
    assert same_as_bytes(ctx, abuf, aoff, alen, bbuf, boff, blen, [0], [0], comp) is not None
