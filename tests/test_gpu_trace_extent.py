"""Compute_Trace_PTS reads its records' own trace bytes and not what lies between them."""
import ctypes
import mmap

import numpy as np
import pytest

from test_gpu_trace_segments import block, make

pytestmark = pytest.mark.gpu


def setup(ts, seed):
    import marvel_b200 as mb
    import oracle
    reads, recs, traces = make(np.random.default_rng(seed), ts)
    ctx = mb.Context()
    ctx.set_filter_params()
    ctx.new_align_spec(0.70, ts, np.full(4, .25, np.float32))
    ctx.load_block(0, block(reads))
    r = np.zeros(len(recs), mb.OVL_DTYPE)
    for i, (ab, bb, ae, be, br) in enumerate(recs):
        r[i]["abpos"], r[i]["bbpos"], r[i]["aepos"], r[i]["bepos"], r[i]["bread"] = ab, bb, ae, be, br
        r[i]["tlen"] = traces[i].size
    raw = [t.astype(np.uint8 if ts <= 125 else np.uint16).view(np.uint8) for t in traces]
    want = [oracle.trace_pts_diffs(reads[0], reads[x["bread"]], x, t, ts) for x, t in zip(r, traces)]
    return ctx, r, raw, want


@pytest.mark.parametrize("ts", [100, 126])
@pytest.mark.parametrize("gap", [0, 1, 63, 64, 65, 5000])
def test_records_apart_and_in_any_order(ts, gap):
    ctx, r, raw, want = setup(ts, ts + gap)
    at = 7 + np.cumsum([0] + [t.size + gap for t in raw[:-1]])
    buf = np.full(int(at[-1]) + raw[-1].size + 3, 201, np.uint8)
    for a, t in zip(at, raw):
        buf[a:a + t.size] = t
    r["toff"] = at
    rng = np.random.default_rng(gap)
    orders = [np.arange(r.size), np.arange(r.size)[::-1]] + [rng.permutation(r.size) for _ in range(4)]
    for o in orders + [np.repeat(rng.permutation(r.size), 3), np.array([r.size - 1, 0])]:
        assert ctx.compute_trace_pts(r[o], buf, 0, 0, 0).tolist() == [want[i] for i in o]
    ctx.close()


def test_distant_records_take_no_memory_for_the_distance():
    import torch
    ctx, r, raw, want = setup(100, 1)
    small = np.concatenate(raw)
    r["toff"] = np.cumsum([0] + [t.size for t in raw[:-1]])
    assert ctx.compute_trace_pts(r, small, 0, 0, 0).tolist() == want
    far = np.zeros(1 << 30, np.uint8)  # its pages are untouched but for the records'
    at = np.linspace(0, far.size - 4096, r.size).astype(np.int64)
    for a, t in zip(at, raw):
        far[a:a + t.size] = t
    r["toff"] = at
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    assert ctx.compute_trace_pts(r, far, 0, 0, 0).tolist() == want
    assert free - torch.cuda.mem_get_info()[0] < 64 << 20
    ctx.close()


def test_bytes_between_records_are_not_read():
    """Two pieces with a page in between that must not be touched."""
    ctx, r, raw, want = setup(100, 2)
    page = mmap.PAGESIZE
    m = mmap.mmap(-1, 64 * page)
    buf = np.frombuffer(m, np.uint8)
    half = r.size // 2
    first, second = np.concatenate(raw[:half]), np.concatenate(raw[half:])
    assert first.size < 8 * page and second.size < 8 * page
    buf[16 * page - first.size:16 * page] = first
    buf[48 * page:48 * page + second.size] = second
    r["toff"][:half] = 16 * page - first.size + np.cumsum([0] + [t.size for t in raw[:half - 1]])
    r["toff"][half:] = 48 * page + np.cumsum([0] + [t.size for t in raw[half:-1]])
    libc = ctypes.CDLL(None, use_errno=True)
    addr = ctypes.c_void_p(buf.ctypes.data + 16 * page)
    assert libc.mprotect(addr, ctypes.c_size_t(32 * page), 0) == 0
    try:
        got = ctx.compute_trace_pts(r, buf, 0, 0, 0).tolist()
    finally:
        assert libc.mprotect(addr, ctypes.c_size_t(32 * page), mmap.PROT_READ | mmap.PROT_WRITE) == 0
    assert got == want
    ctx.close()
