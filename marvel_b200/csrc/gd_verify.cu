// gd_verify.cu -- Compute_Trace_PTS on the device: exact differences of .las records.
//
// Restates dalign/align.c Compute_Trace_PTS (:5286-5397) with the distance part of iter_np
// (:4556-4917): each record is cut at its trace points (one segment per trace-spacing
// interval of the A read), every segment is aligned exactly with the O(np) waves, and the
// segment distances add up to the record's diffs.  GPU mapping: a warp per record forms its
// segments from the trace (a scan of the B lengths), then one thread per segment (segments are
// independent, ~100 bases each) aligns it in a band held in shared memory, distances summed
// per record with atomics; the few segments whose band outgrows it take three wave vectors in
// global scratch.  This is the check
// LAcheck -a runs (utils/LAcheck.c:236-252), for a whole overlap buffer at once.
#include "gd_verify.cuh"

namespace gd
{

constexpr int VT = 128;

__device__ int iter_np_dist(const uint8_t* A, int M, const uint8_t* B, int N, int* b0, int* b1, int* b2)
{
    int del = M - N, low, hgh, D, k, j, i, am, ac, ap;
    int *F0, *F1, *F2, *nf;
    if (del >= 0)
    {
        low = 0;
        hgh = del;
    }
    else
    {
        low = del;
        hgh = 0;
    }
    F1 = b1;
    F0 = b2;
    nf = b0;
    for (k = low - 1; k <= hgh + 1; k++)
        F1[k] = F0[k] = -2;
    F0[0] = -1;
    low += 1;
    hgh -= 1;
    for (D = 0; D <= M + N + 2; D++)
    {
        int* t = nf;
        F2 = F1;
        F1 = F0;
        F0 = t;
        nf = F2;
        if ((D & 1) == 0)
        {
            low -= 1;
            hgh += 1;
        }
        F0[hgh + 1] = F0[low - 1] = -2;
        // one furthest-reaching step (FS_MOVE, align.c:4640-4672): the best of the two
        // waves back, the previous wave plus a substitution, and the neighbour on this wave
#define GD_FS(AP, AM)                                       \
    ap = (AP);                                              \
    am = (AM);                                              \
    ac = F1[k] + 1;                                         \
    if (ac < am)                                            \
        j = (ap < am) ? am : ap;                            \
    else if (ap < ac)                                       \
        j = ac;                                             \
    else                                                    \
        j = ap;                                             \
    i = M - k;                                              \
    {                                                       \
        int lim = (N < i) ? N : i;                          \
        while (j < lim && __ldg(B + j) == __ldg(A + j + k)) \
            j += 1;                                         \
    }                                                       \
    F0[k] = j;
        j = -2;
        for (k = hgh; k > del; k--)
        {
            GD_FS(j + 1, F2[k - 1])
        }
        j = -2;
        for (k = low; k < del; k++)
        {
            GD_FS(F2[k + 1] + 1, j)
        }
        k = del;
        GD_FS(F0[del + 1] + 1, j)
#undef GD_FS
        if (F0[del] >= N)
            return D + abs(del);
    }
    return -1;
}

// The segments of the records, a warp per record: the host used to build them and copy 32 bytes
// a segment (45,000 records, 2.5 M segments: about 90 of the call's 105 ms).
__global__ void __launch_bounds__(VT) k_trace_segments(const OutRec* __restrict__ recs, int64_t n,
                                                      const int64_t* __restrict__ first,
                                                      const uint8_t* __restrict__ trace, uint64_t tlo, int TS,
                                                      int tbytes, int afirst, int bfirst, Segment* __restrict__ seg,
                                                      unsigned* R, DevStatus* st)
{
    const int64_t r = ((int64_t)blockIdx.x * VT + threadIdx.x) >> 5;
    const int lane = lane_id();
    if (r >= n)
        return;
    const OutRec o = recs[r];
    const int inner = trace_inner(o.tlen);
    Segment* const out = seg + first[r];
    const uint8_t* const t = trace + (o.toff - tlo);
    Segment g;
    g.aread = o.aread - afirst;
    g.bread = o.bread - bfirst;
    g.rec = (int32_t)r;
    g.comp = o.flags & 1;
    int top = 0;
    bool bad = false;
    long long bb0 = o.bbpos;  // B position at the chunk's start
    for (int base = 0; base <= inner; base += 32)
    {
        const int i = base + lane;
        int len = 0;
        if (i < inner)
            len = tbytes == 1 ? t[2 * i + 1] : t[4 * i + 2] | (t[4 * i + 3] << 8);
        int x = len;
#pragma unroll
        for (int k = 1; k < 32; k <<= 1)
        {
            const int y = __shfl_up_sync(GD_FULL, x, k);
            if (lane >= k)
                x += y;
        }
        if (i <= inner)
        {
            const long long ab = i ? (long long)(o.abpos / TS + i) * TS : o.abpos;
            const long long ae = i < inner ? (long long)(o.abpos / TS + i + 1) * TS : o.aepos;
            const long long bb = bb0 + x - len, be = i < inner ? bb0 + x : o.bepos;
            if (ae < ab || be < bb || ae > o.aepos || be > o.bepos)
            {
                bad = true;
                g.ab = g.ae = g.bb = g.be = 0;
            }
            else
            {
                g.ab = (int)ab;
                g.ae = (int)ae;
                g.bb = (int)bb;
                g.be = (int)be;
                top = max(top, (g.ae - g.ab) + (g.be - g.bb) + 8);
            }
            out[i] = g;
        }
        bb0 += __shfl_sync(GD_FULL, x, 31);
    }
    top = __reduce_max_sync(GD_FULL, top);
    if (__any_sync(GD_FULL, bad) && lane == 0)
        gd_fail(st, GD_ERR_TRACE, (int)r, 0);
    if (lane == 0 && (unsigned)top > *R)
        atomicMax(R, (unsigned)top);
}

// One thread per segment.  A diagonal's last two waves share one shared-memory word (the newer in
// the low half), updated in place: the sweep down reads the older value of the diagonal below and
// the sweep up that of the diagonal above before either is written, as FS_MOVE's order has
// it.  VBAND diagonals fit ([diagonal][thread], free of bank conflicts); the extension compares 16
// bases of the 2-bit copies at a time.  A thread's three full-width int vectors in global
// scratch took 15.3 ms for the 2.5 M segments of 45,000 records.
constexpr int VBAND = 64;

__global__ void __launch_bounds__(VT) k_trace_pts(DevBlock A, DevBlock B, DevBlock C, const Segment* __restrict__ seg,
                                                 int64_t nseg, int* diffs, unsigned* list, unsigned* nlist, const unsigned* __restrict__ oddA,
                                                 const unsigned* __restrict__ oddB,
                                                 const unsigned* __restrict__ oddC)
{
    __shared__ int band[VBAND][VT];
    const int64_t s = (int64_t)blockIdx.x * VT + threadIdx.x;
    if (s >= nseg)
        return;
    const Segment g = seg[s];
    const DevBlock& bb = g.comp ? C : B;
    const int M = g.ae - g.ab, N = g.be - g.bb, del = M - N;
    const uint32_t a0 = PK_BIAS + (uint32_t)A.boff[g.aread] + (uint32_t)g.ab;
    const uint32_t b0 = PK_BIAS + (uint32_t)bb.boff[g.bread] + (uint32_t)g.bb;
    int low = min(0, del), hgh = max(0, del), d = -1;
    const int room = (VBAND - (hgh - low + 3)) / 2;  // diagonals the band can grow on either side
    if (!(*oddA | *oddB | *oddC) && hgh - low + 3 <= VBAND && N < 32000)
    {
        int* const w0 = &band[0][threadIdx.x] - (low - 1 - room) * VT;  // diagonal k at w0[k * VT]
        const int lo = low - 1 - room, hi = hgh + 1 + room;
        auto lof = [&](int k) { return (int)(short)w0[k * VT]; };
        auto hif = [&](int k) { return w0[k * VT] >> 16; };
        const int none = (int)0xfffefffe;  // -2 in both halves
        for (int k = low - 1; k <= hgh + 1; k++)
            w0[k * VT] = none;
        w0[0] = (int)0xfffeffff;  // the wave before the first: -1 on the main diagonal
        low += 1;
        hgh -= 1;
        auto extend = [&](int j, int k) {
            int n = min(N, M - k) - j;
            while (n > 0)
            {
                const uint32_t pb = b0 + j, pa = a0 + j + k;
                const uint32_t vb =
                    __funnelshift_r(__ldg(bb.pk + (pb >> 4)), __ldg(bb.pk + (pb >> 4) + 1), 2 * pb);
                const uint32_t va = __funnelshift_r(__ldg(A.pk + (pa >> 4)), __ldg(A.pk + (pa >> 4) + 1), 2 * pa);
                const int m = min(__clz((int)__brev(va ^ vb)) >> 1, n);
                j += m;
                if (m < 16)
                    break;
                n -= 16;
            }
            w0[k * VT] = (j & 0xffff) | (w0[k * VT] << 16);
            return j;
        };
        for (int D = 0;; D++)
        {
            if ((D & 1) == 0)
            {
                low -= 1;
                hgh += 1;
                if (low - 1 < lo || hgh + 1 > hi)
                    break;
                if (D)
                    w0[(low - 1) * VT] = w0[(hgh + 1) * VT] = none;
            }
            int j = -2;
            for (int k = hgh; k > del; k--)
                j = extend(max(max(j + 1, hif(k - 1)), lof(k) + 1), k);
            j = -2;
            for (int k = low; k < del; k++)
                j = extend(max(max(hif(k + 1) + 1, j), lof(k) + 1), k);
            j = extend(max(max(lof(del + 1) + 1, j), lof(del) + 1), del);
            if (j >= N)
            {
                d = D + abs(del);
                break;
            }
        }
    }
    if (d < 0)
        list[atomicAdd(nlist, 1u)] = (unsigned)s;
    else if (d)
        atomicAdd(diffs + g.rec, d);
}

__global__ void __launch_bounds__(VT) k_trace_pts_list(DevBlock A, DevBlock B, DevBlock C,
                                                      const Segment* __restrict__ seg,
                                                      const unsigned* __restrict__ list, unsigned nlist, int* scratch,
                                                      int R, int* diffs, DevStatus* st)
{
    const unsigned nthreads = gridDim.x * VT;
    const unsigned tid = blockIdx.x * VT + threadIdx.x;
    int* mem = scratch + (int64_t)tid * 3 * (2 * R + 1);
    int* b0 = mem + R;
    int* b1 = mem + (2 * R + 1) + R;
    int* b2 = mem + 2 * (2 * R + 1) + R;
    for (unsigned i = tid; i < nlist; i += nthreads)
    {
        const Segment g = seg[list[i]];
        const DevBlock& bb = g.comp ? C : B;
        const uint8_t* a = A.bases + A.boff[g.aread] + g.ab;
        const uint8_t* b = bb.bases + bb.boff[g.bread] + g.bb;
        int d = iter_np_dist(a, g.ae - g.ab, b, g.be - g.bb, b0, b1, b2);
        if (d < 0)
        {
            gd_fail(st, GD_ERR_TRACE, (int)g.rec, -1);
            continue;
        }
        atomicAdd(diffs + g.rec, d);
    }
}

// *odd = 1 when a read holds a byte beyond 3; a CTA per read
__global__ void __launch_bounds__(VT) k_block_plain(DevBlock b, unsigned* odd)
{
    if (!plain_bases(b.bases + b.boff[blockIdx.x], b.rlen[blockIdx.x], threadIdx.x, VT))
        *odd = 1;
}

int launch_block_plain(const DevBlock& b, unsigned* odd, cudaStream_t s)
{
    if (b.nreads <= 0)
        return 0;
    k_block_plain<<<b.nreads, VT, 0, s>>>(b, odd);
    GD_LAUNCHED(1);
    GD_CUDA(cudaGetLastError());
    return 0;
}

int launch_trace_segments(const OutRec* recs, int64_t n, const int64_t* first, const uint8_t* trace, uint64_t tlo,
                          int tspace, int tbytes, int afirst, int bfirst, Segment* seg, unsigned* R, DevStatus* st,
                          cudaStream_t s)
{
    if (n <= 0)
        return 0;
    k_trace_segments<<<(unsigned)((n * 32 + VT - 1) / VT), VT, 0, s>>>(recs, n, first, trace, tlo, tspace, tbytes, afirst,
                                                                      bfirst, seg, R, st);
    GD_LAUNCHED(1);
    GD_CUDA(cudaGetLastError());
    return 0;
}

int launch_trace_pts(const DevBlock& A, const DevBlock& B, const DevBlock& C, const Segment* seg, int64_t nseg,
                     int* diffs, unsigned* list, unsigned* nlist, const unsigned* const odd[3], cudaStream_t s)
{
    if (nseg <= 0)
        return 0;
    if (nseg > UINT32_MAX)
    {
        gd_set_error("%lld trace segments exceed the 32-bit segment index of this build", (long long)nseg);
        return -1;
    }
    k_trace_pts<<<(unsigned)((nseg + VT - 1) / VT), VT, 0, s>>>(A, B, C, seg, nseg, diffs, list, nlist, odd[0], odd[1], odd[2]);
    GD_LAUNCHED(1);
    GD_CUDA(cudaGetLastError());
    return 0;
}

int launch_trace_pts_list(const DevBlock& A, const DevBlock& B, const DevBlock& C, const Segment* seg,
                          const unsigned* list, unsigned nlist, int* scratch, int R, int nthreads, int* diffs,
                          DevStatus* st, cudaStream_t s)
{
    k_trace_pts_list<<<nthreads / VT, VT, 0, s>>>(A, B, C, seg, list, nlist, scratch, R, diffs, st);
    GD_LAUNCHED(1);
    GD_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace gd
