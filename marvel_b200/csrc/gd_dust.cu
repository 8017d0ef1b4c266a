// gd_dust.cu -- DBdust's low-complexity scan (db/DBdust.c:219-487) on the device.
//
// The scan of one read is a sequential state machine (a window of triplet counts, a
// left-trimmed run with its own counts, a short list of candidate intervals).  Its state
// after position j follows from bases near j, so k_dust_chunks cuts every read into chunks and
// gives each a thread that starts W positions early (below).  With -b the sums are
// doubles whose rounding carries the read's whole past, so k_dust_read scans one read per
// thread.  Each read's mask is written to its own slice of a device buffer.  Arithmetic follows the
// reference's types: integer pair-count sums, doubles for the thresholds, and with -b
// (biased) double sums of count * skew, computed with explicit round-to-nearest operations
// so that no multiply-add is fused (the reference's x86-64 build has none either).
#include <climits>
#include <cmath>

#include "gd_dust.cuh"

namespace gd
{

struct DustCand
{
    int beg, end;
    double score;
    int prev, next;
};

__device__ __forceinline__ int dtrip(const uint8_t* b, int x)
{
    return (b[x] << 4) | (b[x + 1] << 2) | b[x + 2];
}

__device__ __forceinline__ void dust_retire(int* mask, int& mtop, int beg, int end)
{
    const int c = end + 2;
    if (mask[mtop] + 1 >= beg)
    {
        if (mask[mtop] < c)
            mask[mtop] = c;
    }
    else
    {
        mask[++mtop] = beg;
        mask[++mtop] = c;
    }
}

// -b: one read per thread, counts and candidates in local memory
__global__ void __launch_bounds__(64) k_dust_read(DevBlock blk, int W, double T, double thr2r,
                                                  const double* __restrict__ skew, int minlen, int* out,
                                                  int* __restrict__ nout)
{
    const int r = blockIdx.x * 64 + threadIdx.x;
    if (r >= blk.nreads)
        return;
    const int rlen = blk.rlen[r];
    const uint8_t* b = blk.bases + blk.boff[r];
    int* mask = out + blk.boff[r] + 4ll * r;  // room for rlen + 4 ints
    int mtop = 0;
    mask[0] = -2;
    const int len = rlen - 2;
    if (len > 0)
    {
        DustCand cd[DUST_MAXW + 1];
        int wcount[64], lcount[64];
        for (int e = 0; e < 64; e++)
            wcount[e] = lcount[e] = 0;
        cd[0].beg = -2;
        cd[0].prev = cd[0].next = 0;
        for (int i = 1; i <= W; i++)
            cd[i].next = (i < W) ? i + 1 : -1;
        int freel = 1, wb = -1, lb = -1;
        double wsr = 0., lsr = 0.;
        auto add = [&](int* cnt, int e, double& sr) {
            sr = __dadd_rn(sr, __dmul_rn((double)cnt[e], skew[e]));
            cnt[e]++;
        };
        auto del = [&](int* cnt, int e, double& sr) {
            cnt[e]--;
            sr = __dsub_rn(sr, __dmul_rn((double)cnt[e], skew[e]));
        };
        for (int j = 0; j < len; j++)
        {
            const int c = dtrip(b, j);
            int d;
            if (j > W - 3)
            {
                d = dtrip(b, ++wb);
                del(wcount, d, wsr);
            }
            add(wcount, c, wsr);
            if (lb < wb)
            {
                d = dtrip(b, ++lb);
                del(lcount, d, lsr);
            }
            const double tr = __dmul_rn((double)lcount[c], skew[c]);
            lcount[c]++;
            lsr = __dadd_rn(lsr, tr);
            if (tr >= thr2r)
                while (lb < j)
                {
                    d = dtrip(b, ++lb);
                    del(lcount, d, lsr);
                    if (d == c)
                        break;
                }
            // retire the oldest candidate once its start has left the window
            const int t = cd[0].prev;
            if (t != 0 && cd[t].beg <= wb)
            {
                dust_retire(mask, mtop, cd[t].beg, cd[t].end);
                const int p = cd[t].prev;
                cd[0].prev = p;
                cd[p].next = 0;
                cd[t].next = freel;
                freel = t;
            }
            double lsq = lsr;
            if (wsr <= __dmul_rn(lsq, T))
                continue;
            int jp = cd[0].next, lp = 0, x;
            double ms = 0.;
            for (x = lb; x > wb; x--)
            {
                d = dtrip(b, x);
                add(lcount, d, lsr);
                lsq = lsr;
                if (lsq >= __dmul_rn(T, (double)(j - x)))
                {
                    for (; cd[jp].beg >= x; lp = jp, jp = cd[jp].next)
                        if (cd[jp].score > ms)
                            ms = cd[jp].score;
                    if (lsq >= __dmul_rn(ms, (double)(j - x)))
                    {
                        ms = __ddiv_rn(lsq, (double)(j - x));
                        if (cd[lp].beg == x)
                        {
                            cd[lp].end = j;
                            cd[lp].score = ms;
                        }
                        else
                        {
                            const int n = freel;
                            if (n < 0)
                            {
                                nout[r] = -1;  // candidate pool exhausted
                                return;
                            }
                            freel = cd[n].next;
                            cd[n].beg = x;
                            cd[n].end = j;
                            cd[n].score = ms;
                            cd[n].prev = lp;
                            cd[lp].next = n;
                            cd[n].next = jp;
                            cd[jp].prev = n;
                            lp = n;
                        }
                    }
                }
            }
            for (x++; x <= lb; x++)
            {
                d = dtrip(b, x);
                del(lcount, d, lsr);
            }
        }
        int t;
        while ((t = cd[0].prev) != 0)
        {
            dust_retire(mask, mtop, cd[t].beg, cd[t].end);
            const int p = cd[t].prev;
            cd[0].prev = p;
            cd[p].next = 0;
        }
    }
    // keep intervals of more than minlen positions, as [beg, end + 1), in place
    int n = 0;
    for (int k = 1; k < mtop; k += 2)
        if (mask[k + 1] - mask[k] >= minlen)
        {
            const int bg = mask[k], en = mask[k + 1] + 1;
            mask[n++] = bg;
            mask[n++] = en;
        }
    nout[r] = n;
}


// Without -b: a chunk of a read per thread.  A chunk owns the intervals that start in its
// DUST_CHUNK positions.  The window (wb, j] and the run (lb, j] at position j follow from the
// last W bases: wb = j - (W - 2), and lb is the least position at or beyond wb from which no
// triplet is more frequent than the threshold allows (each step moves it just far enough).  A
// candidate that starts at x is made, raised and tested at positions from x to x + W - 2 only, with
// windows that reach back to x - W, against candidates that start at or behind x.  So a scan
// begun W positions before the chunk, which makes candidates from the chunk's first start on
// only, has the same candidates there as the whole read's scan.  The chunk's retired candidates come
// in order of their starts and are merged as the reference merges them; k_dust_merge joins the
// chunks' lists, which merges the same sequence in pieces.
//
// One thread per read (a 105 Mbp block of 10,020 reads) took 91 ms, its longest reads deciding.
// With chunks the bound is divergence: one step in twenty or so walks the window from the run's start
// down to its own (up to W - 2 places, 29 on average), and with the walk as an inner loop nearly every step of a
// warp waited for some lane's (20 ms at any chunk size).  So a lane is either stepping or walking,
// and every turn of the one loop takes each lane one step or one place further.  The walk counts
// the triplets it meets on top of the run's in a field of its own, valid under the walk's tag,
// so that nothing has to be walked back.  A triplet's counts share one shared-memory word
// ([triplet][thread], free of bank conflicts): window, run, walk and tag, 8 bits each (a
// window holds at most 126 triplets).  Triplets come from the 2-bit copy (any one-to-one code of
// a triplet serves, so its bits stay as they are packed), and the walk compares the run's
// integer sum with a table of the thresholds ceil(T n), which is the comparison of doubles it
// stands for.  The worst chunks lie in tandem repeats, where every step walks: hence the short
// chunks, for more warm-up elsewhere (the block takes 14.5 ms with chunks of 512, 12.1 with 256, 11.2
// with 128, 12.0 with 64).
constexpr int DUST_CHUNK = 128;  // interval starts per chunk
constexpr int DT = 128;          // chunks per block

__global__ void __launch_bounds__(DT) k_dust_chunks(DevBlock blk, int W, double T, int thr2,
                                                    const uint32_t* __restrict__ cfirst, unsigned nchunks, int* out,
                                                    int* __restrict__ ccount)
{
    __shared__ unsigned cnt[64][DT];
    __shared__ int thr[DUST_MAXW + 1];  // (double)s >= T * n  <=>  s >= thr[n], for whole s
    for (int n = threadIdx.x; n <= DUST_MAXW; n += DT)
        thr[n] = (int)fmin(ceil(__dmul_rn(T, (double)n)), 1e9);
    __syncthreads();
    const unsigned g = blockIdx.x * DT + threadIdx.x;
    if (g >= nchunks)
        return;
    int lo = 0, hi = blk.nreads - 1;  // the read of this chunk: the last with cfirst <= g
    while (lo < hi)
    {
        const int mid = (lo + hi + 1) >> 1;
        if (cfirst[mid] <= g)
            lo = mid;
        else
            hi = mid - 1;
    }
    const int r = lo;
    const int len = blk.rlen[r] - 2;
    const uint32_t pk0 = PK_BIAS + (uint32_t)blk.boff[r];
    auto trip = [&](int x) {  // the triplet at x
        const uint32_t i = pk0 + (uint32_t)x;
        return (int)(__funnelshift_r(__ldg(blk.pk + (i >> 4)), __ldg(blk.pk + (i >> 4) + 1), 2 * i) & 63u);
    };
    const int b0 = (int)(g - cfirst[r]) * DUST_CHUNK, b1 = min(b0 + DUST_CHUNK, len);
    int* const list = out + blk.boff[r] + 4ll * r + b0;  // [begin, end] pairs, more than 3 apart
    const int js = max(0, b0 - W), je = min(len, b1 + W - 2);
    unsigned* const my = &cnt[0][threadIdx.x];
    for (int e = 0; e < 64; e++)
        my[e * DT] = 0;
    DustCand cd[DUST_MAXW + 1];
    cd[0].beg = -2;
    cd[0].prev = cd[0].next = 0;
    int freel = 0, used = 0, wb = js - 1, lb = js - 1, ws = 0, ls = 0;
    int n = 0, mbeg = -2, mend = -2;  // the list and its open interval
    auto retire = [&](int beg, int end) {
        if (beg < b0 || beg >= b1)
            return;  // another chunk's
        const int c = end + 2;
        if (mend + 1 >= beg)
            mend = max(mend, c);
        else
        {
            if (mbeg >= 0)
            {
                list[n++] = mbeg;
                list[n++] = mend;
            }
            mbeg = beg;
            mend = c;
        }
    };
    int oldest = INT_MAX;  // start of the oldest candidate
    bool full = false;
    int j = js - 1;
    // the walk: its next place, the last place before its end, sum, tag and place among the candidates
    int x = 0, xend = 0, lw = 0, jp = 0, lp = 0;
    unsigned tag = 0;
    double ms = 0.;
    while (true)
    {
        if (x > xend)
        {
            // one place of the walk
            const int d = trip(x);
            const unsigned v = my[d * DT];
            const unsigned wk = (v >> 24) == tag ? (v >> 16) & 0xffu : 0u;
            lw += (int)(((v >> 8) & 0xffu) + wk);
            my[d * DT] = (v & 0xffffu) | ((wk + 1) << 16) | (tag << 24);
            if (lw >= thr[j - x])
            {
                const double lsq = (double)lw;
                for (; cd[jp].beg >= x; lp = jp, jp = cd[jp].next)
                    if (cd[jp].score > ms)
                        ms = cd[jp].score;
                if (lsq >= __dmul_rn(ms, (double)(j - x)))
                {
                    ms = __ddiv_rn(lsq, (double)(j - x));
                    if (cd[lp].beg == x)
                    {
                        cd[lp].end = j;
                        cd[lp].score = ms;
                    }
                    else
                    {
                        int q = freel;
                        if (q)
                            freel = cd[q].next;
                        else if (used < W)
                            q = ++used;
                        else
                        {
                            full = true;  // candidate pool exhausted
                            break;
                        }
                        cd[q].beg = x;
                        cd[q].end = j;
                        cd[q].score = ms;
                        cd[q].prev = lp;
                        cd[lp].next = q;
                        cd[q].next = jp;
                        cd[jp].prev = q;
                        if (jp == 0)
                            oldest = x;
                        lp = q;
                    }
                }
            }
            x--;
        }
        else
        {
            // one step of the scan
            if (++j >= je)
                break;
            const int c = trip(j);
            if (j - js > W - 3)
            {
                const int d = trip(++wb);
                const unsigned v = my[d * DT] - 1u;
                my[d * DT] = v;
                ws -= (int)(v & 0xffu);
            }
            if (lb < wb)
            {
                const int d = trip(++lb);
                const unsigned v = my[d * DT] - 0x100u;
                my[d * DT] = v;
                ls -= (int)((v >> 8) & 0xffu);
            }
            const unsigned v = my[c * DT];
            ws += (int)(v & 0xffu);
            const int tr = (int)((v >> 8) & 0xffu);
            ls += tr;
            my[c * DT] = v + 0x101u;
            if (tr >= thr2)
                while (lb < j)
                {
                    const int d = trip(++lb);
                    const unsigned u = my[d * DT] - 0x100u;
                    my[d * DT] = u;
                    ls -= (int)((u >> 8) & 0xffu);
                    if (d == c)
                        break;
                }
            // retire the oldest candidate once its start has left the window
            if (oldest <= wb)
            {
                const int t = cd[0].prev;
                retire(cd[t].beg, cd[t].end);
                const int q = cd[t].prev;
                cd[0].prev = q;
                cd[q].next = 0;
                cd[t].next = freel;
                freel = t;
                oldest = q ? cd[q].beg : INT_MAX;
            }
            xend = x = max(wb, b0 - 1);
            if ((double)ws > __dmul_rn((double)ls, T))
            {
                x = lb;
                lw = ls;
                jp = cd[0].next;
                lp = 0;
                ms = 0.;
                if (++tag == 256)  // the tags are used up: clear them
                {
                    tag = 1;
                    for (int e = 0; e < 64; e++)
                        my[e * DT] &= 0xffffu;
                }
            }
        }
    }
    for (int t = cd[0].prev; t != 0 && !full; t = cd[t].prev)
        retire(cd[t].beg, cd[t].end);
    if (mbeg >= 0)
    {
        list[n++] = mbeg;
        list[n++] = mend;
    }
    ccount[g] = full ? -1 : n;
}

// A read's chunk lists joined in place: intervals that touch merged, those of more than minlen
// positions kept as [beg, end + 1)
__global__ void __launch_bounds__(DT) k_dust_merge(DevBlock blk, const uint32_t* __restrict__ cfirst,
                                                   const int* __restrict__ ccount, int minlen, int* out,
                                                   int* __restrict__ nout)
{
    const int r = blockIdx.x * DT + threadIdx.x;
    if (r >= blk.nreads)
        return;
    int* const mask = out + blk.boff[r] + 4ll * r;
    int n = 0, beg = -2, end = -2;
    bool full = false;
    auto keep = [&]() {
        if (beg >= 0 && end - beg >= minlen)
        {
            mask[n++] = beg;
            mask[n++] = end + 1;
        }
    };
    for (unsigned g = cfirst[r]; g < cfirst[r + 1]; g++)
    {
        const int* list = mask + (int)(g - cfirst[r]) * DUST_CHUNK;
        const int m = ccount[g];
        full |= m < 0;
        for (int k = 0; k < m; k += 2)
        {
            const int lb = list[k], le = list[k + 1];
            if (end + 1 >= lb)
                end = max(end, le);
            else
            {
                keep();
                beg = lb;
                end = le;
            }
        }
    }
    keep();
    nout[r] = full ? -1 : n;
}

// packs read r's nout[r] ints to dst + off[r] (one warp per read)
__global__ void k_dust_gather(DevBlock blk, const int* __restrict__ out, const int* __restrict__ nout,
                              const int64_t* __restrict__ off, int* __restrict__ dst)
{
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= blk.nreads)
        return;
    const int* src = out + blk.boff[w] + 4 * w;
    for (int j = lane_id(); j < nout[w]; j += 32)
        dst[off[w] + j] = src[j];
}

int launch_dust_gather(const DevBlock& blk, const int* out, const int* nout, const int64_t* off, int* dst,
                       cudaStream_t s)
{
    if (blk.nreads <= 0)
        return 0;
    const int64_t threads = (int64_t)blk.nreads * 32;
    k_dust_gather<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(blk, out, nout, off, dst);
    GD_LAUNCHED(1);
    GD_CUDA(cudaGetLastError());
    return 0;
}

unsigned dust_chunks(const int32_t* rlen, int nreads, uint32_t* cfirst)
{
    unsigned n = 0;
    for (int r = 0; r < nreads; r++)
    {
        cfirst[r] = n;
        n += rlen[r] > 2 ? (unsigned)((rlen[r] - 2 + DUST_CHUNK - 1) / DUST_CHUNK) : 0u;
    }
    cfirst[nreads] = n;
    return n;
}

int launch_dust(const DevBlock& blk, int window, double thresh, int minlen, bool biased, const double* skew,
                const uint32_t* cfirst, unsigned nchunks, int* ccount, int* out, int* nout, cudaStream_t s)
{
    if (blk.nreads <= 0)
        return 0;
    if (window < 3 || window > DUST_MAXW)
    {
        gd_set_error("DUST window %d outside [3, %d]", window, DUST_MAXW);
        return -1;
    }
    if (biased)
        k_dust_read<<<(unsigned)((blk.nreads + 63) / 64), 64, 0, s>>>(blk, window, thresh, 2. * thresh, skew, minlen, out,
                                                                     nout);
    else
    {
        if (nchunks)
            k_dust_chunks<<<(nchunks + DT - 1) / DT, DT, 0, s>>>(blk, window, thresh, (int)std::ceil(2. * thresh),
                                                                 cfirst, nchunks, out, ccount);
        k_dust_merge<<<(unsigned)((blk.nreads + DT - 1) / DT), DT, 0, s>>>(blk, cfirst, ccount, minlen, out, nout);
        GD_LAUNCHED(1);
    }
    GD_LAUNCHED(1);
    GD_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace gd
