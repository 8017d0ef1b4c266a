// gd_verify.cuh -- Compute_Trace_PTS (exact diffs between trace points) on the device.
#pragma once
#include "gd_align.cuh"

namespace gd
{

// One trace-point interval of one .las record: A[ab..ae) against B[bb..be) (block-relative
// read indices; comp selects the complemented B block).
struct Segment
{
    int32_t aread, bread;
    int32_t ab, ae, bb, be;
    int32_t rec, comp;
};

// trace points strictly inside a record's trace of tlen values (align.c:5355-5389): its segments
// but the last
__host__ __device__ inline int trace_inner(int tlen)
{
    return tlen > 3 ? (tlen - 2) / 2 : 0;
}

// The segments of n records: record r's at seg[first[r] ..].  trace holds the trace bytes from
// offset tlo on.  *R (preset 0) becomes the largest M + N + 8 of a segment; a record whose trace
// runs past its end fails in st.
int launch_trace_segments(const OutRec* recs, int64_t n, const int64_t* first, const uint8_t* trace, uint64_t tlo,
                          int tspace, int tbytes, int afirst, int bfirst, Segment* seg, unsigned* R, DevStatus* st,
                          cudaStream_t s);

// *odd (preset 0) becomes 1 when a read of the block holds a byte beyond 3, which the 2-bit copy loses
int launch_block_plain(const DevBlock& b, unsigned* odd, cudaStream_t s);

// The distance of every segment added to its record's diffs; the segments that outgrow the
// kernel's bands, and all of them where a block's *odd (A's, B's, C's, on the device) is not 0, are
// listed (*nlist preset 0) for launch_trace_pts_list, which compares bytes.
int launch_trace_pts(const DevBlock& A, const DevBlock& B, const DevBlock& C, const Segment* seg, int64_t nseg,
                     int* diffs, unsigned* list, unsigned* nlist, const unsigned* const odd[3], cudaStream_t s);

// The listed segments with bands of any width: threads need 3 * (2R + 1) ints of scratch each,
// R >= segment M + N + 4.
int launch_trace_pts_list(const DevBlock& A, const DevBlock& B, const DevBlock& C, const Segment* seg,
                          const unsigned* list, unsigned nlist, int* scratch, int R, int nthreads, int* diffs,
                          DevStatus* st, cudaStream_t s);

}  // namespace gd
