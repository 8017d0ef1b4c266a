// gd_staging.cuh -- copies between device memory and pageable host memory through pinned staging.
//
// The driver's own pageable path moves one small piece at a time (105 MB of bases took about 25 ms,
// and results into fresh pages as long again).  STAGE_THREADS host threads take STAGE_CHUNK pieces
// in turn, each with two pinned buffers, so that one piece's host copy (and the page faults of a fresh
// result array) runs beside another's transfer.  Small copies and pinned memory go straight.
// Host code only: it needs the runtime's headers and no kernel.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <exception>
#include <thread>

constexpr size_t STAGE_CHUNK = 2u << 20;
constexpr size_t STAGE_MIN = 4u << 20;  // below this the threads cost what they save
constexpr int STAGE_THREADS = 4;

struct Staging
{
    char* buf = nullptr;  // 2 pieces per thread, pinned
    cudaEvent_t ev[2 * STAGE_THREADS] = {};
};

inline void release(Staging& g)
{
    for (cudaEvent_t e : g.ev)
        if (e)
            cudaEventDestroy(e);
    if (g.buf)
        cudaFreeHost(g.buf);
    g = Staging{};
}

// the pinned buffers and their events; false, and nothing kept, where the host has no room for them
inline bool stage_ready(Staging& g)
{
    if (g.buf)
        return true;
    bool ok = true;
    for (cudaEvent_t& e : g.ev)
        ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    ok = ok && cudaMallocHost((void**)&g.buf, 2 * STAGE_THREADS * STAGE_CHUNK) == cudaSuccess;
    if (!ok)
    {
        release(g);
        cudaGetLastError();  // not the next launch check's to find
    }
    return ok;
}

inline bool is_pageable(const void* p)
{
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess)
    {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// dev <-> host (to_dev), n bytes on stream s.  To the device: pageable host memory may be reused on
// return, as after a pageable cudaMemcpyAsync; pinned memory is read until the stream has passed the copy.
// To the host: complete on return.  Without room for the staging the driver's path is taken.
inline cudaError_t stage_copy(Staging& g, void* dev, void* host, size_t n, bool to_dev, cudaStream_t s)
{
    if (n < STAGE_MIN || !is_pageable(host) || !stage_ready(g))
    {
        const cudaError_t e = cudaMemcpyAsync(to_dev ? dev : host, to_dev ? host : dev, n,
                                              to_dev ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost, s);
        return e != cudaSuccess || to_dev ? e : cudaStreamSynchronize(s);
    }
    int dev_id = 0;
    if (const cudaError_t e = cudaGetDevice(&dev_id); e != cudaSuccess)
        return e;
    cudaError_t errs[STAGE_THREADS] = {};
    auto work = [&](int t) {
        cudaError_t& e = errs[t];
        if ((e = cudaSetDevice(dev_id)) != cudaSuccess)
            return;
        struct
        {
            size_t at = 0, len = 0;  // the piece in flight in this buffer
        } fly[2];
        auto land = [&](int b) {
            if (fly[b].len == 0 || e != cudaSuccess)
                return;
            e = cudaEventSynchronize(g.ev[2 * t + b]);
            if (e == cudaSuccess && !to_dev)
                memcpy((char*)host + fly[b].at, g.buf + (2 * t + b) * STAGE_CHUNK, fly[b].len);
            fly[b].len = 0;
        };
        int b = 0;
        for (size_t at = t * STAGE_CHUNK; at < n && e == cudaSuccess; at += STAGE_THREADS * STAGE_CHUNK, b ^= 1)
        {
            land(b);
            if (e != cudaSuccess)
                return;
            char* const pin = g.buf + (2 * t + b) * STAGE_CHUNK;
            const size_t len = std::min(STAGE_CHUNK, n - at);
            if (to_dev)
            {
                memcpy(pin, (const char*)host + at, len);
                e = cudaMemcpyAsync((char*)dev + at, pin, len, cudaMemcpyHostToDevice, s);
            }
            else
                e = cudaMemcpyAsync(pin, (const char*)dev + at, len, cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess)
                e = cudaEventRecord(g.ev[2 * t + b], s);
            fly[b].at = at;
            fly[b].len = len;
        }
        land(b);
        land(b ^ 1);
    };
    std::thread th[STAGE_THREADS];
    for (int t = 1; t < STAGE_THREADS; t++)
    {
        try
        {
            th[t] = std::thread(work, t);
        }
        catch (const std::exception&)
        {
            work(t);  // no thread to be had: its share here
        }
    }
    work(0);
    for (std::thread& x : th)
        if (x.joinable())
            x.join();
    for (cudaError_t e : errs)
        if (e != cudaSuccess)
        {
            cudaStreamSynchronize(s);  // no transfer of this call may meet the next one's pieces
            return e;
        }
    return cudaSuccess;
}
