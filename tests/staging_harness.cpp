// gd_staging.cuh against a runtime of its own: a stream whose copies run only when something waits for
// them, allocations and copies that fail when they are told to.  Prints a line per failed check.
#include <cerrno>
#include <cstdio>
#include <cstdlib>
#include <dlfcn.h>
#include <functional>
#include <map>
#include <mutex>
#include <pthread.h>
#include <set>
#include <string>
#include <vector>

#include "gd_staging.cuh"

static std::mutex mu;
static std::vector<std::function<void()>> queue_;   // the stream
static std::map<cudaEvent_t, size_t> marks;         // events recorded: the queue's length then
static size_t done;
static std::set<cudaEvent_t> events;
static std::set<void*> pinned;
static bool fail_pin, fail_event, fail_thread;
static int fail_copy = -1, copies, sticky;

static void run_to(size_t n)
{
    for (; done < n; done++)
        queue_[done]();
}

extern "C"
{
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p)
{
    a->type = pinned.count((void*)p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaGetLastError()
{
    const int e = sticky;
    sticky = 0;
    return (cudaError_t)e;
}
cudaError_t cudaMallocHost(void** p, size_t n)
{
    if (fail_pin)
        return (cudaError_t)(sticky = cudaErrorMemoryAllocation);
    *p = malloc(n);
    pinned.insert(*p);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p)
{
    pinned.erase(p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned)
{
    if (fail_event && events.size() == 3)
        return (cudaError_t)(sticky = cudaErrorMemoryAllocation);
    *e = (cudaEvent_t)malloc(1);
    events.insert(*e);
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e)
{
    events.erase(e);
    free(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t)
{
    std::lock_guard<std::mutex> g(mu);
    marks[e] = queue_.size();
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e)
{
    std::lock_guard<std::mutex> g(mu);
    run_to(marks[e]);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t)
{
    std::lock_guard<std::mutex> g(mu);
    run_to(queue_.size());
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind kind, cudaStream_t)
{
    std::lock_guard<std::mutex> g(mu);
    if (copies++ == fail_copy)
        return cudaErrorUnknown;
    // pageable sources are read in the call, as the runtime promises
    bool late = false;
    for (void* p : pinned)
    {
        const char* x = (const char*)(kind == cudaMemcpyHostToDevice ? s : d);
        late = late || (x >= (char*)p && x < (char*)p + 2 * STAGE_THREADS * STAGE_CHUNK);
    }
    if (!late && kind == cudaMemcpyHostToDevice)
    {
        run_to(queue_.size());
        memcpy(d, s, n);
    }
    else
        queue_.push_back([=] { memcpy(d, s, n); });
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d)
{
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int)
{
    return cudaSuccess;
}
// stands before the C library's for std::thread too
int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x)
{
    using Fn = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
    static const Fn real = (Fn)dlsym(RTLD_NEXT, "pthread_create");
    return fail_thread ? EAGAIN : real(t, a, f, x);
}
}

static int bad;

static void check(bool ok, const std::string& what)
{
    if (!ok)
    {
        printf("%s\n", what.c_str());
        bad++;
    }
}

static std::vector<unsigned char> bytes(size_t n, unsigned seed)
{
    std::vector<unsigned char> v(n);
    for (size_t i = 0; i < n; i++)
        v[i] = (unsigned char)((i * 2654435761u + seed) >> 13);
    return v;
}

static void both_ways(Staging& g, size_t n, const std::string& what)
{
    std::vector<unsigned char> src = bytes(n, (unsigned)n), dev(n + 1, 77), back(n + 1, 55), keep = src;
    check(stage_copy(g, dev.data(), src.data(), n, true, nullptr) == cudaSuccess, what + ": up failed");
    std::fill(src.begin(), src.end(), 0);  // pageable memory may be reused on return
    cudaStreamSynchronize(nullptr);
    check(std::equal(keep.begin(), keep.end(), dev.begin()) && dev[n] == 77, what + ": up");
    check(stage_copy(g, dev.data(), back.data(), n, false, nullptr) == cudaSuccess, what + ": down failed");
    check(std::equal(keep.begin(), keep.end(), back.begin()) && back[n] == 55, what + ": down");
    check(cudaGetLastError() == cudaSuccess, what + ": an error is left behind");
}

int main()
{
    const size_t C = STAGE_CHUNK, M = STAGE_MIN, sizes[] = {0,         1,         M - 1,         M,         M + 1,
                                                            3 * C - 1, 3 * C,     3 * C + 1,     4 * C + 5, 7 * C + 1,
                                                            8 * C,     8 * C + 1, 16 * C + 3000, 17 * C - 1};
    for (int mode = 0; mode < 4; mode++)
    {
        fail_pin = mode == 1;
        fail_event = mode == 2;
        fail_thread = mode == 3;
        Staging g;
        for (size_t n : sizes)
            both_ways(g, n, "mode " + std::to_string(mode) + ", " + std::to_string(n) + " bytes");
        const bool staged = mode == 0 || mode == 3;
        check((g.buf != nullptr) == staged && events.size() == (staged ? 2 * STAGE_THREADS : 0),
              "mode " + std::to_string(mode) + ": " + std::to_string(events.size()) + " events");
        release(g);
        check(events.empty() && pinned.empty(), "mode " + std::to_string(mode) + ": not all released");
        fail_pin = fail_event = fail_thread = false;
        both_ways(g, M + 1, "after mode " + std::to_string(mode));  // room again: staged again
        check(g.buf != nullptr, "after mode " + std::to_string(mode) + ": not staged");
        release(g);
    }
    // a copy that fails: the error comes back, and the next call's data are its own
    for (int up = 0; up < 2; up++)
        for (int at = 0; at < 11; at++)
        {
            Staging g;
            std::vector<unsigned char> a = bytes(11 * C, 1), b = bytes(11 * C, 2);
            copies = 0;
            fail_copy = at;
            check(stage_copy(g, a.data(), b.data(), a.size(), up, nullptr) == cudaErrorUnknown, "failed copy unreported");
            fail_copy = -1;
            both_ways(g, 9 * C + 1, "after a failed copy");
            release(g);
        }
    // pinned memory goes straight
    {
        Staging g;
        void* p;
        cudaMallocHost(&p, M + 1);
        std::vector<unsigned char> dev = bytes(M + 1, 3);
        check(stage_copy(g, dev.data(), p, M + 1, false, nullptr) == cudaSuccess && !memcmp(p, dev.data(), M + 1) && !g.buf,
              "pinned");
        cudaFreeHost(p);
    }
    return bad != 0;
}
