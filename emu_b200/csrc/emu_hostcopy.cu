// emu_hostcopy.cu -- copies between device memory and the caller's host
// memory, which is pageable unless the caller pinned it.
//
// A copy to fresh pageable memory (numpy's) is bound by the host: one thread
// takes the page faults and moves the bytes out of the driver's staging buffer
// (219 MB in 46.5 ms, 4.7 GB/s, where the link carries 55).  Large copies go
// through a pinned ring of the context in chunks, and a few threads move the
// chunks between the ring and the caller's memory while the next ones cross
// the link: 15 ms (six or eight threads 14-15, chunks of 2 MB 17; threads
// woken by a condition variable for each chunk 18).
#include "emu_context.cuh"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <exception>
#include <iterator>
#include <memory>
#include <new>
#include <thread>
#include <vector>

namespace {

constexpr size_t kChunk = (size_t)1 << 20;
constexpr int kSlots = 8;
// below this memory is mostly reused by the allocator, its pages in place, and
// the plain copy is as fast (8 MB: 0.5 against 0.8 ms; fresh, 2.2 against 1.5)
constexpr size_t kStagedMin = (size_t)16 << 20;
constexpr int kWorkers = 4;

bool is_pageable(const void* p)
{
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// the ring, whole or not at all (a copy then goes the plain way; the next one
// asks again)
bool ring_ready(emu_context* ctx)
{
    if (ctx->ring) return true;
    for (auto& e : ctx->ring_event)
        if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) e = nullptr;
    bool ok = std::all_of(std::begin(ctx->ring_event), std::end(ctx->ring_event), [](cudaEvent_t e) { return e; });
    ok = ok && emu_ctx::host_malloc(&ctx->ring, kChunk * kSlots) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        ctx->ring = nullptr;
        emu_ctx::ring_free(ctx);
    }
    return ok;
}

// Chunks handed out in order; done[i]: chunk i has been moved.  The workers
// poll (a chunk takes a fraction of a millisecond; waking a sleeping thread
// for each cost as much).
struct Work {
    std::atomic<long long> ready{0}, next{0};
    std::atomic<bool> stop{false};
    long long total = 0;
    std::unique_ptr<std::atomic<char>[]> done;
    bool start(long long n)
    {
        total = n;
        done.reset(new (std::nothrow) std::atomic<char>[(size_t)n]);
        for (long long i = 0; done && i < n; i++) done[i].store(0, std::memory_order_relaxed);
        return done != nullptr;
    }
    void wait(long long i) const
    {
        while (!done[i].load(std::memory_order_acquire)) std::this_thread::yield();
    }
};

// a worker: takes the next chunk and moves it once it is ready
template <class Move>
void work_loop(Work& w, Move move)
{
    for (;;) {
        const long long i = w.next.fetch_add(1, std::memory_order_relaxed);
        if (i >= w.total) return;
        while (w.ready.load(std::memory_order_acquire) <= i) {
            if (w.stop.load(std::memory_order_relaxed)) return;
            std::this_thread::yield();
        }
        move(i);
        w.done[i].store(1, std::memory_order_release);
    }
}

struct Workers {
    Work& w;
    std::vector<std::thread> t;
    ~Workers()
    {
        w.stop.store(true);
        for (auto& x : t) x.join();
    }
};

// start the workers; false when not one could be started (nothing is thrown
// through the C interface)
template <class Move>
bool start(Workers& ws, Move move)
{
    const unsigned hc = std::max(2u, std::thread::hardware_concurrency());
    const int n = (int)std::min<unsigned>(kWorkers, hc / 2);
    try {
        ws.t.reserve(n);
        for (int i = 0; i < n; i++) ws.t.emplace_back([&ws, move] { work_loop(ws.w, move); });
    } catch (const std::exception&) {
    }
    return !ws.t.empty();
}

}  // namespace

void emu_ctx::ring_free(emu_context* ctx)
{
    if (ctx->ring) host_free(ctx->ring);
    ctx->ring = nullptr;
    for (auto& e : ctx->ring_event)
        if (e) {
            cudaEventDestroy(e);
            e = nullptr;
        }
}

int emu_ctx::copy_to_host(emu_context* ctx, void* dst, const void* src, size_t bytes)
{
    cudaStream_t st = ctx->stream;
    auto plain = [&]() -> int {
        CU(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st));
        CU(cudaStreamSynchronize(st));
        return EMU_OK;
    };
    if (bytes < kStagedMin || !is_pageable(dst) || !ring_ready(ctx)) return plain();
    int r;
    char* const d = static_cast<char*>(dst);
    const char* const s = static_cast<const char*>(src);
    const long long n = (long long)((bytes + kChunk - 1) / kChunk);
    auto size = [=](long long i) { return std::min(kChunk, bytes - (size_t)i * kChunk); };
    Work w;
    if (!w.start(n)) return plain();
    char* const ring = ctx->ring;
    Workers ws{w, {}};
    auto issue = [&](long long i) -> int {
        CU(cudaMemcpyAsync(ring + (i % kSlots) * kChunk, s + i * kChunk, size(i), cudaMemcpyDeviceToHost, st));
        CU(cudaEventRecord(ctx->ring_event[i % kSlots], st));
        return EMU_OK;
    };
    for (long long i = 0; i < std::min<long long>(n, kSlots); i++)
        if ((r = issue(i))) return r;
    // (the workers poll: none while the stream still works)
    CU(cudaEventSynchronize(ctx->ring_event[0]));
    if (!start(ws, [=](long long i) { std::memcpy(d + i * kChunk, ring + (i % kSlots) * kChunk, size(i)); })) return plain();
    for (long long i = 0; i < n; i++) {
        CU(cudaEventSynchronize(ctx->ring_event[i % kSlots]));
        w.ready.store(i + 1, std::memory_order_release);
        // the slot of the chunk before this one is refilled when it is moved
        const long long f = i - kSlots / 2;
        if (f >= 0 && f + kSlots < n) {
            w.wait(f);
            if ((r = issue(f + kSlots))) return r;
        }
    }
    for (long long i = std::max<long long>(0, n - kSlots); i < n; i++) w.wait(i);
    return EMU_OK;
}

int emu_ctx::copy_to_device(emu_context* ctx, void* dst, const void* src, size_t bytes)
{
    cudaStream_t st = ctx->stream;
    auto plain = [&]() -> int {
        CU(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st));
        CU(cudaStreamSynchronize(st));
        return EMU_OK;
    };
    if (bytes < kStagedMin || !is_pageable(src) || !ring_ready(ctx)) return plain();
    char* const d = static_cast<char*>(dst);
    const char* const s = static_cast<const char*>(src);
    const long long n = (long long)((bytes + kChunk - 1) / kChunk);
    auto size = [=](long long i) { return std::min(kChunk, bytes - (size_t)i * kChunk); };
    Work w;
    if (!w.start(n)) return plain();
    char* const ring = ctx->ring;
    // (the workers poll: none while the stream still works)
    CU(cudaStreamSynchronize(st));
    Workers ws{w, {}};
    if (!start(ws, [=](long long i) { std::memcpy(ring + (i % kSlots) * kChunk, s + i * kChunk, size(i)); })) return plain();
    // chunk i is handed out (its slot's last copy has completed) kSlots / 2
    // chunks before it is copied
    constexpr long long kLag = kSlots / 2;
    for (long long i = 0; i < n + kLag; i++) {
        if (i < n) {
            if (i >= kSlots) CU(cudaEventSynchronize(ctx->ring_event[i % kSlots]));
            w.ready.store(i + 1, std::memory_order_release);
        }
        const long long c = i - kLag;
        if (c < 0) continue;
        w.wait(c);
        CU(cudaMemcpyAsync(d + c * kChunk, ring + (c % kSlots) * kChunk, size(c), cudaMemcpyHostToDevice, st));
        CU(cudaEventRecord(ctx->ring_event[c % kSlots], st));
    }
    CU(cudaStreamSynchronize(st));
    return EMU_OK;
}
