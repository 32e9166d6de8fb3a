"""The copies through the pinned ring (emu_hostcopy.cu) on the host, against a
stand-in for the CUDA runtime whose copies are made at once: both directions
at sizes around the threshold and around whole chunks, and calls of the
runtime or of the allocator that fail.  A copy that cannot have the ring goes
the plain way, nothing is thrown, and the next copy asks for the ring again."""
import os
import shutil
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CONTEXT = r"""
#pragma once
#include <cstddef>
#include <cstring>
#include <string>
typedef int cudaError_t;
typedef void* cudaStream_t;
typedef int* cudaEvent_t;
enum { cudaSuccess = 0, cudaErrorMemoryAllocation = 2 };
enum { cudaMemoryTypeUnregistered = 0, cudaMemoryTypeHost = 1 };
enum { cudaMemcpyHostToDevice, cudaMemcpyDeviceToHost, cudaEventDisableTiming };
enum { EMU_OK = 0, EMU_ERR_CUDA = 32 };
struct cudaPointerAttributes { int type; };
extern int fail_event, fail_host, plain_copies, ring_copies, events, rings, throw_new;
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { a->type = cudaMemoryTypeUnregistered; return 0; }
inline cudaError_t cudaGetLastError() { return 0; }
inline const char* cudaGetErrorString(cudaError_t) { return ""; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, int)
{
    if (fail_event > 0 && --fail_event == 0) return 2;
    *e = new int(0);
    events++;
    return 0;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; events--; return 0; }
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { return e ? 0 : 1; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t e) { return e ? 0 : 1; }
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return 0; }
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, int, cudaStream_t)
{
    std::memcpy(d, s, n);
    (n <= (1u << 20) ? ring_copies : plain_copies)++;
    return 0;
}
struct emu_context {
    cudaStream_t stream = nullptr;
    char* ring = nullptr;
    cudaEvent_t ring_event[8] = {};
    std::string err;
};
namespace emu_ctx {
template <class T>
cudaError_t host_malloc(T** p, size_t n)
{
    if (fail_host) { fail_host = 0; return 2; }
    *p = (T*)std::malloc(n);
    rings++;
    return 0;
}
inline cudaError_t host_free(void* p) { std::free(p); rings--; return 0; }
inline int fail(emu_context* c, int code, const std::string& m) { c->err = m; return code; }
int copy_to_host(emu_context*, void*, const void*, size_t);
int copy_to_device(emu_context*, void*, const void*, size_t);
void ring_free(emu_context*);
}
#define CU(call)                                                                                     \
    do {                                                                                             \
        const cudaError_t e_ = (call);                                                               \
        if (e_ != cudaSuccess) return emu_ctx::fail(ctx, EMU_ERR_CUDA, #call);                       \
    } while (0)
"""

MAIN = r"""
#include "emu_hostcopy.cu"
#include <cstdio>
#include <cstdlib>
int fail_event, fail_host, plain_copies, ring_copies, events, rings, throw_new;
void* operator new(size_t n)
{
    if (throw_new > 0 && --throw_new == 0) throw std::bad_alloc();
    void* p = std::malloc(n);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

static const size_t K = 1u << 20;
static int check(emu_context* c, size_t n, bool up, const char* what)
{
    char* a = (char*)std::malloc(n);
    char* b = (char*)std::malloc(n + 64);
    for (size_t i = 0; i < n; i++) a[i] = (char)((i * 2654435761u) >> 13);
    std::memset(b, 0x5a, n + 64);
    const int r = up ? emu_ctx::copy_to_device(c, b, a, n) : emu_ctx::copy_to_host(c, b, a, n);
    int bad = r != 0 || std::memcmp(a, b, n) != 0;
    for (int i = 0; i < 64; i++) bad |= b[n + i] != 0x5a;
    std::free(a);
    std::free(b);
    if (bad) std::printf("%s: %zu bytes, up %d, returned %d\n", what, n, (int)up, r);
    return bad;
}

int main()
{
    int bad = 0;
    for (int up = 0; up < 2; up++) {
        emu_context c;
        const size_t m = 16 * K;
        plain_copies = ring_copies = 0;
        bad |= check(&c, m - 8, up, "below the threshold");
        if (plain_copies != 1 || ring_copies != 0) { std::printf("ring below the threshold\n"); bad = 1; }
        for (size_t n : {m, m + 8, m + K - 8, m + K, m + K + 8, m + 7 * K - 8, m + 8 * K + 8, 40 * K, 41 * K - 8})
            bad |= check(&c, n, up, "ring");
        if (plain_copies != 1) { std::printf("plain above the threshold\n"); bad = 1; }
        emu_ctx::ring_free(&c);
        // an event or the memory cannot be had: the plain way, then the ring
        for (int k = 1; k <= 8; k++) {
            emu_context d;
            fail_event = k;
            plain_copies = 0;
            bad |= check(&d, 20 * K, up, "event fails");
            if (plain_copies != 1 || events != 0 || rings != 0) { std::printf("event %d: half a ring\n", k); bad = 1; }
            bad |= check(&d, 20 * K, up, "after an event failed");
            if (plain_copies != 1) { std::printf("ring not asked for again\n"); bad = 1; }
            emu_ctx::ring_free(&d);
        }
        emu_context d;
        fail_host = 1;
        bad |= check(&d, 20 * K, up, "memory fails");
        bad |= check(&d, 20 * K, up, "after memory failed");
        // an allocation throws
        for (int k = 1; k <= 8; k++) {
            throw_new = k;
            try {
                bad |= check(&d, 20 * K, up, "allocation throws");
            } catch (...) {
                std::printf("an exception left the call (allocation %d)\n", k);
                bad = 1;
            }
            throw_new = 0;
        }
        emu_ctx::ring_free(&d);
        if (events != 0 || rings != 0) { std::printf("left over\n"); bad = 1; }
    }
    std::printf(bad ? "bad\n" : "ok\n");
    return bad;
}
"""


def test_ring_copies_on_the_host(tmp_path):
    shutil.copy(os.path.join(ROOT, "emu_b200", "csrc", "emu_hostcopy.cu"), tmp_path)
    (tmp_path / "emu_context.cuh").write_text(CONTEXT)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "hostcopy"
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", str(tmp_path / "main.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
