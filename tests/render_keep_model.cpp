// CPU test of csrc/sms_keep.h against a device of 2 GiB: prints "ok" or the
// first check that fails.
#include "sms_keep.h"

#include <cstdio>
#include <map>

static const size_t kCapacity = (size_t)2 << 30;
static std::map<void *, size_t> g_blocks;
static size_t g_used = 0;
static cudaError_t g_last = cudaSuccess;
static int g_device = 0;

extern "C" cudaError_t cudaMalloc(void **p, size_t bytes) {
    if (g_device == 0) {
        if (g_used + bytes > kCapacity) return g_last = cudaErrorMemoryAllocation;
        g_used += bytes;
    }
    *p = new char;
    g_blocks[*p] = g_device == 0 ? bytes : 0;
    return cudaSuccess;
}
extern "C" cudaError_t cudaFree(void *p) {
    auto it = g_blocks.find(p);
    if (it == g_blocks.end()) { std::printf("freed twice\n"); return cudaErrorInvalidValue; }
    g_used -= it->second;
    g_blocks.erase(it);
    delete static_cast<char *>(p);
    return cudaSuccess;
}
extern "C" cudaError_t cudaMallocHost(void **p, size_t n) { *p = new char[n]; return cudaSuccess; }
extern "C" cudaError_t cudaFreeHost(void *p) { delete[] static_cast<char *>(p); return cudaSuccess; }
extern "C" cudaError_t cudaGetLastError(void) { cudaError_t e = g_last; g_last = cudaSuccess; return e; }
extern "C" cudaError_t cudaGetDevice(int *d) { *d = g_device; return cudaSuccess; }

#define CHECK(x) do { if (!(x)) { std::printf("%d: %s\n", __LINE__, #x); return 1; } } while (0)

int main() {
    using namespace sms;
    const size_t MiB = (size_t)1 << 20;
    {
        RenderKeep a(0), b(0), other(1);
        RenderBuffers r, s, o;
        void *p = nullptr, *q = nullptr;
        // kept: 900 MiB with a, 900 MiB with b, a block on another device
        CHECK(a.take(900 * MiB, r) == cudaSuccess && r.block && r.host);
        CHECK(b.take(900 * MiB, s) == cudaSuccess);
        a.give(r);
        b.give(s);
        g_device = 1;
        CHECK(other.take(700 * MiB, o) == cudaSuccess);
        other.give(o);
        g_device = 0;
        CHECK(!r.block && g_used == 1800 * MiB);
        // the next render takes what is kept
        CHECK(a.take(100 * MiB, r) == cudaSuccess && r.bytes == 900 * MiB && g_used == 1800 * MiB);
        // an allocation that needs it gets the kept block of b, not a's, which is in use
        CHECK(device_malloc(&p, 1000 * MiB) == cudaSuccess && g_used == 1900 * MiB);
        CHECK(cudaGetLastError() == cudaSuccess);
        // one that cannot be had fails as before, its error reported
        CHECK(device_malloc(&q, 1000 * MiB) == cudaErrorMemoryAllocation);
        CHECK(cudaGetLastError() == cudaErrorMemoryAllocation);
        cudaFree(p);
        a.give(r);
        // a render of b that needs it gets a's block
        CHECK(b.take(1500 * MiB, s) == cudaSuccess && g_used == 1500 * MiB);
        b.give(s);   // too large to keep
        CHECK(g_used == 0);
        // a failed take is given back empty
        CHECK(b.take(3000 * MiB, s) == cudaErrorMemoryAllocation && !s.block && s.bytes == 0);
        b.give(s);
        g_device = 1;
        CHECK(other.take(700 * MiB, o) == cudaSuccess && o.bytes == 700 * MiB);   // untouched
        other.give(o);
        g_device = 0;
    }
    CHECK(g_used == 0 && g_blocks.empty());
    std::printf("ok\n");
    return 0;
}
