// sms_keep.h -- render buffers that a context keeps between renders, and device
// allocation that gives them back when memory runs out.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <mutex>
#include <vector>

#include <cuda_runtime.h>

namespace sms {

// Buffers of one render call, owned by the caller between take and give: a
// device block and two words of pinned host memory.
struct RenderBuffers {
    char *block = nullptr;
    size_t bytes = 0;
    uint32_t *host = nullptr;
};

class RenderKeep;

// Every context's kept buffers, by device.
struct RenderKeeps {
    std::mutex mutex;
    std::vector<RenderKeep *> all;
};
inline RenderKeeps &render_keeps() {
    static RenderKeeps *k = new RenderKeeps;   // outlives every context
    return *k;
}

// A render's path state (643 MB for the default wavefront with SMS queries) and
// its pinned words took 0.8 ms to allocate and free, as long as a small image
// takes to render; larger blocks are not kept.
constexpr size_t kRenderKeepBytes = (size_t)1 << 30;

// cudaMalloc on the current device; when it is out of memory, the blocks that
// contexts keep on that device are freed and it is tried once more.
inline cudaError_t device_malloc(void **p, size_t bytes);

// The buffers a context keeps.  Several threads may take at once: the first one
// gets what is kept.
class RenderKeep {
  public:
    explicit RenderKeep(int device) : device_(device) {
        std::lock_guard<std::mutex> lock(render_keeps().mutex);
        render_keeps().all.push_back(this);
    }
    ~RenderKeep() {
        {
            std::lock_guard<std::mutex> lock(render_keeps().mutex);
            auto &all = render_keeps().all;
            all.erase(std::remove(all.begin(), all.end(), this), all.end());
        }
        free_block();
        if (kept_.host) cudaFreeHost(kept_.host);
    }
    RenderKeep(const RenderKeep &) = delete;
    RenderKeep &operator=(const RenderKeep &) = delete;

    int device() const { return device_; }

    // A block of at least `bytes`; `out` goes back through give() on failure too.
    cudaError_t take(size_t bytes, RenderBuffers &out) {
        {
            std::lock_guard<std::mutex> lock(mutex_);
            out = kept_;
            kept_ = RenderBuffers{};
        }
        cudaError_t e = cudaSuccess;
        if (out.bytes < bytes) {
            if (out.block) cudaFree(out.block);
            out.block = nullptr;
            out.bytes = 0;
            void *p = nullptr;
            e = device_malloc(&p, bytes);
            if (e == cudaSuccess) {
                out.block = static_cast<char *>(p);
                out.bytes = bytes;
            }
        }
        if (e == cudaSuccess && !out.host)
            e = cudaMallocHost(reinterpret_cast<void **>(&out.host), 2 * sizeof(uint32_t));
        return e;
    }

    // The larger block stays.
    void give(RenderBuffers &buf) {
        if (buf.bytes > kRenderKeepBytes) {
            cudaFree(buf.block);
            buf.block = nullptr;
            buf.bytes = 0;
        }
        {
            std::lock_guard<std::mutex> lock(mutex_);
            if (buf.bytes >= kept_.bytes) std::swap(buf, kept_);
        }
        if (buf.block) cudaFree(buf.block);
        if (buf.host) cudaFreeHost(buf.host);
        buf = RenderBuffers{};
    }

    // Frees the kept device block; whether there was one.
    bool free_block() {
        char *block;
        {
            std::lock_guard<std::mutex> lock(mutex_);
            block = kept_.block;
            kept_.block = nullptr;
            kept_.bytes = 0;
        }
        if (block) cudaFree(block);
        return block != nullptr;
    }

  private:
    const int device_;
    std::mutex mutex_;
    RenderBuffers kept_;
};

inline cudaError_t device_malloc(void **p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaErrorMemoryAllocation) return e;
    int device = 0;
    bool freed = false;
    if (cudaGetDevice(&device) == cudaSuccess) {
        std::lock_guard<std::mutex> lock(render_keeps().mutex);
        for (RenderKeep *k : render_keeps().all)
            if (k->device() == device) freed = k->free_block() || freed;
    }
    if (!freed) return e;
    cudaGetLastError();   // the first attempt's error is not the caller's
    return cudaMalloc(p, bytes);
}

}  // namespace sms
