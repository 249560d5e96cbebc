// Page-locked host buffers: the pool a codec's readers share, and the growing
// buffer each reader has from it.
#pragma once

#include <cuda_runtime_api.h>

#include <cstddef>
#include <cstdint>
#include <cstring>
#include <memory>
#include <mutex>
#include <utility>

namespace frt {

// Page-locked host buffers that a codec's readers hand on to the next reader:
// locking a reader's 16-32 MB took 4 ms each time, more than reading a 25 MB
// file through it.  At most MAX_BUFFERS of at most MAX_BYTES are kept, the
// largest of those given; the rest is released at once, and all of them when a
// buffer cannot be had otherwise, or the codec and its last reader are gone.
class PinnedPool {
  public:
    static constexpr size_t MAX_BUFFERS = 2, MAX_BYTES = 64u << 20;

    ~PinnedPool() { clear(); }

    // A kept buffer of at least `want` bytes (the smallest), or null.
    uint8_t *take(size_t want, size_t *cap)
    {
        std::lock_guard<std::mutex> lk(mu);
        Buffer *best = nullptr;
        for (Buffer &b : kept)
            if (b.p && b.cap >= want && (!best || b.cap < best->cap)) best = &b;
        if (!best) return nullptr;
        *cap = best->cap;
        return std::exchange(best->p, nullptr);
    }

    // Keeps p, in the place of the smallest where there is none and p is
    // larger, or releases it.  Nothing may be using it any more.
    void give(uint8_t *p, size_t cap)
    {
        if (!p) return;
        if (cap <= MAX_BYTES) {
            std::lock_guard<std::mutex> lk(mu);
            Buffer *least = nullptr;
            for (Buffer &b : kept)
                if (!least || (least->p && (!b.p || b.cap < least->cap))) least = &b;
            if (!least->p || least->cap < cap) {
                std::swap(p, least->p);
                least->cap = cap;
            }
        }
        if (p) cudaFreeHost(p);
    }

    // Releases what is kept.
    void clear()
    {
        std::lock_guard<std::mutex> lk(mu);
        for (Buffer &b : kept)
            if (b.p) cudaFreeHost(std::exchange(b.p, nullptr));
    }

  private:
    struct Buffer {
        uint8_t *p = nullptr;
        size_t cap = 0;
    };
    std::mutex mu;
    Buffer kept[MAX_BUFFERS];
};

// Host bytes in page-locked memory, so H2D copies run at full link speed; from
// the codec's pool, and back to it where no copy can still be reading them.
struct PinnedBytes {
    std::shared_ptr<PinnedPool> pool;
    uint8_t *p = nullptr;
    size_t n = 0, cap = 0;
    bool idle = true; // no copy in flight
    ~PinnedBytes() { drop(); }
    void drop()
    {
        if (p && pool && idle) pool->give(p, cap);
        else if (p) cudaFreeHost(p);
        p = nullptr;
    }
    bool reserve(size_t want)
    {
        if (want <= cap) return true;
        size_t nc = cap ? cap : 1 << 20;
        while (nc < want) nc *= 2;
        uint8_t *q = pool ? pool->take(want, &nc) : nullptr;
        if (!q && !lock(&q, nc)) {
            if (!pool) return false;
            pool->clear(); // what is kept may be what is missing
            if (!lock(&q, nc)) return false;
        }
        if (n) memcpy(q, p, n);
        drop();
        p = q;
        cap = nc;
        return true;
    }
    bool resize(size_t m)
    {
        if (!reserve(m)) return false;
        n = m;
        return true;
    }

  private:
    static bool lock(uint8_t **q, size_t bytes)
    {
        if (cudaMallocHost((void **)q, bytes) == cudaSuccess) return true;
        cudaGetLastError();
        *q = nullptr;
        return false;
    }
};

} // namespace frt
