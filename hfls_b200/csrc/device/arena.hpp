// Device memory of one owner (a context, or one phase of a set-up), freed
// with it.  A set-up needs some 160 buffers, most of them small, and every
// cudaMalloc and cudaFree is a driver call of 20 to 100 us (6 of the 19 ms
// of the reference problem's whole run, and far more while other processes of
// the machine call the driver too), so buffers under ARENA_OWN bytes share
// chunks of ARENA_CHUNK bytes: about 30 calls instead of 160.  Nothing
// outlives the owner and nothing is shared between owners.
//
// A dry arena allocates nothing (its buffers are null) and only counts what
// the same calls would take.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <utility>
#include <vector>

namespace htf {

class DevArena {
public:
    explicit DevArena(bool dry = false) : dry_(dry) {}
    DevArena(const DevArena &) = delete;
    DevArena &operator=(const DevArena &) = delete;
    ~DevArena() { clear(); }

    cudaError_t get(void **p, size_t bytes) {
        bytes = (std::max<size_t>(bytes, 1) + ALIGN - 1) / ALIGN * ALIGN;
        if (bytes >= ARENA_OWN) return own(p, bytes);
        if (bytes > left_) {
            void *c = nullptr;
            if (own(&c, ARENA_CHUNK, true) != cudaSuccess) {
                cudaGetLastError();                  // no room for a chunk: the buffer alone may still fit
                return own(p, bytes);
            }
            next_ = static_cast<char *>(c);
            left_ = ARENA_CHUNK;
        }
        *p = next_;
        if (!dry_) next_ += bytes;
        left_ -= bytes;
        return cudaSuccess;
    }

    // frees a buffer with memory of its own now; one in a chunk stays until the end
    void release(void *p) {
        for (size_t i = 0; i < bufs_.size(); ++i)
            if (bufs_[i].p == p && !bufs_[i].chunk) {
                cudaFree(p);
                bufs_.erase(bufs_.begin() + i);
                return;
            }
    }

    void swap(DevArena &o) {
        bufs_.swap(o.bufs_);
        std::swap(next_, o.next_);
        std::swap(left_, o.left_);
    }

    bool dry() const { return dry_; }

    size_t bytes() const {
        size_t t = 0;
        for (auto &b : bufs_) t += b.bytes;
        return t;
    }

    void clear() {
        for (auto &b : bufs_)
            if (b.p) cudaFree(b.p);
        bufs_.clear();
        next_ = nullptr;
        left_ = 0;
    }

private:
    static constexpr size_t ALIGN = 512, ARENA_OWN = size_t(2) << 20, ARENA_CHUNK = size_t(8) << 20;
    struct Buf {
        void *p;
        size_t bytes;
        bool chunk;
    };
    cudaError_t own(void **p, size_t bytes, bool chunk = false) {
        const cudaError_t e = dry_ ? cudaSuccess : cudaMalloc(p, bytes);
        if (e == cudaSuccess) bufs_.push_back({*p, bytes, chunk});
        return e;
    }
    std::vector<Buf> bufs_;
    bool dry_;
    char *next_ = nullptr;
    size_t left_ = 0;
};

}  // namespace htf
