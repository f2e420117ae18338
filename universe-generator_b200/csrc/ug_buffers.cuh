// ug_buffers.cuh -- device memory of a batch and of the calls on it, and host pages of results.
#pragma once
#include <cuda_runtime.h>
#include <sys/mman.h>

#include <algorithm>
#include <cstdint>
#include <thread>
#include <vector>

namespace ug {

// A batch's fixed buffers, carved from chunks: a cudaMalloc and its cudaFree take 0.3 to
// 0.6 ms together and a universe has about thirty buffers (creating, running and releasing
// a 20 k candidate job: 6.3 -> 3.7 ms).  The first chunk is about what the universes
// take (2 to 64 MiB: a small universe does not map what it does not need), later ones
// double.  Freed with the batch.
class Arena {
public:
    ~Arena() {
        for (void* c : chunks_) cudaFree(c);
    }
    // Size of the first chunk: about what will be taken.
    void expect(size_t bytes) { next_ = std::min(kMost, std::max<size_t>((size_t)2 << 20, bytes)); }
    cudaError_t take(size_t bytes, void** out) {
        bytes = (std::max<size_t>(bytes, 1) + 255) / 256 * 256;
        if (bytes > kMost / 4) return chunk(bytes, out);
        if (bytes > left_) {
            const size_t n = std::max(next_, bytes);
            void* c = nullptr;
            const cudaError_t e = chunk(n, &c);
            if (e != cudaSuccess) return e;
            cur_ = (char*)c;
            left_ = n;
            next_ = std::min(2 * n, kMost);
        }
        *out = cur_;
        cur_ += bytes;
        left_ -= bytes;
        return cudaSuccess;
    }

private:
    static constexpr size_t kMost = (size_t)64 << 20;
    cudaError_t chunk(size_t bytes, void** out) {
        const cudaError_t e = cudaMalloc(out, bytes);
        if (e == cudaSuccess) chunks_.push_back(*out);
        return e;
    }
    std::vector<void*> chunks_;
    char* cur_ = nullptr;
    size_t left_ = 0, next_ = (size_t)4 << 20;
};

// Device buffers of a read-back or frame call, kept by its batch for the next call on it
// (which runs on the same stream).  A call's buffers are taken with get(); end() keeps them
// and frees what the call did not use, so the cache never holds more than one call needs.
class CallBuffers {
public:
    ~CallBuffers() {
        for (Block& b : blocks_) cudaFree(b.p);
    }
    void* get(size_t bytes) {
        bytes = std::max<size_t>(bytes, 1);
        Block* best = nullptr;
        for (Block& b : blocks_)
            if (!b.used && b.n >= bytes && b.n <= 2 * bytes + (1 << 16) && (!best || b.n < best->n)) best = &b;
        if (!best) {
            void* p = nullptr;
            if (cudaMalloc(&p, bytes) != cudaSuccess) {  // make room: drop what this call does not hold
                cudaGetLastError();
                drop();
                if (cudaMalloc(&p, bytes) != cudaSuccess) return nullptr;
            }
            blocks_.push_back(Block{p, bytes, false});
            best = &blocks_.back();
        }
        best->used = true;
        return best->p;
    }
    void end() {
        drop();
        for (Block& b : blocks_) b.used = false;
    }

private:
    struct Block {
        void* p;
        size_t n;
        bool used;
    };
    void drop() {
        size_t k = 0;
        for (Block& b : blocks_) {
            if (b.used)
                blocks_[k++] = b;
            else
                cudaFree(b.p);
        }
        blocks_.resize(k);
    }
    std::vector<Block> blocks_;
};
struct CallScope {
    CallBuffers& b;
    ~CallScope() { b.end(); }
};

// Backs the pages of a host result with memory while the GPU computes it: a copy into fresh
// pages is bound by their faults, one at a time (268 MB: 55 to 68 ms, into touched pages 17
// ms).  Contents are kept; without the call (older kernels) the copy faults as before.
class PagesAhead {
public:
    PagesAhead() = default;
    ~PagesAhead() { wait(); }
    void add(void* p, size_t bytes) {
#ifdef MADV_POPULATE_WRITE
        if (!p || bytes < ((size_t)4 << 20)) return;
        const uintptr_t page = 4096, a = ((uintptr_t)p + page - 1) / page * page, e = ((uintptr_t)p + bytes) / page * page;
        const size_t n = std::min<size_t>(8, (e - a) >> 22);
        if (n == 0) return;
        const size_t part = ((e - a) / n + page - 1) / page * page;
        for (size_t i = 0; i < n; i++) {
            const uintptr_t b = a + i * part, m = b < e ? std::min<size_t>(part, e - b) : 0;
            if (!m) break;
            try {
                threads_.emplace_back([b, m] { madvise((void*)b, m, MADV_POPULATE_WRITE); });
            } catch (...) {  // no thread to be had: the copy faults instead
                return;
            }
        }
#else
        (void)p;
        (void)bytes;
#endif
    }
    void wait() {
        for (std::thread& t : threads_) t.join();
        threads_.clear();
    }

private:
    std::vector<std::thread> threads_;
};

}  // namespace ug
