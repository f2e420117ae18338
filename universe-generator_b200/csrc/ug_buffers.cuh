// ug_buffers.cuh -- device memory of a batch and of the calls on it, and host pages of results.
#pragma once
#include <cuda_runtime.h>
#include <sys/mman.h>

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <thread>
#include <vector>

namespace ug {

// Device blocks of finished read-back and frame calls, kept for the next ones of any batch of
// the process while there is a batch.  A block belongs to one call at a time and comes back
// when that call's work has ended, so calls of several threads, batches and streams are as
// independent as with buffers of their own.  A job that reads parameters and trajectories in
// turn allocates nothing from its second pass on.  At most kKeep bytes are kept, the longest
// unused go first; all go where an allocation of the library finds no memory, and with the
// last batch.  The densities of 32 frames of 1024 x 1024 and two observers of 25 k paths need
// 0.9 GB (64.9 ms a call; 71.6 with a bound of 256 MB, which most of it exceeds).
class CallBuffers {
public:
    struct Block {
        void* p;
        size_t n;
        int dev;
    };
    static constexpr size_t kKeep = (size_t)1 << 30;

    static CallBuffers& get() {  // never destroyed: a batch may outlive static objects
        static CallBuffers* b = new CallBuffers;
        return *b;
    }
    // A kept block of about this size, or a new one; p is null when there is no memory.
    Block take(size_t bytes);
    // The blocks of a finished call.
    void give(std::vector<Block>& blocks) {
        std::lock_guard<std::mutex> lock(mu_);
        for (const Block& b : blocks) {
            if (users_ == 0 || b.n > kKeep) {
                cudaFree(b.p);
                continue;
            }
            kept_.push_back(b);
            bytes_ += b.n;
        }
        blocks.clear();
        size_t k = 0;
        for (; bytes_ > kKeep; k++) {
            bytes_ -= kept_[k].n;
            cudaFree(kept_[k].p);
        }
        kept_.erase(kept_.begin(), kept_.begin() + k);
    }
    void drop() {
        std::lock_guard<std::mutex> lock(mu_);
        free_all();
    }
    // A batch: while there is one, blocks are kept.
    struct User {
        User() {
            std::lock_guard<std::mutex> lock(get().mu_);
            get().users_++;
        }
        ~User() {
            std::lock_guard<std::mutex> lock(get().mu_);
            if (--get().users_ == 0) get().free_all();
        }
        User(const User&) = delete;
    };

private:
    void free_all() {
        for (Block& b : kept_) cudaFree(b.p);
        kept_.clear();
        bytes_ = 0;
    }
    std::mutex mu_;
    std::vector<Block> kept_;  // the longest unused first
    size_t bytes_ = 0;
    int users_ = 0;
};

// cudaMalloc of the library's own buffers: where there is no memory, the blocks kept from
// finished calls are given back, and it is tried once more.
inline cudaError_t dev_malloc(void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    CallBuffers::get().drop();
    e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation) cudaGetLastError();  // reported here, not at a later launch
    return e;
}
template <class T>
cudaError_t dev_malloc(T** p, size_t bytes) {
    return dev_malloc((void**)p, bytes);
}

inline CallBuffers::Block CallBuffers::take(size_t bytes) {
    Block r{nullptr, bytes, 0};
    cudaGetDevice(&r.dev);
    {
        std::lock_guard<std::mutex> lock(mu_);
        auto best = kept_.end();
        for (auto b = kept_.begin(); b != kept_.end(); ++b)
            if (b->dev == r.dev && b->n >= bytes && b->n <= 2 * bytes + (1 << 16) && (best == kept_.end() || b->n < best->n))
                best = b;
        if (best != kept_.end()) {
            r = *best;
            kept_.erase(best);
            bytes_ -= r.n;
            return r;
        }
    }
    if (dev_malloc(&r.p, bytes) != cudaSuccess) r.p = nullptr;
    return r;
}

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
            size_t n = std::max(next_, bytes);
            void* c = nullptr;
            cudaError_t e = chunk(n, &c);
            if (e == cudaErrorMemoryAllocation && n > bytes)  // less than a chunk is left: what is asked
                e = chunk(n = bytes, &c);
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
        const cudaError_t e = dev_malloc(out, bytes);
        if (e == cudaSuccess) chunks_.push_back(*out);
        return e;
    }
    std::vector<void*> chunks_;
    char* cur_ = nullptr;
    size_t left_ = 0, next_ = (size_t)4 << 20;
};

// The buffers of one call.  A batch's call (on the batch's stream) takes them from the kept ones
// and gives them back at its end, after the stream's work (an early return may leave some); a
// call without a batch has its own.
class CallScope {
public:
    CallScope() = default;
    explicit CallScope(cudaStream_t st) : kept_(true), st_(st) {}
    CallScope(const CallScope&) = delete;
    ~CallScope() {
        if (blocks_.empty()) return;
        if (kept_) {
            cudaStreamSynchronize(st_);
            CallBuffers::get().give(blocks_);
        } else {
            for (CallBuffers::Block& b : blocks_) cudaFree(b.p);
        }
    }
    template <class T>
    T* get(size_t n) {
        const size_t bytes = std::max<size_t>(n, 1) * sizeof(T);
        CallBuffers::Block b{nullptr, bytes, 0};
        if (kept_)
            b = CallBuffers::get().take(bytes);
        else if (dev_malloc(&b.p, bytes) != cudaSuccess)
            b.p = nullptr;
        if (b.p) blocks_.push_back(b);
        return (T*)b.p;
    }

private:
    bool kept_ = false;
    cudaStream_t st_ = nullptr;
    std::vector<CallBuffers::Block> blocks_;
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
