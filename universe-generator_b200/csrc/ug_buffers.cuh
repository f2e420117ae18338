// ug_buffers.cuh -- device memory of a batch and of the calls on it, and host pages of results.
#pragma once
#include <cuda_runtime.h>
#include <sys/mman.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <mutex>
#include <thread>
#include <vector>

namespace ug {

// cudaMalloc of the library's own buffers: where there is no memory, the blocks that batches
// keep from finished calls are given back, and it is tried once more.
inline cudaError_t dev_malloc(void** p, size_t bytes);
template <class T>
cudaError_t dev_malloc(T** p, size_t bytes) {
    return dev_malloc((void**)p, bytes);
}

// Device buffers of a batch's finished read-back and frame calls, kept for its next ones
// (which run on the same stream).  A block belongs to one call at a time, so calls of
// several threads on one batch are as independent as with buffers of their own.  A job that
// reads parameters and trajectories in turn allocates nothing from its second pass on.  All
// batches together keep at most kKeep bytes; beyond that a batch gives its longest unused
// blocks back.  The densities of 32 frames of 1024 x 1024 and two observers of 25 k paths
// need 0.9 GB (64.9 ms a call; 71.6 with a bound of 256 MB, which most of it exceeds).
class CallBuffers {
public:
    struct Block {
        void* p;
        size_t n;
    };
    CallBuffers() {
        std::lock_guard<std::mutex> lock(all_mu());
        all().push_back(this);
    }
    ~CallBuffers() {
        {
            std::lock_guard<std::mutex> lock(all_mu());
            all().erase(std::find(all().begin(), all().end(), this));
        }
        drop();
    }
    CallBuffers(const CallBuffers&) = delete;
    // A kept block of about this size, or a new one; p is null when there is no memory.
    Block take(size_t bytes) {
        {
            std::lock_guard<std::mutex> lock(mu_);
            auto best = kept_.end();
            for (auto b = kept_.begin(); b != kept_.end(); ++b)
                if (b->n >= bytes && b->n <= 2 * bytes + (1 << 16) && (best == kept_.end() || b->n < best->n)) best = b;
            if (best != kept_.end()) {
                const Block r = *best;
                kept_.erase(best);
                total() -= r.n;
                return r;
            }
        }
        Block r{nullptr, bytes};
        if (dev_malloc(&r.p, bytes) != cudaSuccess) r.p = nullptr;
        return r;
    }
    // The blocks of a finished call.
    void give(std::vector<Block>& blocks) {
        std::lock_guard<std::mutex> lock(mu_);
        for (const Block& b : blocks) {
            if (b.n > kKeep) {
                cudaFree(b.p);
                continue;
            }
            kept_.push_back(b);
            total() += b.n;
        }
        blocks.clear();
        size_t k = 0;
        for (; k < kept_.size() && total() > kKeep; k++) {
            total() -= kept_[k].n;
            cudaFree(kept_[k].p);
        }
        kept_.erase(kept_.begin(), kept_.begin() + k);
    }
    void drop() {
        std::lock_guard<std::mutex> lock(mu_);
        for (Block& b : kept_) {
            total() -= b.n;
            cudaFree(b.p);
        }
        kept_.clear();
    }
    static void drop_all() {
        std::lock_guard<std::mutex> lock(all_mu());
        for (CallBuffers* c : all()) c->drop();
    }
    static constexpr size_t kKeep = (size_t)1 << 30;

private:
    // every cache of the process (never destroyed: a batch may outlive static objects)
    static std::mutex& all_mu() {
        static std::mutex* m = new std::mutex;
        return *m;
    }
    static std::vector<CallBuffers*>& all() {
        static std::vector<CallBuffers*>* v = new std::vector<CallBuffers*>;
        return *v;
    }
    static std::atomic<size_t>& total() {  // kept by all of them
        static std::atomic<size_t> n{0};
        return n;
    }
    std::mutex mu_;
    std::vector<Block> kept_;  // the longest unused first
};

inline cudaError_t dev_malloc(void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    CallBuffers::drop_all();
    e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation) cudaGetLastError();  // reported here, not at a later launch
    return e;
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

// The buffers of one call: taken from its batch's kept ones and given back at the end, or
// (no cache) the call's own.
class CallScope {
public:
    explicit CallScope(CallBuffers* cache) : cache_(cache ? cache : &own_) {}
    CallScope(const CallScope&) = delete;
    ~CallScope() { cache_->give(blocks_); }
    template <class T>
    T* get(size_t n) {
        const CallBuffers::Block b = cache_->take(std::max<size_t>(n, 1) * sizeof(T));
        if (b.p) blocks_.push_back(b);
        return (T*)b.p;
    }

private:
    CallBuffers own_;
    CallBuffers* cache_;
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
