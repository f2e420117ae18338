"""Device memory of batches and calls (ug_buffers.cuh) on a stand-in for the CUDA runtime:
host memory with a limit, which counts allocations and checks that blocks are whole."""

import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "universe-generator_b200", "csrc")

RUNTIME = r"""
#pragma once
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <cstdlib>
#include <map>
#include <mutex>
enum cudaError_t { cudaSuccess = 0, cudaErrorMemoryAllocation = 2 };
inline std::mutex g_mu;
inline std::map<void*, size_t> g_live;
inline size_t g_used = 0, g_limit = SIZE_MAX, g_mallocs = 0, g_frees = 0;
inline cudaError_t cudaMalloc(void** p, size_t n) {
    std::lock_guard<std::mutex> lock(g_mu);
    if (n > g_limit - g_used) return cudaErrorMemoryAllocation;
    *p = malloc(16);  // never touched: sizes are what counts
    g_live[*p] = n;
    g_used += n;
    g_mallocs++;
    return cudaSuccess;
}
inline cudaError_t cudaFree(void* p) {
    if (!p) return cudaSuccess;
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_live.count(p)) abort();  // not allocated, or freed twice
    g_used -= g_live[p];
    g_live.erase(p);
    free(p);
    g_frees++;
    return cudaSuccess;
}
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
using cudaStream_t = struct Stream*;
inline int g_device = 0;
inline std::atomic<size_t> g_waits{0};
inline cudaError_t cudaGetDevice(int* d) { *d = g_device; return cudaSuccess; }
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { g_waits++; return cudaSuccess; }
"""

PROLOGUE = r"""
#include <cstdio>
#include <cstdlib>
#include <set>
#include "ug_buffers.cuh"
using namespace ug;
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); exit(1); } } while (0)
constexpr size_t MB = (size_t)1 << 20;
"""

PROGRAMS = {
    # calls of several threads and batches never hold the same block
    "threads": r"""
int main() {
    {
        CallBuffers::User batch[2];
        std::mutex mu;
        std::set<void*> held;
        auto work = [&](unsigned seed) {
            for (int i = 0; i < 3000; i++) {
                CallScope s((cudaStream_t) nullptr);
                char* p[3];
                for (auto& q : p) {
                    q = s.get<char>((1 + rand_r(&seed) % 5) * MB);
                    CHECK(q);
                    std::lock_guard<std::mutex> lock(mu);
                    CHECK(held.insert(q).second);
                }
                std::lock_guard<std::mutex> lock(mu);
                for (auto q : p) held.erase(q);
            }
        };
        std::vector<std::thread> t;
        for (unsigned k = 0; k < 8; k++) t.emplace_back(work, k);
        for (auto& x : t) x.join();
    }
    CHECK(g_live.empty());
}
""",
    # calls of different kinds in turn allocate nothing once each has run; what is kept is bounded
    # and goes with the last batch; a call's stream is waited for before its blocks come back
    "in_turn": r"""
int main() {
    auto params = [&] { CallScope s((cudaStream_t) nullptr); s.get<char>(MB); s.get<char>(24 * MB); s.get<char>(24 * MB); s.get<char>(12 * MB); };
    auto positions = [&] { CallScope s((cudaStream_t) nullptr); s.get<char>(100 * MB); };
    params();
    CHECK(g_live.empty());  // no batch
    {
        CallBuffers::User batch;
        {
            CallBuffers::User other;
            params(), positions();
            const size_t n = g_mallocs, f = g_frees, w = g_waits;
            for (int i = 0; i < 4; i++) params(), positions();
            CHECK(g_mallocs == n && g_frees == f && g_waits == w + 8);
        }
        CHECK(g_used == 161 * MB);
        for (size_t k = 1; k < 160; k++) {
            { CallScope s((cudaStream_t) nullptr); s.get<char>(k * 7 * MB); s.get<char>(k * 3 * MB); }
            CHECK(g_used <= CallBuffers::kKeep);
        }
        { CallScope s((cudaStream_t) nullptr); s.get<char>(CallBuffers::kKeep + 1); }
        CHECK(g_used <= CallBuffers::kKeep && g_used > 0);
        { CallScope own; CHECK(own.get<char>(MB)); }
    }
    CHECK(g_live.empty());
}
""",
    # a block stays on its device
    "devices": r"""
int main() {
    CallBuffers::User batch;
    { CallScope s((cudaStream_t) nullptr); s.get<char>(8 * MB); }
    g_device = 1;
    { CallScope s((cudaStream_t) nullptr); s.get<char>(8 * MB); }
    CHECK(g_mallocs == 2);
    g_device = 0;
    { CallScope s((cudaStream_t) nullptr); s.get<char>(8 * MB); }
    CHECK(g_mallocs == 2);
}
""",
    # what is kept makes room for an allocation that would fail; what calls hold does not
    "room": r"""
int main() {
    {
        CallBuffers::User batch;
        g_limit = 300 * MB;
        CallScope held((cudaStream_t) nullptr);
        CHECK(held.get<char>(80 * MB));
        { CallScope s((cudaStream_t) nullptr); s.get<char>(100 * MB); s.get<char>(40 * MB); }
        CHECK(g_used == 220 * MB);
        int64_t* p = nullptr;
        CHECK(dev_malloc(&p, 200 * MB) == cudaSuccess && g_used == 280 * MB);
        Arena arena;
        void* q = nullptr;
        CHECK(arena.take(100 * MB, &q) != cudaSuccess && !held.get<char>(100 * MB));
        cudaFree(p);
        { CallScope s((cudaStream_t) nullptr); s.get<char>(200 * MB); }
        CHECK(arena.take(100 * MB, &q) == cudaSuccess && g_used == 180 * MB);
    }
    CHECK(g_live.empty());
}
""",
    # memory for what is asked but not for a whole chunk
    "chunk": r"""
int main() {
    {
        Arena arena;
        arena.expect(32 * MB);
        g_limit = 50 * MB;
        void* p = nullptr;
        CHECK(arena.take(10 * MB, &p) == cudaSuccess && g_used == 32 * MB);
        for (int i = 0; i < 3; i++) CHECK(arena.take(10 * MB, &p) == cudaSuccess);
        CHECK(g_used == 42 * MB && arena.take(10 * MB, &p) == cudaErrorMemoryAllocation);
        CHECK(arena.take(8 * MB, &p) == cudaSuccess);
    }
    CHECK(g_live.empty());
}
""",
    # a scarce device: several threads' calls make room for one another and never lock up
    "room_threads": r"""
int main() {
    {
        CallBuffers::User batch;
        g_limit = 4 * 12 * MB;
        auto work = [&](unsigned seed) {
            for (int i = 0; i < 2000; i++) {
                CallScope s((cudaStream_t) nullptr);
                s.get<char>((1 + rand_r(&seed) % 6) * MB);
                s.get<char>((1 + rand_r(&seed) % 6) * MB);
            }
        };
        std::vector<std::thread> t;
        for (unsigned k = 0; k < 4; k++) t.emplace_back(work, k);
        for (auto& x : t) x.join();
    }
    CHECK(g_live.empty());
}
""",
}


@pytest.mark.parametrize("name", PROGRAMS)
def test_program(name, tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    src = tmp_path / (name + ".cpp")
    src.write_text(PROLOGUE + PROGRAMS[name])
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(tmp_path), "-I", CSRC, "-o", tmp_path / name, src],
                   check=True)
    r = subprocess.run([tmp_path / name], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
