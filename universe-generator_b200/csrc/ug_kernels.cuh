// ug_kernels.cuh -- declarations shared by the round-pipeline kernels and
// the host runtime.
#pragma once
#include "ug_device.cuh"

namespace ug {

constexpr int kMaxUni = 1024;

// Work decomposition of one round across all universes (device resident).
struct RoundInfo {
    int32_t n_uni;
    int32_t total_tiles;
    int32_t total_surv;
    int32_t compact_done;
    int32_t any_active;
    int32_t mixed_ok;      // universes in the mixed prefilter this round
    int32_t gemm_next;     // k_surv_gemm: product tiles handed out so far
    int32_t pad1;
    int32_t total_gray;
    int32_t t64_next;      // k_test64: tiles of 32 candidates handed out so far
    int32_t tile_next;     // mixed prefilter: tiles handed out beyond the first gridDim.x
    int32_t confl_next;    // k_conflicts: survivors handed out so far
    int32_t total_sev;     // k_surv_gemm warp tiles
    int32_t total_spt;     // survivor timesteps (k_surv_hash / k_commit items)
    int32_t tile_off[kMaxUni + 1];   // prefilter tiles: first tile of the i-th universe in tile order
    int32_t tile_uni[kMaxUni];       // the universe at position i of the tile order
    int32_t tile_full[kMaxUni];      // universe u: tiles of kTile candidates, then ...
    int32_t tile_rows[kMaxUni];      // ... tiles of this many (32, 64 or kTile)
    int32_t surv_off[kMaxUni + 1];
    int32_t surv_off_o[kMaxUni + 1];  // survivor offsets of the universes in tile order
    int32_t sev_off[kMaxUni + 1];
    int32_t sev_off_o[kMaxUni + 1];   // product tile offsets of the universes in tile order
    int32_t spt_off[kMaxUni + 1];
};

// Term k of the survivor product: sin term of frequency b at k = kseq_s(b),
// its cos term (even b) at kseq_s(b) + 1.
__host__ __device__ __forceinline__ int kseq_s(int b) { return (b - 2) + ((b - 1) >> 1); }
__host__ __device__ __forceinline__ int kseq_len(int F) { return kseq_s(F) + 1 + ((F & 1) ? 0 : 1); }

constexpr int kseq_len_max() { return kMaxF - 2 + (kMaxF - 1) / 2 + 2; }  // kMaxF is even

__device__ __forceinline__ int find_uni(const int32_t* off, int n, int item) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= item)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// Candidates that the mixed prefilter leaves to the FP64 retest this round, in no order:
// (universe, offset in the round), RoundInfo::total_gray of them.  The first mask_cap
// carry a bit per timestep where a pair lies in the guard band: every pair of the other
// timesteps is decided, so the retest evaluates those timesteps alone.
struct RetestQueue {
    int2* item;      // [sum of B_max]
    uint4* mask;     // [mask_cap][2]
    int32_t mask_cap;
    int32_t cap;
};
// k_test64: per CTA, the coefficient columns of its 32 candidates (1+1D crossings: and
// their trajectories), and for the knot stream its draws.
constexpr int kT64Threads = 256;
constexpr int kT64Pos = 32 * 3 * 16;    // positions of a stage
constexpr int kT64Tests = 32 * 16;      // (candidate, timestep) tests of a stage
constexpr int kT64Cells = 2048;         // occupied cells of their windows
struct Scratch64 {
    double* coef;
    size_t coef_stride;
    double *wgt, *phase;  // [term][axis * 32 + candidate]
    uint16_t* freq;
    size_t knot_stride;
};
constexpr int kMaskWords = kMaxF / 32;
static_assert(kMaskWords == 8, "a mask is two uint4");

// Kernels (ug_kernels.cu)
__global__ void k_plan(const UniDev* __restrict__ U, UniCtl* ctl, RoundInfo* info, int nsm);
__global__ void k_test64(const UniDev* __restrict__ U, UniCtl* ctl, RoundInfo* info, Scratch64 sc, int all);
__global__ void k_retest(const UniDev* __restrict__ U, UniCtl* ctl, RoundInfo* info, RetestQueue rq);
__global__ void k_compact(const UniDev* __restrict__ U, UniCtl* ctl, RoundInfo* info);
__global__ void k_surv_gen(const UniDev* __restrict__ U, UniCtl* ctl, RoundInfo* info, int warp_bytes);
__global__ void k_surv_gemm(const UniDev* __restrict__ U, UniCtl* ctl, RoundInfo* info);
__global__ void k_surv_hash(const UniDev* __restrict__ U, UniCtl* ctl, RoundInfo* info);
__global__ void k_restore_gen(const UniDev* __restrict__ U, int u, const int64_t* __restrict__ idx, int m);
__global__ void k_probe(const UniDev* __restrict__ U, int u, int64_t n_slots, uint64_t seed, int64_t n, int bins,
                        unsigned long long* proposed, unsigned long long* accepted);
__global__ void k_conflicts(const UniDev* __restrict__ U, UniCtl* ctl, RoundInfo* info);
__global__ void k_greedy(const UniDev* __restrict__ U, UniCtl* ctl, RoundInfo* info);
__global__ void k_commit(const UniDev* __restrict__ U, UniCtl* ctl, RoundInfo* info);
__global__ void k_rehash(const UniDev* __restrict__ U, UniCtl* ctl, int u, int64_t n_slots);
__global__ void k_positions(const UniDev* __restrict__ U, int u, int64_t n, double* __restrict__ out);
__global__ void k_gather_accepted(const UniDev* __restrict__ U, const int64_t* __restrict__ off,
                                  int64_t* __restrict__ idx, int32_t* __restrict__ gid);

// k_greedy: admissions and groups of a round's survivors, two windows of contact lists
// (padded so that the lanes' lists start on different banks).
constexpr int kListPitch = kConflictCap + 4;
constexpr size_t kGreedySmem = ((size_t)2 * kSmaxCap + 2 * 32 * kListPitch) * sizeof(int32_t);

// k_surv_gemm: warp tiles of kGemmRows rows x 32 timesteps.
constexpr int kGemmRows = 16;
__host__ __device__ __forceinline__ int gemm_tiles(int rows, int T) {
    return (rows + kGemmRows - 1) / kGemmRows * ((T + 31) >> 5);
}

// Shared memory of k_surv_gen per warp (bytes), for F <= kMaxF.
constexpr int kSurvWarps = 4;
constexpr size_t kSurvSmemPerWarp = (size_t)3 * (kMaxF + 1) * 2 * sizeof(double) + 3 * sizeof(double) +
                                    (size_t)kMaxF * (sizeof(int32_t) + 2 * sizeof(double));
// k_surv_gen on a batch without knot-stream universes: one axis of alpha / beta
constexpr size_t kSurvSmemAxis = (size_t)2 * (kMaxF + 1) * sizeof(double);
// k_retest: the candidate's term-ordered coefficient rows and its phases
constexpr int kRowK = kseq_len_max();
constexpr size_t kRetestSmem = (size_t)3 * (kRowK + kMaxF) * sizeof(double);

}  // namespace ug
