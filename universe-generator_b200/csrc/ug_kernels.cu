// ug_kernels.cu -- the round pipeline of the batched RSA packer.
//
// One round of every active universe:
//   k_plan         round sizes, phase transitions, tile decomposition
//   k_test64       FP64 form: every candidate against the committed packing, a CTA per
//                  32 candidates (also the universes of a mixed batch that the tensor-core
//                  test does not take)
//   k_prefilter_mixed (ug_mixed.cu) + k_retest
//                  mixed form: the tensor-core test, then the FP64 test of the
//                  timesteps that its guard band left undecided
//   k_compact      survivors in candidate-index order (deterministic)
//   k_surv_gen     FP64 coefficients of the survivors (term-ordered rows)
//   k_surv_gemm    their FP64 trajectories as an FP64 tensor product
//   k_surv_hash    round-table insert of every survivor timestep
//   k_conflicts    each survivor's contacts with EARLIER survivors of the round
//   k_greedy       in-order resolution: survivor i is admitted iff it touches
//                  no admitted earlier survivor (group rules in group modes)
//   k_commit       admitted trajectories appended to the collision grid
// Non-survivors collide with the committed packing, which only grows, so they
// are rejected by sequential RSA as well; survivors are decided in index
// order against the round's earlier admissions.  The accepted set is
// therefore exactly sequential RSA over the candidate stream -- the
// exact-index admission of cuda/braid_knot.cu:433-462, made device-resident.
#include "ug_dmma.cuh"
#include "ug_kernels.cuh"

#include <algorithm>
#include <type_traits>

namespace ug {

// ------------------------------------------------------------------ plan

// Closes the bucket ending at phase position in_phase (a multiple of q) with the
// count cur; true when the phase stops there: 32 buckets, more than 1e6
// candidates decided, and the last 32 buckets' count / (32 q) below thr.
__device__ __forceinline__ bool win_close(int64_t q, int64_t& nb, int64_t& sum, int64_t& cur, int64_t* ring,
                                          double thr, int64_t in_phase) {
    if (q <= 0 || in_phase <= 0 || in_phase % q) return false;
    const int slot = (int)(nb & 31);
    if (nb >= 32) sum -= ring[slot];
    ring[slot] = cur;
    sum += cur;
    cur = 0;
    nb++;
    return nb >= 32 && in_phase > 1000000 && (double)sum / (double)(32 * q) < thr;
}

// Exclusive prefix of v over the 256 threads of the block; *total gets the sum.
// Every thread of the block must call it (it synchronises the block).
__device__ __forceinline__ int block_excl_scan256(int v, int* wsum, int* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += x;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    int wpre = 0, tot = 0;
    for (int k = 0; k < 8; k++) {
        if (k < warp) wpre += wsum[k];
        tot += wsum[k];
    }
    __syncthreads();  // wsum is reused by the next call
    *total = tot;
    return wpre + incl - v;
}

// The next round of every universe: the last round's windows closed (also of a universe that
// waits for the host to grow its buffers), phases switched, round sizes and tiles.  Planning
// a planned round again changes nothing but the epoch of a round table not yet written.
__global__ void k_plan(const UniDev* __restrict__ U, UniCtl* ctl, RoundInfo* info, int nsm) {
    __shared__ int32_t ntiles[kMaxUni];
    __shared__ int32_t cost[kMaxUni];
    __shared__ int32_t order[kMaxUni];
    __shared__ unsigned long long s_work;
    __shared__ int32_t s_busy;
    if (threadIdx.x == 0) {
        s_work = 0;
        s_busy = 0;
    }
    __syncthreads();
    const int n = info->n_uni;
    for (int u = threadIdx.x; u < n; u += blockDim.x) {
        UniCtl& c = ctl[u];
        const UniDev& d = U[u];
        int B = 0;
        // tile cost: the slowest prefilter tile of the last round that timed any; before
        // that, dim * T stands in (all universes start together, so one round uses one kind)
        if (c.tile_ns > 0) c.tile_cost = c.tile_ns;
        cost[u] = c.tile_cost > 0 ? c.tile_cost : d.dim * d.T;
        c.tile_ns = 0;
        // the last round's admissions (k_greedy) and newly occupied cells (k_commit)
        // close the windows' buckets; rounds end on bucket boundaries
        {
            const int64_t nc = c.round_new;
            c.round_new = 0;
            c.filled += nc;
            if (c.last_used > 0 && (c.state == ST_ACTIVE || c.state == ST_GROW)) {
                const int64_t in_phase = c.next_cand - c.phase_start;
                c.win_cur += c.accepted_round;
                c.fwin_cur += nc;
                const bool sa = win_close(c.win_q, c.win_nb, c.win_sum, c.win_cur, c.win_ring, c.win_thr, in_phase);
                const bool sf = win_close(c.fwin_q, c.fwin_nb, c.fwin_sum, c.fwin_cur, c.fwin_ring, c.sub_fill_rate,
                                          in_phase);
                if (sa || sf) c.phase_end = c.next_cand;  // stops below
            }
            c.last_used = 0;
        }
        if (c.state == ST_ACTIVE) {
            for (int guard = 0; guard < 2; guard++) {
                const bool over = c.next_cand >= c.phase_end ||
                                  (c.phase == 1 && c.max_n > 0 && c.n_unique >= c.max_n);
                if (!over) break;
                if (c.phase == 1 && d.group_mode == GROUP_SUBPATH) {
                    c.phase = 2;
                    c.phase1_end = c.next_cand;
                    c.phase_start = c.next_cand;
                    c.phase_end = c.next_cand + c.sub_budget;
                    c.round_B = c.B_cap;  // fresh adaptation (braid_cuda.cu:952)
                    c.win_thr = c.sub_accept_rate;
                    c.win_q = win_bucket(c.sub_accept_rate);
                    c.win_nb = c.win_sum = c.win_cur = 0;
                    c.fwin_q = win_bucket(c.sub_fill_rate);
                    c.fwin_nb = c.fwin_sum = c.fwin_cur = 0;
                    continue;
                }
                c.state = ST_DONE;
                break;
            }
            if (c.state == ST_ACTIVE) {
                int64_t left = c.phase_end - c.next_cand;
                const int64_t in_phase = c.next_cand - c.phase_start;
                if (c.win_q > 0) left = min(left, c.win_q - in_phase % c.win_q);
                if (c.fwin_q > 0) left = min(left, c.fwin_q - in_phase % c.fwin_q);
                const int cap = c.round_B < d.B_max ? c.round_B : d.B_max;  // per-round buffers hold B_max
                B = (int)(left < (int64_t)cap ? left : (int64_t)cap);
            }
        }
        c.B = B;
        c.round_base = c.next_cand;
        c.S = c.S_raw = c.trunc = c.stop_at = 0;
        if (B > 0) c.epoch = (c.epoch + 1) & 0xFFFFFF;
        ntiles[u] = (B + kTile - 1) / kTile;
        if (B > 0) {
            atomicAdd(&s_work, (unsigned long long)cost[u] * ntiles[u]);
            atomicAdd(&s_busy, 1);
        }
    }
    __syncthreads();
    // Tiles of the tensor-core test take kTile candidates.  Where one such tile is long
    // against the round's work per SM, its universe's tiles are cut to 64 or 32: a tile of
    // 64 takes about two thirds of the time (generation and products do not shrink, the
    // tests do), one of 32 half, but two to four times the SMs share them.  A universe
    // alone also cuts the tiles of its last, partial wave.  Per job: four 3+1 universes of
    // T = 113 to 253 (40 tiles a round on 148 SMs) 18.3 -> 15.0 ms of prefilter, one of
    // T = 128 (up to 512 tiles) 37.3 -> 35.3 ms.
    const unsigned long long per_sm = s_work / nsm;
    for (int u = threadIdx.x; u < n; u += blockDim.x) {
        const int nt = ntiles[u];
        int full = nt, rows = kTile;
        if (nt > 0 && U[u].mx_ok) {
            if ((unsigned long long)cost[u] >= 2 * per_sm) {
                full = 0;
                rows = (unsigned long long)cost[u] >= 4 * per_sm ? 32 : 64;
            } else if (s_busy == 1 && nt > nsm) {
                const int rest = nt % nsm;  // whole waves alone have no last wave to share
                if (rest > 0 && rest * 2 <= nsm) {
                    rows = rest * 4 <= nsm ? 32 : 64;
                    full = nt - rest;
                }
            }
            if (rows < kTile) ntiles[u] = full + (ctl[u].B - full * kTile + rows - 1) / rows;
        }
        info->tile_full[u] = full;
        info->tile_rows[u] = rows;
    }
    __syncthreads();
    // Tiles are handed out costliest universe first, so the long tiles start in
    // the first wave instead of trailing the round (order does not change results).
    for (int u = threadIdx.x; u < n; u += blockDim.x) {
        const int cu = ntiles[u] > 0 ? cost[u] : -1;
        int rank = 0;
        for (int v = 0; v < n; v++) {
            const int cv = ntiles[v] > 0 ? cost[v] : -1;
            rank += cv > cu || (cv == cu && v < u);
        }
        order[rank] = u;
    }
    __syncthreads();
    __shared__ int32_t wsum[8];
    int acc = 0;
    for (int b0 = 0; b0 < n; b0 += 256) {  // k_plan runs as one block of 256 threads
        const int i = b0 + threadIdx.x;
        const int nt = i < n ? ntiles[order[i]] : 0;
        int tot;
        const int p = block_excl_scan256(nt, wsum, &tot);
        if (i < n) {
            info->tile_off[i] = acc + p;
            info->tile_uni[i] = order[i];
        }
        acc += tot;
    }
    if (threadIdx.x == 0) {
        info->tile_off[n] = acc;
        info->total_tiles = acc;
        info->any_active = acc > 0;
        info->total_surv = 0;
        info->total_gray = 0;
        info->t64_next = 0;
        info->compact_done = 0;
        info->tile_next = 0;
        info->confl_next = 0;
        info->gemm_next = 0;
    }
}

// ------------------------------------------------------------- prefilter

// FP64 test of candidate idx against the committed packing.  Returns true
// when it is rejected.  Group mode: *g gets the single group touched (-1 none).
__device__ bool test64(const UniDev& d, int64_t n_slots, const double* alpha, const double* beta,
                       const double* a2, bool group, int32_t* g, int* nev, int* nvis = nullptr) {
    *g = -1;
    const int T = d.T, F1 = d.F + 1;
    if (d.dim == 1 && d.cross1d) {
        double P[kMaxF];
        for (int t = 0; t < T; t++) P[t] = eval64(d, alpha, beta, 1, a2[0], t);
        *nev = T;
        for (int64_t s = 0; s < n_slots; s++) {
            const Pt64* q = d.pts + UG_IDX(s * T + T - 1, d.slot_cap * T) + 1 - T;
            double d0 = torus_delta(P[0] - __ldcg(&q[0].c[0]));
            bool hit = hit1(d0, d.cell, d.inclusive);
            for (int t = 1; t < T && !hit; t++) {
                const double d1 = torus_delta(P[t] - __ldcg(&q[t].c[0]));
                hit = hit1(d1, d.cell, d.inclusive) || crosses_step(d0, d1);
                d0 = d1;
            }
            if (hit) {
                if (!group) return true;
                const int32_t gq = __ldcg(&q[0].gid);
                if (*g == -1)
                    *g = gq;
                else if (*g != gq)
                    return true;
            }
        }
        return false;
    }
    const int64_t cpt = cells_per_t(d);
    for (int oi = 0; oi < T; oi++) {
        const int t = __ldg(d.order + oi);
        double P[3];
        for (int ax = 0; ax < d.dim; ax++) P[ax] = eval64(d, alpha + ax * F1, beta + ax * F1, 1, a2[ax], t);
        *nev = oi + 1;
        if (contacts64(d, t, P, group, g, cpt, nvis)) return true;
    }
    return false;
}

// Diagnostic probe (braid_cuda3d.cu:1650-1660): n fresh candidates of the stream
// keyed by `seed` tested against the final packing (plain exclusion), counted per
// bin of the x axis's sin1 offset a2 over [-1, 1).
__global__ void __launch_bounds__(kTile) k_probe(const UniDev* __restrict__ U, int u, int64_t n_slots,
                                                 uint64_t seed, int64_t n, int bins,
                                                 unsigned long long* proposed, unsigned long long* accepted) {
    extern __shared__ unsigned long long probe_hist[];  // [2][bins]
    for (int i = threadIdx.x; i < 2 * bins; i += blockDim.x) probe_hist[i] = 0;
    __syncthreads();
    UniDev d = U[u];
    d.seed = seed;
    double alpha[3 * (kMaxF + 1)], beta[3 * (kMaxF + 1)], a2[3];
    int32_t bj[kMaxF];
    double wj[kMaxF];
    const int F1 = d.F + 1;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        if (d.rng == RNG_KNOT)
            gen_knot64(d, (uint64_t)i, alpha, beta, a2, bj, wj, 1);
        else
            for (int ax = 0; ax < d.dim; ax++) a2[ax] = gen_philox64(d, (uint64_t)i, ax, alpha + ax * F1, beta + ax * F1, 1);
        int32_t g;
        int nev;
        const bool free = !test64(d, n_slots, alpha, beta, a2, false, &g, &nev);
        int b = (int)floor((a2[0] + 1.0) * 0.5 * bins);
        b = b < 0 ? 0 : (b >= bins ? bins - 1 : b);
        atomicAdd(&probe_hist[b], 1ull);
        if (free) atomicAdd(&probe_hist[bins + b], 1ull);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < bins; i += blockDim.x) {
        if (probe_hist[i]) atomicAdd(&proposed[i], probe_hist[i]);
        if (probe_hist[bins + i]) atomicAdd(&accepted[i], probe_hist[bins + i]);
    }
}

__device__ __forceinline__ bool group_phase(const UniDev& d, const UniCtl& c) {
    return d.group_mode == GROUP_UNIQUE || (d.group_mode == GROUP_SUBPATH && c.phase == 2);
}

// --------------------------------------------------------------- compact

__global__ void __launch_bounds__(256) k_compact(const UniDev* __restrict__ U, UniCtl* ctl,
                                                 RoundInfo* info) {
    __shared__ int32_t wsum[8];
    __shared__ int32_t s_running;
    __shared__ bool s_last;
    const int u = blockIdx.x;
    const UniDev& d = U[u];
    UniCtl& c = ctl[u];
    const int B = c.B;
    const int nwords = (B + 31) >> 5;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_running = 0;
    __syncthreads();
    for (int base = 0; base < nwords; base += 256) {
        const int w = base + tid;
        uint32_t bits = w < nwords ? d.surv_bits[w] : 0u;
        if (w == nwords - 1 && (B & 31)) bits &= (1u << (B & 31)) - 1u;
        const int cnt = __popc(bits);
        int incl = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        int wpre = 0, tot = 0;
        for (int k = 0; k < 8; k++) {
            if (k < warp) wpre += wsum[k];
            tot += wsum[k];
        }
        int rank = s_running + wpre + incl - cnt;
        while (bits) {
            const int bit = __ffs(bits) - 1;
            bits &= bits - 1;
            if (rank <= d.S_max) d.surv_off[UG_IDX(rank, d.S_max + 1)] = w * 32 + bit;
            rank++;
        }
        __syncthreads();
        if (tid == 0) s_running += tot;
        __syncthreads();
    }
    const int S_raw = s_running;
    const int S = S_raw < d.S_max ? S_raw : d.S_max;
    for (int r = tid; r < S; r += 256) d.ccount[r] = 0;
    if (tid == 0) {
        c.S_raw = S_raw;
        c.S = S;
        c.trunc = S;
        __threadfence();
        s_last = atomicAdd(&info->compact_done, 1) == info->n_uni - 1;
    }
    __syncthreads();
    if (s_last) {  // the last block: work offsets of every universe, as block scans
        __threadfence();
        const int n = info->n_uni;
        int acc = 0, sev = 0, spt = 0, acc_o = 0, sev_o = 0;
        for (int b0 = 0; b0 < n; b0 += 256) {
            const int v = b0 + tid;
            int Sv = 0, sevv = 0, sptv = 0, So = 0, sevo = 0;
            if (v < n) {
                Sv = *(volatile int32_t*)&ctl[v].S;
                sevv = gemm_tiles(Sv * U[v].dim, U[v].T);
                sptv = Sv * U[v].T;
                // the same survivors and product tiles, universes in tile order (costliest first)
                const int uo = info->tile_uni[v];
                So = *(volatile int32_t*)&ctl[uo].S;
                sevo = gemm_tiles(So * U[uo].dim, U[uo].T);
            }
            int t1, t2, t3, t4, t5;
            const int p1 = block_excl_scan256(Sv, wsum, &t1);
            const int p2 = block_excl_scan256(sevv, wsum, &t2);
            const int p3 = block_excl_scan256(sptv, wsum, &t3);
            const int p4 = block_excl_scan256(So, wsum, &t4);
            const int p5 = block_excl_scan256(sevo, wsum, &t5);
            if (v < n) {
                info->surv_off[v] = acc + p1;
                info->sev_off[v] = sev + p2;
                info->spt_off[v] = spt + p3;
                info->surv_off_o[v] = acc_o + p4;
                info->sev_off_o[v] = sev_o + p5;
            }
            acc += t1;
            sev += t2;
            spt += t3;
            acc_o += t4;
            sev_o += t5;
        }
        if (tid == 0) {
            info->surv_off[n] = acc;
            info->sev_off[n] = sev;
            info->spt_off[n] = spt;
            info->surv_off_o[n] = acc_o;
            info->sev_off_o[n] = sev_o;
            info->total_surv = acc;
            info->total_sev = sev;
            info->total_spt = spt;
        }
    }
}

// ------------------------------------------------------------ survivors

// Round table entry of (timestep t, block lin): one 8-byte word per (t, block),
// epoch in the high half so no table is ever cleared.  A direct table replaced an
// open-addressing hash keyed by (epoch, t, block): one exchange per insert instead of
// a probe, a compare-and-swap and an exchange, and a quarter of the memory.
__device__ __forceinline__ uint64_t* rentry(const UniDev& d, int t, int64_t lin) {
    return d.rhead + UG_IDX((int64_t)t * d.rblocks + lin, (int64_t)d.T * d.rblocks);
}
// Head survivor of the chain of (t, block) this round (-1 none).
__device__ __forceinline__ int32_t rtab_head(const UniDev& d, int epoch, int t, int64_t lin) {
    const uint64_t v = __ldcg(rentry(d, t, lin));
    return (v >> 32) == (uint64_t)(uint32_t)epoch ? (int32_t)(uint32_t)v : -1;
}

// Warp-cooperative FP64 regeneration of axis ax of candidate idx (Philox
// stream) into shared memory: Philox blocks are spread over the lanes, the
// normalisation sum runs in ascending b on lane 0 -- the same operations, in
// the same order, as the thread-per-candidate gen_philox64, so the
// coefficients are identical.
__device__ __forceinline__ void warp_gen64_axis(const UniDev& d, uint64_t idx, int ax, double* alpha, double* beta,
                                                double* a2, int lane) {
    const int F = d.F, F1 = F + 1;
    double* al = alpha + ax * F1;
    double* bt = beta + ax * F1;
    for (int p = lane; 2 * p <= F; p += 32) {
        const uint4 o = philox_block(d.seed, idx, ax, p);
        if (p == 0) {
            a2[ax] = d.pin ? 0.0 : (double)o.x * (1.0 / 2147483648.0) - 1.0;
            continue;
        }
        const int be = 2 * p, bo = 2 * p + 1;
        const double Ee = -log(((double)o.x + 0.5) * (1.0 / 4294967296.0));
        al[be] = (o.z & 1u) ? -Ee : Ee;
        bt[be] = (double)(o.z >> 1) * (1.0 / 2147483648.0) * kPi;
        if (bo <= F) {
            const double Eo = -log(((double)o.y + 0.5) * (1.0 / 4294967296.0));
            al[bo] = (o.w & 1u) ? -Eo : Eo;
        }
    }
    __syncwarp();
    double sum = 0.0;
    if (lane == 0)
        for (int b = 2; b <= F; b++) sum += fabs(al[b]);
    sum = __shfl_sync(0xffffffffu, sum, 0);
    for (int b = 2 + lane; b <= F; b += 32) {
        const double e = al[b];
        double amp = fabs(e) / sum / (double)b;
        if (e < 0.0) amp = -amp;
        if (b & 1) {
            al[b] = amp;
            bt[b] = 0.0;
        } else {
            double sf, cf;
            sincos(bt[b], &sf, &cf);
            al[b] = amp * cf;
            bt[b] = amp * sf;
        }
    }
    __syncwarp();
}

// The knot stream's coefficients (gen_knot64's draws and operations) by one warp: lane 0
// draws and sums in list order, the lanes take the logarithms, sines and divisions, whose
// FP64 chains were most of a lane's work: T = 65, all 64 terms of 3 axes, 122 -> 67 us a round.
// ph: nw phases.
__device__ __forceinline__ void warp_knot64(const UniDev& d, uint64_t idx, double* alpha, double* beta, double* a2,
                                            int32_t* bj, double* wj, double* ph, int lane) {
    Xo r;
    if (lane == 0) r.seed(knot_seed(d.seed, idx));
    const int nw = d.nw, F1 = d.F + 1;
    const bool full = (uint32_t)nw == d.modmax;  // every frequency once
    for (int ax = 0; ax < d.dim; ax++) {
        double* al = alpha + ax * F1;
        double* bt = beta + ax * F1;
        for (int b = lane; b < F1; b += 32) al[b] = bt[b] = 0.0;
        if (full)
            for (int j = lane; j < nw; j += 32) bj[j] = j + 2;
        __syncwarp();
        if (lane == 0) {
            if (full) {
                for (int j = nw - 1; j > 0; j--) {
                    const int k = (int)r.below((uint32_t)(j + 1));
                    const int32_t tmp = bj[j];
                    bj[j] = bj[k];
                    bj[k] = tmp;
                }
            } else {
                for (int j = 0; j < nw; j++) {
                    int b = 0;
                    bool dup = true;
                    for (int guard = 0; dup && guard < 64; guard++) {
                        b = (int)r.below(d.modmax) + 2;
                        dup = false;
                        for (int k = 0; k < j; k++) dup |= bj[k] == b;
                    }
                    bj[j] = b;
                }
            }
            for (int j = 0; j < nw; j++) wj[j] = 1.0 - r.f64();
            for (int j = 0; j < nw; j++) {
                const int b = bj[j];
                if (r.flip()) bj[j] = -b;
                if (!(b & 1)) ph[j] = r.f64() * kPi;
            }
            a2[ax] = d.pin ? 0.0 : (r.f64() * 2.0 - 1.0);
        }
        __syncwarp();
        for (int j = lane; j < nw; j += 32) wj[j] = -log(wj[j]);
        __syncwarp();
        double sum = 0.0;
        if (lane == 0)
            for (int j = 0; j < nw; j++) sum += wj[j];
        sum = __shfl_sync(0xffffffffu, sum, 0);
        for (int j0 = 0; j0 < nw; j0 += 32) {
            const int j = j0 + lane, b = j < nw ? abs(bj[j]) : 1;
            double amp = 0.0, sf = 0.0, cf = 0.0;
            if (j < nw) {
                amp = wj[j] / sum / (double)b;
                if (bj[j] < 0) amp = -amp;
                if (!(b & 1)) sincos(ph[j], &sf, &cf);
            }
            auto add = [&]() {
                if (b & 1)
                    al[b] += amp;
                else
                    add_even_term(al[b], bt[b], amp, sf, cf);
            };
            if (full) {
                if (j < nw) add();
            } else {  // few terms may list a frequency twice: added in term order
                for (int q = 0; q < min(32, nw - j0); q++) {
                    if (lane == q) add();
                    __syncwarp();
                }
            }
        }
        __syncwarp();
    }
}

// All axes of candidate idx by one warp.
__device__ __forceinline__ void warp_gen64(const UniDev& d, uint64_t idx, double* alpha, double* beta,
                                       double* a2, int32_t* bj, double* wj, double* ph, int lane) {
    if (d.rng == RNG_KNOT) {
        warp_knot64(d, idx, alpha, beta, a2, bj, wj, ph, lane);
    } else {
        for (int ax = 0; ax < d.dim; ax++) warp_gen64_axis(d, idx, ax, alpha, beta, a2, lane);
    }
}

// Rows r * dim + ax of the term-ordered coefficient matrix of one survivor.
__device__ __forceinline__ void store_coef_rows(const UniDev& d, int r, const double* alpha, const double* beta,
                                                const double* a2, int lane) {
    const int F = d.F, F1 = F + 1, R = d.Rpad;
    [[maybe_unused]] const int64_t ncoef = (int64_t)d.K * R;
    for (int ax = 0; ax < d.dim; ax++) {
        const int row = r * d.dim + ax;
        const double* al = alpha + ax * F1;
        const double* bt = beta + ax * F1;
        for (int b = 2 + lane; b <= F; b += 32) {
            const int64_t k = kseq_s(b);
            d.coef[UG_IDX(k * R + row, ncoef)] = al[b];
            if (!(b & 1)) d.coef[UG_IDX((k + 1) * R + row, ncoef)] = bt[b];
        }
        if (lane == 0) d.a2row[UG_IDX(row, R)] = a2[ax];
    }
}

// Survivor trajectories in three steps.
//
// k_surv_gen: one warp per survivor regenerates its FP64 coefficients
// (warp-parallel Philox blocks, sequential normalisation sum in ascending b --
// the same operations as the thread-per-candidate prefilter, so identical
// values) and stores them as rows r * dim + ax of the term-ordered matrix coef.
__global__ void __launch_bounds__(32 * kSurvWarps) k_surv_gen(const UniDev* __restrict__ U,
                                                                UniCtl* ctl, RoundInfo* info, int warp_bytes) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    unsigned char* my = smem_raw + (size_t)wib * warp_bytes;
    double* alpha = (double*)my;
    double* beta = alpha + 3 * (kMaxF + 1);
    double* a2 = beta + 3 * (kMaxF + 1);
    double* wj = a2 + 3;
    double* ph = wj + kMaxF;
    int32_t* bj = (int32_t*)(ph + kMaxF);
    const int n_uni = info->n_uni, total = info->total_surv;
    const int gwarp = blockIdx.x * kSurvWarps + wib, nwarps = gridDim.x * kSurvWarps;
    for (int item = gwarp; item < total; item += nwarps) {
        const int u = find_uni(info->surv_off, n_uni, item);
        const int r = item - info->surv_off[u];
        const UniDev& d = U[u];
        const UniCtl& c = ctl[u];
        const uint64_t idx = (uint64_t)(c.round_base + d.surv_off[UG_IDX(r, d.S_max + 1)]);
        if (d.rng == RNG_PHILOX) {
            // one axis at a time in a (F+1)-entry buffer pair, rows written as they are
            // finished: warp_gen64's operations per axis, a quarter of its shared memory
            const int F = d.F, R = d.Rpad;
            [[maybe_unused]] const int64_t ncoef = (int64_t)d.K * R;
            double* al = (double*)my;
            double* bt = al + (kMaxF + 1);
            for (int ax = 0; ax < d.dim; ax++) {
                const int row = r * d.dim + ax;
                for (int p = lane; 2 * p <= F; p += 32) {
                    const uint4 o = philox_block(d.seed, idx, ax, p);
                    if (p == 0) {
                        d.a2row[UG_IDX(row, R)] = d.pin ? 0.0 : (double)o.x * (1.0 / 2147483648.0) - 1.0;
                        continue;
                    }
                    const int be = 2 * p, bo = 2 * p + 1;
                    const double Ee = -log(((double)o.x + 0.5) * (1.0 / 4294967296.0));
                    al[be] = (o.z & 1u) ? -Ee : Ee;
                    bt[be] = (double)(o.z >> 1) * (1.0 / 2147483648.0) * kPi;
                    if (bo <= F) {
                        const double Eo = -log(((double)o.y + 0.5) * (1.0 / 4294967296.0));
                        al[bo] = (o.w & 1u) ? -Eo : Eo;
                    }
                }
                __syncwarp();
                double sum = 0.0;
                if (lane == 0)
                    for (int b = 2; b <= F; b++) sum += fabs(al[b]);
                sum = __shfl_sync(0xffffffffu, sum, 0);
                for (int b = 2 + lane; b <= F; b += 32) {
                    const double e = al[b];
                    double amp = fabs(e) / sum / (double)b;
                    if (e < 0.0) amp = -amp;
                    const int64_t k = kseq_s(b);
                    if (b & 1) {
                        d.coef[UG_IDX(k * R + row, ncoef)] = amp;
                    } else {
                        double sf, cf;
                        sincos(bt[b], &sf, &cf);
                        d.coef[UG_IDX(k * R + row, ncoef)] = amp * cf;
                        d.coef[UG_IDX((k + 1) * R + row, ncoef)] = amp * sf;
                    }
                }
                __syncwarp();
            }
            continue;
        }
        warp_gen64(d, idx, alpha, beta, a2, bj, wj, ph, lane);
        store_coef_rows(d, r, alpha, beta, a2, lane);
        __syncwarp();
    }
}

// Checkpoint restore: the coefficient rows of m given admissions (explicit
// candidate indices) of universe u, as k_surv_gen writes them for survivors.
__global__ void __launch_bounds__(32 * kSurvWarps) k_restore_gen(const UniDev* __restrict__ U, int u,
                                                                   const int64_t* __restrict__ idx, int m) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    unsigned char* my = smem_raw + (size_t)wib * kSurvSmemPerWarp;
    double* alpha = (double*)my;
    double* beta = alpha + 3 * (kMaxF + 1);
    double* a2 = beta + 3 * (kMaxF + 1);
    double* wj = a2 + 3;
    double* ph = wj + kMaxF;
    int32_t* bj = (int32_t*)(ph + kMaxF);
    const UniDev& d = U[u];
    const int gwarp = blockIdx.x * kSurvWarps + wib, nwarps = gridDim.x * kSurvWarps;
    for (int r = gwarp; r < m; r += nwarps) {
        warp_gen64(d, (uint64_t)idx[r], alpha, beta, a2, bj, wj, ph, lane);
        store_coef_rows(d, r, alpha, beta, a2, lane);
        __syncwarp();
    }
}

// k_surv_gemm: X[row][t] = wrap(a2 + invsinz_t * sum_k coef[k][row] KT[k][t]), one warp per
// tile of 16 rows x 32 timesteps (less at the last timesteps), as FP64 tensor products
// over ascending k: eval64's operations in eval64's order.  The operands come straight
// from L1/L2 two steps of eight terms ahead; the small tile keeps a round of few survivors
// on many warps.  FP64 FMAs from shared memory waited for their operands (a lane's 4 x 8
// outputs take 48 bytes of shared memory per 32 FMAs: two thirds of the FP64 rate at best).
// Per round: 2+1 T = 256, 270 survivors 84 -> 42 us; 3+1 T = 128, 1800 52 -> 33 us; a
// 32-universe batch 152 -> 120 us.
__global__ void __launch_bounds__(128) k_surv_gemm(const UniDev* __restrict__ U, UniCtl* ctl,
                                                   RoundInfo* info) {
    const int lane = threadIdx.x & 31, gl = lane >> 2, tl = lane & 3;
    const int n_uni = info->n_uni, total = info->total_sev;
    // tiles handed out one at a time, costliest universes first (a tile's cost is
    // its universe's term count K, 24 to 384); the next claimed when one starts
    int item = 0, next = 0;
    if (lane == 0) item = atomicAdd(&info->gemm_next, 1);
    item = __shfl_sync(0xffffffffu, item, 0);
    for (; item < total; item = __shfl_sync(0xffffffffu, next, 0)) {
        if (lane == 0) next = atomicAdd(&info->gemm_next, 1);
        const int pos = find_uni(info->sev_off_o, n_uni, item);
        const int u = info->tile_uni[pos];
        const int local = item - info->sev_off_o[pos];
        const UniDev& d = U[u];
        const int T = d.T, dim = d.dim, K = d.K, R = d.Rpad, TP = d.Tpad;
        const int ntb = (T + 31) >> 5;
        const int rb = local / ntb, tb = local - rb * ntb;
        const int t0 = tb * 32, nn = min(4, (T - t0 + 7) >> 3);  // timestep blocks of 8
        const double* Ag = d.coef + rb * kGemmRows + gl;  // tile rows below Rpad
        const double* Bg = d.KT + t0 + gl;                // tile timesteps below Tpad
        struct Step {
            double a[4], b[4][2];
        };
        auto fetch = [&](int k0, Step& s) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int k = k0 + 4 * h + tl;
                const bool on = k < K;
                s.a[2 * h] = on ? Ag[(size_t)k * R] : 0.0;
                s.a[2 * h + 1] = on ? Ag[(size_t)k * R + 8] : 0.0;
#pragma unroll
                for (int j = 0; j < 4; j++) s.b[j][h] = on && j < nn ? __ldg(Bg + (size_t)k * TP + 8 * j) : 0.0;
            }
        };
        double acc[4][4];
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int q = 0; q < 4; q++) acc[j][q] = 0.0;
        Step s[3];
        fetch(0, s[0]);
        fetch(8, s[1]);
        for (int k0 = 0; k0 < K; k0 += 24) {
#pragma unroll
            for (int h = 0; h < 3; h++) {
                if (k0 + 8 * h >= K) break;
                fetch(k0 + 8 * (h + 2), s[(h + 2) % 3]);
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (j < nn) dmma_16x8x8(acc[j], s[h].a, s[h].b[j]);
            }
        }
        const int nrows = ctl[u].S * dim;
        [[maybe_unused]] const int64_t nspos = (int64_t)d.S_max * T;
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int row = rb * kGemmRows + gl + 8 * q;
            if (row >= nrows) continue;
            const int r = row / dim, ax = row - r * dim;
            const double a2 = d.a2row[UG_IDX(row, R)];
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int t = t0 + 8 * j + 2 * tl + e;
                    if (t < T)
                        d.spos[UG_IDX((int64_t)r * T + t, nspos)].c[ax] =
                            torus_wrap(fma(acc[j][2 * q + e], __ldg(d.invsinz + t), a2));
                }
        }
    }
}

// Round-table block of a cell: 2^rblock_shift cells per axis (host-chosen per
// universe, at least 2), so the 3 neighbour cells of a point span at most 2
// blocks per axis (3 only at the seam of a partial last block).
static_assert(2 * kMaxF <= 1024, "k_conflicts packs block coordinates in 10 bits");
__device__ __forceinline__ int rblock_gw(const UniDev& d) {
    return (d.gw + (1 << d.rblock_shift) - 1) >> d.rblock_shift;
}

// k_surv_hash: one thread per survivor timestep inserts the point into the
// round table (entry: t, block; tagged with the epoch).
__global__ void __launch_bounds__(256) k_surv_hash(const UniDev* __restrict__ U, UniCtl* ctl,
                                                   RoundInfo* info) {
    const int n_uni = info->n_uni, total = info->total_spt;
    for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < total; w += gridDim.x * blockDim.x) {
        const int u = find_uni(info->spt_off, n_uni, w);
        const UniDev& d = U[u];
        const UniCtl& c = ctl[u];
        const int T = d.T;
        const int local = w - info->spt_off[u];
        const int r = local / T, t = local - r * T;
        Pt64* q = d.spos + UG_IDX((int64_t)r * T + t, (int64_t)d.S_max * T);
        int bc[3] = {0, 0, 0};
#pragma unroll
        for (int ax = 0; ax < 3; ax++) {
            if (ax < d.dim)
                bc[ax] = cell_of(q->c[ax], d.cell, d.gw) >> d.rblock_shift;
            else
                q->c[ax] = 0.0;
        }
        const uint64_t ep = (uint64_t)(uint32_t)c.epoch;
        const uint64_t old = atomicExch((unsigned long long*)rentry(d, t, lin_cell(bc, d.dim, rblock_gw(d))),
                                        (unsigned long long)((ep << 32) | (uint32_t)r));
        q->next = (old >> 32) == ep ? (int32_t)(uint32_t)old : -1;
        q->gid = -1;
    }
}

// 1+1D crossing rule in FP64: trajectory P[0..T) against the accepted paths `first`,
// first + step, ...; stops on *stop (another thread found a contact) outside group rounds.
// True on rejection; group rounds keep the single touched group in *g.
__device__ __forceinline__ bool cross64(const UniDev& d, const double* P, int64_t n_slots, int first, int step,
                                        bool group, int32_t* g, volatile int32_t* stop) {
    const int T = d.T;
    for (int64_t s = first; s < n_slots; s += step) {
        if (!group && *stop) return false;
        const Pt64* q = d.pts + UG_IDX(s * T + T - 1, d.slot_cap * T) + 1 - T;
        double d0 = torus_delta(P[0] - __ldcg(&q[0].c[0]));
        bool hit = hit1(d0, d.cell, d.inclusive);
        // the path's points 4 timesteps at a time (4 independent loads in flight)
        for (int t0 = 1; t0 < T && !hit; t0 += 4) {
            double qv[4];
#pragma unroll
            for (int k = 0; k < 4; k++) qv[k] = t0 + k < T ? __ldcg(&q[t0 + k].c[0]) : 0.0;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (hit || t0 + k >= T) break;
                const double d1 = torus_delta(P[t0 + k] - qv[k]);
                hit = hit1(d1, d.cell, d.inclusive) || crosses_step(d0, d1);
                d0 = d1;
            }
        }
        if (!hit) continue;
        if (!group) return true;
        const int32_t gq = __ldcg(&q[0].gid);
        if (*g == -1)
            *g = gq;
        else if (*g != gq)
            return true;
    }
    return false;
}

// The FP64 form's test of every candidate of the round (of the universes outside the
// tensor-core path in a mixed batch), a CTA per tile of 32 candidates:
//   generation   blocks, logarithms and sines spread over all threads, the normalisation
//                summed in ascending b by a thread per (candidate, axis); the knot stream is
//                drawn by a lane per candidate.  Term-ordered coefficient columns in the
//                CTA's own scratch (L2-resident), a column per (axis, candidate).
//   evaluation   16 or 32 timesteps at a time in endpoint-first order, as FP64 tensor
//                products over the live candidates' columns: eval64's bits.
//   test         the dilated filter for every (candidate, timestep), then the windows of
//                those it passes, then the chains of the occupied cells, each step over a
//                queue of the CTA (as in the mixed prefilter's epilogue).
// Bound by FP64 issue (about 110 FP64 instructions to generate a term) and the chains.  A
// warp per candidate, lanes over 32 timesteps, summed and (knot stream) drew on one lane;
// per job: 3+1 L2-ball T = 100, 200 k candidates 6.4 -> 3.45 ms; knot stream 2+1 T = 120,
// two terms, 200 k 4.9 -> 1.4; T = 65, all terms, 80 k 19.0 -> 1.7.
template <int D>
struct Test64 {
    const UniDev& U;
    int t;
    const double* P;
    int32_t* grp;  // group rounds: the candidate's group (shared by the CTA)
    int* nvis;
    Nbhd<D> nb;
    __device__ __forceinline__ Test64(const UniDev& U_, int t_, const double* P_, const int* c, int32_t* grp_, int* nvis_)
        : U(U_), t(t_), P(P_), grp(grp_), nvis(nvis_) {
        int z[D];
#pragma unroll
        for (int ax = 0; ax < D; ax++) z[ax] = 0;
        nbhd_make<D>(U, c, z, z, nb);
    }
    __device__ __forceinline__ bool operator()(int32_t p, int32_t& nx) {
        const Pt64* q = U.pts + UG_IDX((int64_t)p * U.T + t, U.slot_cap * U.T);
        const Pt64 Q = *q;
        nx = Q.next;
        ++*nvis;
        if (U.gkey_shift > 0) {  // coarse chains: only the points of the 3^D window cells count
#pragma unroll
            for (int ax = 0; ax < D; ax++)
                if (cyc_dist(cell_of(Q.c[ax], U.cell, U.gw), nb.v[ax][0], U.gw) >= nb.n[ax]) return false;
        }
        double X[3];
#pragma unroll
        for (int ax = 0; ax < D; ax++) X[ax] = P[ax];
        if (!pair_hit64(U, X, Q.c)) return false;
        if (!grp) return true;
        int cur = *(volatile int32_t*)grp;
        if (cur == -1) cur = atomicCAS(grp, -1, Q.gid);
        return cur != -1 && cur != Q.gid;
    }
};

// Draws of the knot stream (cuda/braid_knot.cu:111-166 order) by one lane per candidate:
// per axis the frequencies (perm, low bits) with their sign flips (bit 15), the uniforms of
// the weights (1 - u) and the phases; a2.  Frequencies are shuffled in shared memory.
__device__ __forceinline__ void knot_draws(const UniDev& d, uint64_t idx, int cand, uint16_t* perm, const Scratch64& sc,
                                           size_t cta, double* a2) {
    Xo r;
    r.seed(knot_seed(d.seed, idx));
    const int nw = d.nw, rows = 32 * d.dim;
    uint16_t* p = perm + cand;  // [j][32]
    for (int ax = 0; ax < d.dim; ax++) {
        const size_t o = cta * sc.knot_stride + (size_t)(ax * 32 + cand);
        if ((uint32_t)nw == d.modmax) {
            for (int j = 0; j < nw; j++) p[32 * j] = (uint16_t)(j + 2);
            for (int j = nw - 1; j > 0; j--) {
                const int k = (int)r.below((uint32_t)(j + 1));
                const uint16_t tmp = p[32 * j];
                p[32 * j] = p[32 * k];
                p[32 * k] = tmp;
            }
        } else {
            for (int j = 0; j < nw; j++) {
                int b = 0;
                bool dup = true;
                for (int guard = 0; dup && guard < 64; guard++) {
                    b = (int)r.below(d.modmax) + 2;
                    dup = false;
                    for (int k = 0; k < j; k++) dup |= p[32 * k] == b;
                }
                p[32 * j] = (uint16_t)b;
            }
        }
        for (int j = 0; j < nw; j++) sc.wgt[o + (size_t)j * rows] = 1.0 - r.f64();
        for (int j = 0; j < nw; j++) {
            const int b = p[32 * j];
            const bool neg = r.flip();
            if (!(b & 1)) sc.phase[o + (size_t)j * rows] = r.f64() * kPi;
            sc.freq[o + (size_t)j * rows] = (uint16_t)(b | (neg ? 0x8000 : 0));
        }
        a2[ax * 32 + cand] = d.pin ? 0.0 : (r.f64() * 2.0 - 1.0);
    }
}

__global__ void __launch_bounds__(kT64Threads, 2) k_test64(const UniDev* __restrict__ U, UniCtl* ctl, RoundInfo* info,
                                                           Scratch64 sc, int all) {
    __shared__ double s_P[kT64Pos], s_a2[96], s_sum[96];
    __shared__ uint2 s_q[kT64Tests];
    __shared__ __align__(16) uint2 s_cells[kT64Cells];
    __shared__ int32_t s_t[kMaxF], s_rej[32], s_grp[32], s_slot[32];
    __shared__ int s_nq, s_nc, s_item;
    __shared__ uint32_t s_live;
    static_assert(sizeof(s_cells) >= (size_t)kMaxF * 32 * sizeof(uint16_t), "the frequencies shuffle in the cells' place");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gl = lane >> 2, tl = lane & 3;
    volatile int32_t* vrej = s_rej;
    double* G = sc.coef + (size_t)blockIdx.x * sc.coef_stride;
    const int n_uni = info->n_uni, total = info->total_tiles * (kTile / 32);
    for (;;) {
        __syncthreads();  // the tile before is done with the shared arrays
        if (tid == 0) s_item = atomicAdd(&info->t64_next, 1);
        __syncthreads();
        const int item = s_item;
        if (item >= total) break;
        const int pos = find_uni(info->tile_off, n_uni, item >> 2);
        const int u = info->tile_uni[pos];
        const UniDev& d = U[u];
        UniCtl& c = ctl[u];
        const int off0 = (item - info->tile_off[pos] * 4) * 32;
        if ((!all && d.mx_ok) || off0 >= c.B) continue;
        const int nv = min(32, c.B - off0);
        const uint64_t idx0 = (uint64_t)(c.round_base + off0);
        const int dim = d.dim, T = d.T, F = d.F, K = d.K, rows = 32 * dim;
        const bool group = group_phase(d, c), cross = dim == 1 && d.cross1d;
        for (int t = tid; t < T; t += kT64Threads) s_t[t] = cross ? t : __ldg(d.order + t);
        if (tid < 32) {
            s_rej[tid] = tid < nv ? 0 : 1;
            s_grp[tid] = -1;
        }
        // ---- coefficients: G[k][ax * 32 + candidate]
        if (d.rng == RNG_KNOT) {
            const int nw = d.nw;
            const size_t o = (size_t)blockIdx.x * sc.knot_stride;
            if (warp == 0 && lane < nv)
                knot_draws(d, idx0 + lane, lane, reinterpret_cast<uint16_t*>(s_cells), sc, blockIdx.x, s_a2);
            const bool full = (uint32_t)nw == d.modmax;  // every frequency once
            if (!full)
                for (int e = tid; e < K * rows; e += kT64Threads) G[e] = 0.0;
            __syncthreads();
            for (int e = tid; e < nw * rows; e += kT64Threads) {
                if ((e % rows & 31) < nv) {
                    double* w = sc.wgt + o + e;
                    *w = -log(*w);
                }
            }
            __syncthreads();
            if (tid < rows && (tid & 31) < nv) {
                const double* w = sc.wgt + o + tid;
                double sum = 0.0;
#pragma unroll 4
                for (int j = 0; j < nw; j++) sum += w[(size_t)j * rows];
                s_sum[tid] = sum;
            }
            __syncthreads();
            // few terms may list a frequency twice: then a thread per row adds in term order
            const int nj = full ? nw : 1, step = full ? 1 : nw;
            for (int e = tid; e < nj * rows; e += kT64Threads) {
                const int row = e % rows, j0 = e / rows;
                if ((row & 31) >= nv) continue;
                for (int j = j0; j < j0 + step; j++) {
                    const size_t at = o + (size_t)j * rows + row;
                    const int fb = sc.freq[at], b = fb & 0x7fff, k = kseq_s(b);
                    double amp = sc.wgt[at] / s_sum[row] / (double)b;
                    if (fb & 0x8000) amp = -amp;
                    double* g = G + (size_t)k * rows + row;
                    if (full) *g = 0.0;
                    if (b & 1) {
                        *g += amp;
                    } else {
                        double sf, cf;
                        sincos(sc.phase[at], &sf, &cf);
                        if (full) g[rows] = 0.0;
                        add_even_term(*g, g[rows], amp, sf, cf);
                    }
                }
            }
        } else {
            const int np = (F >> 1) + 1;
            for (int e = tid; e < np * rows; e += kT64Threads) {
                const int row = e % rows, p = e / rows, ax = row >> 5;
                const uint4 o = philox_block(d.seed, idx0 + (row & 31), ax, p);
                if (p == 0) {
                    s_a2[row] = d.pin ? 0.0 : (double)o.x * (1.0 / 2147483648.0) - 1.0;
                    continue;
                }
                const int be = 2 * p, bo = 2 * p + 1;
                double* g = G + (size_t)kseq_s(be) * rows + row;
                const double Ee = -log(((double)o.x + 0.5) * (1.0 / 4294967296.0));
                g[0] = (o.z & 1u) ? -Ee : Ee;
                g[rows] = (double)(o.z >> 1) * (1.0 / 2147483648.0) * kPi;  // the phase, until the cosine term
                if (bo <= F) {
                    const double Eo = -log(((double)o.y + 0.5) * (1.0 / 4294967296.0));
                    g[2 * rows] = (o.w & 1u) ? -Eo : Eo;
                }
            }
            __syncthreads();
            if (tid < rows) {
                double sum = 0.0;
#pragma unroll 8
                for (int b = 2; b <= F; b++) sum += fabs(G[(size_t)kseq_s(b) * rows + tid]);
                s_sum[tid] = sum;
            }
            __syncthreads();
            for (int e = tid; e < (F - 1) * rows; e += kT64Threads) {
                const int row = e % rows, b = e / rows + 2;
                double* g = G + (size_t)kseq_s(b) * rows + row;
                const double v = *g;
                double amp = fabs(v) / s_sum[row] / (double)b;
                if (v < 0.0) amp = -amp;
                if (b & 1) {
                    *g = amp;
                } else {
                    double sf, cf;
                    sincos(g[rows], &sf, &cf);
                    *g = amp * cf;
                    g[rows] = amp * sf;
                }
            }
        }
        // ---- timesteps, in stages
        const int64_t cpt = cells_per_t(d);
        int nev = 0, nvis = 0;
        for (int c0 = 0; c0 < T;) {
            __syncthreads();  // coefficients written; the stage before is tested
            if (warp == 0) {
                const uint32_t lv = __ballot_sync(0xffffffffu, s_rej[lane] == 0);
                if ((lv >> lane) & 1u) s_slot[__popc(lv & ((1u << lane) - 1u))] = lane;
                if (lane == 0) {
                    s_live = lv;
                    s_nq = s_nc = 0;
                }
            }
            __syncthreads();
            const int nl = __popc(s_live);
            if (nl == 0) break;
            const int width = nl > 16 && !cross ? 16 : 32;  // positions: at most 32 x 3 x 16
            const int nc = min(width, T - c0), nn = (nc + 7) >> 3, L = nl * dim;
            // A warp per 16 rows x 8 or 16 timesteps: 16 once 8 would be more jobs than warps.  The
            // operands come from L2, 32 terms ahead with 8 timesteps, 16 with 16: with all timesteps
            // of a stage in one warp, eight terms ahead, a step of eight terms took 1700 cycles and
            // warps without rows idled (two-term knots 1.84 -> 1.43 ms per job, 3+1 L2-ball 3.9 ->
            // 3.45; 8 timesteps throughout: 1.44 and 3.96).
            auto product = [&](auto pair, int job) {
                constexpr int kN = decltype(pair)::value;
                const int nj = (nn + kN - 1) / kN, m0 = job / nj * 16, n0 = job % nj * 8 * kN;
                const int i0 = min(m0 + gl, L - 1), i1 = min(m0 + gl + 8, L - 1);
                const double* A0 = G + (i0 % dim) * 32 + s_slot[i0 / dim];
                const double* A1 = G + (i1 % dim) * 32 + s_slot[i1 / dim];
                const double* B[kN];
#pragma unroll
                for (int n = 0; n < kN; n++) B[n] = d.KT + s_t[min(c0 + n0 + 8 * n + gl, T - 1)];
                struct Step {
                    double a[4], b[kN][2];
                };
                auto fetch = [&](int k0, Step& st) {
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int k = k0 + 4 * h + tl;
                        const bool on = k < K;
                        st.a[2 * h] = on ? A0[(size_t)k * rows] : 0.0;
                        st.a[2 * h + 1] = on ? A1[(size_t)k * rows] : 0.0;
#pragma unroll
                        for (int n = 0; n < kN; n++) st.b[n][h] = on ? __ldg(B[n] + (size_t)k * d.Tpad) : 0.0;
                    }
                };
                constexpr int kAhead = 4 / kN;
                double acc[kN][4] = {};
                Step st[kAhead];
#pragma unroll
                for (int h = 0; h < kAhead; h++) fetch(8 * h, st[h]);
                for (int k0 = 0; k0 < K; k0 += 8 * kAhead) {
#pragma unroll
                    for (int h = 0; h < kAhead; h++) {
#pragma unroll
                        for (int n = 0; n < kN; n++) dmma_16x8x8(acc[n], st[h].a, st[h].b[n]);
                        fetch(k0 + 8 * (kAhead + h), st[h]);
                    }
                }
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const int i = m0 + gl + 8 * q;
                    if (i >= L) continue;
                    const double a2 = s_a2[(i % dim) * 32 + s_slot[i / dim]];
#pragma unroll
                    for (int n = 0; n < kN; n++)
#pragma unroll
                        for (int e = 0; e < 2; e++) {
                            const int col = n0 + 8 * n + 2 * tl + e;
                            if (col >= nc) continue;
                            const double X = torus_wrap(fma(acc[n][2 * q + e], __ldg(d.invsinz + s_t[c0 + col]), a2));
                            if (cross)  // the trajectories, behind the coefficients
                                G[(size_t)K * 32 + (size_t)s_slot[i] * T + c0 + col] = X;
                            else
                                s_P[i * width + col] = X;
                        }
                }
            };
            const int mt = (L + 15) / 16;
            if (mt * nn <= kT64Threads / 32)
                for (int job = warp; job < mt * nn; job += kT64Threads / 32) product(std::integral_constant<int, 1>{}, job);
            else
                for (int job = warp; job < mt * ((nn + 1) / 2); job += kT64Threads / 32) product(std::integral_constant<int, 2>{}, job);
            __syncthreads();
            c0 += width;
            if (cross) continue;
            const int tb = c0 - width;
            // the filter
            for (int i = tid; i < nl * nc; i += kT64Threads) {
                const int sl = i / nc, j = i - sl * nc;
                nev++;
                int cc[3] = {0, 0, 0};
                int64_t lin = 0;
#pragma unroll
                for (int ax = 0; ax < 3; ax++)
                    if (ax < dim) {
                        cc[ax] = cell_of(s_P[(sl * dim + ax) * width + j], d.cell, d.gw);
                        lin = lin * d.occ1_gw + (cc[ax] >> d.occ1_shift);
                    }
                const int64_t b = (int64_t)s_t[tb + j] * d.occ1_per_t + lin;
                if ((__ldg(d.occ1 + UG_IDX(b >> 5, d.occ1_words)) >> (b & 31)) & 1u) {
                    const int at = atomicAdd(&s_nq, 1);
                    s_q[UG_IDX(at, kT64Tests)] = make_uint2((uint32_t)(sl << 8 | j), (uint32_t)(cc[0] | cc[1] << 10 | cc[2] << 20));
                }
            }
            __syncthreads();
            // windows, then chains
            auto run = [&](auto dc) {
                constexpr int D = decltype(dc)::value;
                auto with = [&](int e, auto&& f) {
                    const uint2 q = s_q[e];
                    const int sl = q.x >> 8, j = q.x & 255, cand = s_slot[sl];
                    if (vrej[cand]) return;
                    double P[D];
                    int cc[D];
#pragma unroll
                    for (int ax = 0; ax < D; ax++) {
                        P[ax] = s_P[(sl * D + ax) * width + j];
                        cc[ax] = (q.y >> (10 * ax)) & 1023u;
                    }
                    Test64<D> test(d, s_t[tb + j], P, cc, group ? s_grp + cand : nullptr, &nvis);
                    if (f(test)) vrej[cand] = 1;
                };
                const int nq = s_nq;
                for (int e = tid; e < nq; e += kT64Threads)
                    with(e, [&](Test64<D>& test) {
                        if constexpr (D == 1) {
                            return nbhd_scan<1>(d, test.t, test.nb, cpt, test);
                        } else {
                            auto put = [&](int o0, int o1, int o2) {
                                const int at = atomicAdd(&s_nc, 1);
                                if (at < kT64Cells) {
                                    s_cells[at] = make_uint2((uint32_t)e | (uint32_t)o0 << 16, (uint32_t)o1 | (uint32_t)o2 << 16);
                                    return false;
                                }
                                if constexpr (D == 3)
                                    return brick_cell_visit(d, test.t, test.nb, cpt, o0, o1, o2, test);
                                else
                                    return brick_cell_visit2(d, test.t, test.nb, cpt, o0, o1, test);
                            };
                            if constexpr (D == 3)
                                return nbhd_cells3(d, test.t, test.nb, put);
                            else
                                return nbhd_cells2(d, test.t, test.nb, [&](int o0, int o1) { return put(o0, o1, 0); });
                        }
                    });
                __syncthreads();
                if constexpr (D > 1) {
                    const int ncell = min(s_nc, kT64Cells);
                    for (int i = tid; i < ncell; i += kT64Threads) {
                        const uint2 cl = s_cells[i];
                        with(cl.x & 0xffffu, [&](Test64<D>& test) {
                            if constexpr (D == 3)
                                return brick_cell_visit(d, test.t, test.nb, cpt, (int)(cl.x >> 16), (int)(cl.y & 0xffffu),
                                                        (int)(cl.y >> 16), test);
                            else
                                return brick_cell_visit2(d, test.t, test.nb, cpt, (int)(cl.x >> 16), (int)(cl.y & 0xffffu),
                                                         test);
                        });
                    }
                }
            };
            if (dim == 3)
                run(std::integral_constant<int, 3>{});
            else if (dim == 2)
                run(std::integral_constant<int, 2>{});
            else
                run(std::integral_constant<int, 1>{});
        }
        if (cross) {  // eight threads per candidate over the accepted paths
            const int cand = tid >> 3, part = tid & 7;
            __syncthreads();
            if (cand < nv) {
                int32_t g = -1;
                if (part == 0) nev = T;
                if (cross64(d, G + (size_t)K * 32 + (size_t)cand * T, c.n_slots, part, 8, group, &g, vrej + cand)) vrej[cand] = 1;
                if (group && g != -1) {
                    const int32_t old = atomicCAS(&s_grp[cand], -1, g);
                    if (old != -1 && old != g) vrej[cand] = 1;
                }
            }
        }
        for (int o = 16; o > 0; o >>= 1) nev += __shfl_xor_sync(0xffffffffu, nev, o);
        for (int o = 16; o > 0; o >>= 1) nvis += __shfl_xor_sync(0xffffffffu, nvis, o);
        if (lane == 0) {
            if (nev) atomicAdd((unsigned long long*)&c.evals_fp64, (unsigned long long)nev);
            if (all && nev) atomicAdd((unsigned long long*)&c.evals, (unsigned long long)nev);
            if (all && nvis) atomicAdd((unsigned long long*)&c.visits, (unsigned long long)nvis);
        }
        __syncthreads();
        if (warp == 0) {
            const uint32_t sb = __ballot_sync(0xffffffffu, s_rej[lane] == 0);
            if (lane == 0) d.surv_bits[UG_IDX(off0 >> 5, d.B_max / 32)] = sb;
            if (d.group_mode != GROUP_NONE && lane < nv) d.g0[UG_IDX(off0 + lane, d.B_max)] = s_grp[lane];
        }
    }
}

// warp_gen64_axis of all axes by a whole block, as term-ordered rows (row pitch kRowK):
// blocks, logarithms and sines spread over the threads, the normalisation
// summed in ascending b by one lane per axis.
__device__ __forceinline__ void block_gen64(const UniDev& d, uint64_t idx, double* rows, double* phase, double* a2,
                                            double* sums) {
    const int F = d.F, np = (F >> 1) + 1;
    for (int e = threadIdx.x; e < d.dim * np; e += blockDim.x) {
        const int ax = e / np, p = e - ax * np;
        double* row = rows + ax * kRowK;
        const uint4 o = philox_block(d.seed, idx, ax, p);
        if (p == 0) {
            a2[ax] = d.pin ? 0.0 : (double)o.x * (1.0 / 2147483648.0) - 1.0;
            continue;
        }
        const int be = 2 * p, bo = 2 * p + 1;
        const double Ee = -log(((double)o.x + 0.5) * (1.0 / 4294967296.0));
        row[kseq_s(be)] = (o.z & 1u) ? -Ee : Ee;
        phase[ax * kMaxF + be - 1] = (double)(o.z >> 1) * (1.0 / 2147483648.0) * kPi;
        if (bo <= F) {
            const double Eo = -log(((double)o.y + 0.5) * (1.0 / 4294967296.0));
            row[kseq_s(bo)] = (o.w & 1u) ? -Eo : Eo;
        }
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0 && (int)(threadIdx.x >> 5) < d.dim) {
        const double* row = rows + (threadIdx.x >> 5) * kRowK;
        double sum = 0.0;
#pragma unroll 4
        for (int b = 2; b <= F; b++) sum += fabs(row[kseq_s(b)]);
        sums[threadIdx.x >> 5] = sum;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < d.dim * (F - 1); e += blockDim.x) {
        const int ax = e / (F - 1), b = e - ax * (F - 1) + 2;
        double* row = rows + ax * kRowK + kseq_s(b);
        const double v = row[0];
        double amp = fabs(v) / sums[ax] / (double)b;
        if (v < 0.0) amp = -amp;
        if (b & 1) {
            row[0] = amp;
        } else {
            double sf, cf;
            sincos(phase[ax * kMaxF + b - 1], &sf, &cf);
            row[0] = amp * cf;
            row[1] = amp * sf;
        }
    }
    __syncthreads();
}

// The mixed form's retest, one block of four warps per undecided candidate (few per round:
// one candidate's latency bounds the launch).  Only the timesteps of its mask are
// evaluated, 32 at a time, eight per warp as FP64 tensor products (the axes are rows), with
// eval64's bits.  Candidates without a mask (the crossing rule, or beyond the
// masks' room) are tested at all timesteps.  Per round, against a lane per
// timestep of all T: 2+1 unique groups T = 256 (380 candidates, ~60 timesteps each)
// 167 -> 108 us, 3+1 T = 128 (310) 50 -> 23 us.
__global__ void __maxnreg__(128) k_retest(const UniDev* __restrict__ U, UniCtl* ctl, RoundInfo* info,
                                          RetestQueue rq) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int32_t s_hit, s_g, s_nt;
    __shared__ int32_t s_t[kMaxF];
    __shared__ double s_P[32][3], s_sum[3], a2[3], s_traj[kMaxF];
    double* rows = (double*)smem_raw;  // [3][kRowK], phases [3][kMaxF]
    double* phase = rows + 3 * kRowK;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gl = lane >> 2, tl = lane & 3;
    volatile int32_t* vhit = &s_hit;
    const int total = min(info->total_gray, rq.cap);
    for (int item = blockIdx.x; item < total; item += gridDim.x) {
        const int2 it = rq.item[item];
        const UniDev& d = U[it.x];
        UniCtl& c = ctl[it.x];
        const int off = it.y, T = d.T, K = d.K, dim = d.dim;
        const uint64_t idx = (uint64_t)(c.round_base + off);
        const bool group = group_phase(d, c), cross = dim == 1 && d.cross1d;
        const bool masked = !cross && item < rq.mask_cap;
        block_gen64(d, idx, rows, phase, a2, s_sum);
        if (tid == 0) {
            s_hit = 0;
            // masked: the group that the decided timesteps touched
            s_g = masked && group ? d.g0[UG_IDX(off, d.B_max)] : -1;
        }
        // the timesteps to evaluate
        if (masked) {
            if (warp == 0) {
                const uint32_t* m = reinterpret_cast<const uint32_t*>(rq.mask + 2 * (int64_t)item);
                uint32_t w = lane < kMaskWords ? m[lane] : 0u;
                int incl = __popc(w);
                const int mine = incl;
                for (int o = 1; o < kMaskWords; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += v;
                }
                for (int at = incl - mine; w; w &= w - 1) s_t[at++] = lane * 32 + __ffs(w) - 1;
                if (lane == kMaskWords - 1) s_nt = incl;
            }
        } else {
            for (int t = tid; t < T; t += blockDim.x) s_t[t] = cross ? t : __ldg(d.order + t);
            if (tid == 0) s_nt = T;
        }
        __syncthreads();
        const int nt = s_nt;
        const int64_t cpt = cells_per_t(d);
        int32_t g = s_g;
        bool hitl = false;
        int nev = 0;
        for (int t0 = 0; t0 < nt; t0 += 32) {
            const int n = min(32, nt - t0);
            if (8 * warp < n) {
                const int q = 8 * warp + gl;  // this lane's timestep as a column of B
                const double* B = d.KT + s_t[t0 + min(q, n - 1)];
                const double* A = rows + (gl < dim ? gl * kRowK : 0);
                double acc[2] = {0.0, 0.0};
                double bv[2][8];  // two batches of eight steps' basis values
                auto fetch = [&](int k0, double* v) {
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const int k = k0 + 4 * j + tl;
                        v[j] = k < K ? __ldg(B + (int64_t)k * d.Tpad) : 0.0;
                    }
                };
                fetch(0, bv[0]);
                for (int k0 = 0; k0 < K; k0 += 64) {
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        fetch(k0 + 32 * (h + 1), bv[h ^ 1]);
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            const int k = k0 + 32 * h + 4 * j + tl;
                            dmma_8x8x4(acc, gl < dim && k < K ? A[k] : 0.0, bv[h][j]);
                        }
                    }
                }
                if (gl < dim)
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        const int col = 8 * warp + 2 * tl + j;
                        if (col < n) s_P[col][gl] = torus_wrap(fma(acc[j], __ldg(d.invsinz + s_t[t0 + col]), a2[gl]));
                    }
            }
            __syncthreads();
            nev += n;
            // a timestep's contacts on a lane of its own, spread over the warps
            const int e = (lane >> 2) * 4 + warp;
            if (cross) {
                if (tid < n) s_traj[t0 + tid] = s_P[tid][0];
            } else if ((lane & 3) == 0 && e < n) {
                double P[3];
                for (int ax = 0; ax < 3; ax++) P[ax] = ax < dim ? s_P[e][ax] : 0.0;
                if (contacts64(d, s_t[t0 + e], P, group, &g, cpt, nullptr)) {
                    hitl = true;
                    *vhit = 1;
                }
            }
            __syncthreads();
            if (*vhit) break;
        }
        if (cross) {
            hitl = cross64(d, s_traj, c.n_slots, tid, blockDim.x, group, &g, vhit);
            if (hitl) *vhit = 1;
        }
        // any rejection, or (group rounds) two distinct groups touched
        if (group && g != -1) {
            const int32_t old = atomicCAS(&s_g, -1, g);
            if (old != -1 && old != g) hitl = true;
        }
        const bool rej = __syncthreads_or(hitl);
        if (tid == 0) {
            if (nev) atomicAdd((unsigned long long*)&c.evals_fp64, (unsigned long long)nev);
            if (!rej) atomicOr(&d.surv_bits[UG_IDX(off >> 5, d.B_max / 32)], 1u << (off & 31));
            if (d.group_mode != GROUP_NONE) d.g0[UG_IDX(off, d.B_max)] = s_g;
        }
        __syncthreads();
    }
}

// The set of earlier survivors r' < r that survivor r touches (Chebyshev contact at any
// timestep; plus crossings in 1+1D).  A warp per survivor, lanes over timesteps; a block of
// four warps where the round's survivors leave most of them idle.  A lane's chain of
// dependent loads (its point, the round table's heads, the heads' points, the chains)
// bounds it, so the loads of each link are issued together, four blocks of the window at
// a time.  Against one probe after another and a warp per survivor, per round: 2+1
// T = 256, 270 survivors 101 -> 30 us; 3+1 T = 128, 1800 65 -> 35 us; a 32-universe
// batch 133 -> 119 us.  A block serves a survivor up to two per resident CTA: beyond that
// the warps are all busy and short T leaves a block's lanes without a timestep.
__global__ void __launch_bounds__(128) k_conflicts(const UniDev* __restrict__ U, UniCtl* ctl,
                                                    RoundInfo* info) {
    __shared__ int32_t s_cnt[4], s_item;
    __shared__ int32_t s_list[4][kConflictCap];
    __shared__ uint32_t s_seen[4][kSmaxCap / 32];  // earlier survivors already listed
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int n_uni = info->n_uni, total = info->total_surv;
    const bool wide = total <= 2 * (int)gridDim.x;
    const int gt = wide ? threadIdx.x : lane, gn = wide ? 128 : 32;  // thread of the survivor's group
    volatile int32_t* cnt = &s_cnt[wide ? 0 : wib];
    volatile int32_t* lst = s_list[wide ? 0 : wib];
    uint32_t* seen = s_seen[wide ? 0 : wib];
    auto sync = [&]() {
        if (wide)
            __syncthreads();
        else
            __syncwarp();
    };
    // Survivors are handed out one at a time, costliest universes first (their cost
    // differs by the timesteps and dimension); the next one is claimed when an item
    // starts so the atomic's latency hides behind the item.
    int item = 0, next = 0;
    auto settle = [&](int v) -> int {  // the value of the group's first thread
        if (!wide) return __shfl_sync(0xffffffffu, v, 0);
        if (threadIdx.x == 0) s_item = v;
        __syncthreads();
        return s_item;
    };
    if (gt == 0) item = atomicAdd(&info->confl_next, 1);
    item = settle(item);
    while (item < total) {
        if (gt == 0) next = atomicAdd(&info->confl_next, 1);
        const int pos = find_uni(info->surv_off_o, n_uni, item);
        const int u = info->tile_uni[pos];
        const int r = item - info->surv_off_o[pos];
        const UniDev& d = U[u];
        UniCtl& c = ctl[u];
        const int T = d.T;
        if (gt == 0) *cnt = 0;
        for (int i = gt; i <= r >> 5; i += gn) seen[i] = 0u;
        sync();
        // each earlier survivor once (it is met at many timesteps): with a search of the
        // list instead, lanes that met it together listed it twice and overfilled the list
        auto add = [&](int32_t r2) {
            const uint32_t bit = 1u << (r2 & 31);
            if (atomicOr(&seen[UG_IDX(r2 >> 5, kSmaxCap / 32)], bit) & bit) return;
            const int at = atomicAdd((int32_t*)cnt, 1);
            if (at < kConflictCap) lst[at] = r2;
        };
        if (d.dim == 1 && d.cross1d) {
            const Pt64* P = d.spos + UG_IDX((int64_t)r * T + T - 1, (int64_t)d.S_max * T) + 1 - T;
            for (int r2 = gt; r2 < r; r2 += gn) {
                const Pt64* Q = d.spos + UG_IDX((int64_t)r2 * T + T - 1, (int64_t)d.S_max * T) + 1 - T;
                double d0 = torus_delta(P[0].c[0] - Q[0].c[0]);
                bool hit = hit1(d0, d.cell, d.inclusive);
                // both paths' points 4 timesteps at a time (independent loads in flight)
                for (int t0 = 1; t0 < T && !hit; t0 += 4) {
                    double pv[4], qv[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        pv[k] = t0 + k < T ? P[t0 + k].c[0] : 0.0;
                        qv[k] = t0 + k < T ? Q[t0 + k].c[0] : 0.0;
                    }
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        if (hit || t0 + k >= T) break;
                        const double d1 = torus_delta(pv[k] - qv[k]);
                        hit = hit1(d1, d.cell, d.inclusive) || crosses_step(d0, d1);
                        d0 = d1;
                    }
                }
                if (hit) add(r2);
            }
        } else {
            const int gw = d.gw, gwb = rblock_gw(d), rbs = d.rblock_shift;
            for (int t = gt; t < T; t += gn) {
                const Pt64 P = d.spos[UG_IDX((int64_t)r * T + t, (int64_t)d.S_max * T)];
                const Pt64* St = d.spos + t;
                // distinct round-table blocks of the 3 neighbour cells per axis:
                // bl[ax] packs up to three 10-bit block coordinates, nbk[ax] counts them
                // (registers only: every index below is a compile-time constant)
                uint32_t bl[3] = {0u, 0u, 0u};
                int nbk[3] = {1, 1, 1};
#pragma unroll
                for (int ax = 0; ax < 3; ax++) {
                    if (ax < d.dim) {
                        const int c0 = cell_of(P.c[ax], d.cell, gw);
                        const uint32_t v0 = (uint32_t)((c0 == 0 ? gw - 1 : c0 - 1) >> rbs);
                        const uint32_t v1 = (uint32_t)(c0 >> rbs);
                        const uint32_t v2 = (uint32_t)((c0 == gw - 1 ? 0 : c0 + 1) >> rbs);
                        uint32_t pk = v0;
                        int n = 1;
                        if (v1 != v0) pk |= v1 << (10 * n++);
                        if (v2 != v0 && v2 != v1) pk |= v2 << (10 * n++);
                        bl[ax] = pk;
                        nbk[ax] = n;
                    }
                }
                auto test = [&](int32_t r2, const Pt64& Q) {
                    if (r2 < r && pair_hit64(d, P.c, Q.c)) add(r2);
                };
                const int nc = nbk[0] * nbk[1] * nbk[2];
                for (int c0 = 0; c0 < nc; c0 += 4) {  // block combinations, four at a time
                    int32_t h[4];
                    Pt64 Q[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const int cc = c0 + k, i2 = cc % nbk[2], i01 = cc / nbk[2], i1 = i01 % nbk[1], i0 = i01 / nbk[1];
                        const int bc[3] = {(int)((bl[0] >> (10 * i0)) & 1023u), (int)((bl[1] >> (10 * i1)) & 1023u),
                                           (int)((bl[2] >> (10 * i2)) & 1023u)};
                        h[k] = -1;
                        if (cc < nc) h[k] = rtab_head(d, c.epoch, t, lin_cell(bc, d.dim, gwb));
                    }
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        if (h[k] >= 0) Q[k] = St[UG_IDX((int64_t)h[k] * T, (int64_t)d.S_max * T)];
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        if (h[k] < 0) continue;
                        test(h[k], Q[k]);
                        for (int32_t r2 = Q[k].next; r2 >= 0;) {
                            const Pt64 N = St[UG_IDX((int64_t)r2 * T, (int64_t)d.S_max * T)];
                            test(r2, N);
                            r2 = N.next;
                        }
                    }
                }
            }
        }
        sync();
        // more than kConflictCap contacts: the list keeps kConflictCap of them and the
        // count says so; the resolver rejects on any admitted one and otherwise stops
        // the round at this survivor
        const int n = *cnt;
        const int ns = n < kConflictCap ? n : kConflictCap;
        for (int i = gt; i < ns; i += gn) d.clist[UG_IDX((int64_t)r * kConflictCap + i, (int64_t)d.S_max * kConflictCap)] = lst[i];
        if (gt == 0) d.ccount[UG_IDX(r, d.S_max)] = n;
        sync();
        item = settle(next);
    }
}

// ------------------------------------------------------------- resolver

// One warp per universe: survivors in index order; admit survivor r iff the
// sequential-RSA rule holds against the round's earlier admissions.  32 survivors are a
// window; the next window's contact lists come into shared memory while one is decided,
// and the counts (and pre-round groups) a window before that, so that no step waits for
// global memory: 3+1 T = 128, 1800 survivors 67 -> 34 us a round; unique groups at T = 256,
// 270 survivors 115 -> 62 us, 51 us since they are decided from registers.
__global__ void __launch_bounds__(32) k_greedy(const UniDev* __restrict__ U, UniCtl* ctl,
                                               RoundInfo* info) {
    extern __shared__ __align__(16) int32_t greedy_smem[];
    int32_t* acc_s = greedy_smem;
    int32_t* gid_s = acc_s + kSmaxCap;
    int32_t* lists = gid_s + kSmaxCap;  // [2][32][kListPitch]
    const int u = blockIdx.x;
    const int lane = threadIdx.x;
    const UniDev& d = U[u];
    UniCtl& c = ctl[u];
    if (c.B == 0) return;
    const int S = c.S;
    const int S_eff = c.trunc < S ? c.trunc : S;
    const bool group = group_phase(d, c);
    const bool unique_group = d.group_mode == GROUP_UNIQUE;
    const int64_t room = d.slot_cap - c.n_slots, n_slots = c.n_slots, max_n = c.phase == 1 ? c.max_n : 0;
    int k = 0, stop_at = S_eff;
    int64_t n_unique = c.n_unique, n_sub = c.n_sub;
    bool grow = false, hit_max = false, undecided = false;
    auto load_cnt = [&](int r0) { return r0 + lane < S_eff ? d.ccount[UG_IDX(r0 + lane, d.S_max)] : 0; };
    auto load_g0 = [&](int r0) {
        return group && r0 + lane < S_eff
                   ? d.g0[UG_IDX(d.surv_off[UG_IDX(r0 + lane, d.S_max + 1)], d.B_max)]
                   : -1;
    };
    auto stage = [&](int r0, int n_all) {  // this lane's survivor's list, 16 bytes at a time
        int32_t* dst = lists + ((r0 >> 5) & 1) * 32 * kListPitch + lane * kListPitch;
        const int32_t* src = d.clist + UG_IDX((int64_t)(r0 + lane < S_eff ? r0 + lane : 0) * kConflictCap,
                                              (int64_t)d.S_max * kConflictCap);
        const int n = min(n_all, (int)kConflictCap);
        for (int i = 0; i < n; i += 4)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                             (uint32_t)__cvta_generic_to_shared(dst + i)),
                         "l"(src + i)
                         : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int cnt0 = load_cnt(0), cnt1 = load_cnt(32), g00 = load_g0(0), g01 = load_g0(32);
    stage(0, cnt0);
    bool stopped = false;
    for (int r0 = 0; r0 < S_eff && !stopped; r0 += 32) {
        const int cnt2 = load_cnt(r0 + 64), g02 = load_g0(r0 + 64);
        stage(r0 + 32, cnt1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        const int32_t* win = lists + ((r0 >> 5) & 1) * 32 * kListPitch;
        const int nvalid = min(32, S_eff - r0);
        int lim = nvalid;  // survivors of the window that are decided
        if (!group) {
            // Plain rounds: each lane gathers its survivor's listed contacts -- admitted ones
            // from earlier windows (certain rejection) and a bit mask of the earlier lanes of
            // this one -- and the warp then decides the 32 in index order from those masks:
            // the same decisions as one at a time, as group rounds take them.
            const int r = r0 + lane;
            uint32_t dep = 0;
            bool ext = false;
            const bool over = cnt0 > kConflictCap;
            const int n = over ? kConflictCap : cnt0;
            for (int i = 0; i < n; i++) {
                const int r2 = win[lane * kListPitch + i];
                if (r2 < r0)
                    ext |= acc_s[UG_IDX(r2, kSmaxCap)] >= 0;
                else
                    dep |= 1u << (r2 - r0);
            }
            // In-order greedy over the window's lanes: a lane decides once every lane it
            // depends on has decided (dependencies point to lower lanes only, so the
            // lowest undecided lane is always ready; one pass per link of the longest
            // dependency chain, usually one).
            const uint32_t valid = nvalid >= 32 ? 0xffffffffu : ((1u << nvalid) - 1u);
            uint32_t und = valid, accm = 0;
            while (und) {
                const bool ready = ((und >> lane) & 1u) && !(dep & und);
                accm |= __ballot_sync(0xffffffffu, ready && !ext && !(dep & accm));
                und &= ~__ballot_sync(0xffffffffu, ready);
            }
            // Where the one-at-a-time scan would stop: at lane j it first checks the
            // room left (stop before j), then an admitted j with an over-full list
            // (undecided: stop before j), then the unique cap (stop after j).
            const int acc_before = __popc(accm & ((1u << lane) - 1u));
            const bool mine = (accm >> lane) & 1u;
            const uint32_t b_room = __ballot_sync(0xffffffffu, lane < nvalid && k + acc_before >= room);
            const uint32_t b_over = __ballot_sync(0xffffffffu, mine && over);
            const uint32_t b_max = __ballot_sync(0xffffffffu, mine && max_n > 0 && n_unique + acc_before + 1 >= max_n);
            if (b_room | b_over | b_max) {
                const int j = __ffs(b_room | b_over | b_max) - 1;
                stopped = true;
                lim = j;
                if ((b_room >> j) & 1u) {
                    grow = true;
                } else if ((b_over >> j) & 1u) {
                    undecided = true;
                } else {
                    lim = j + 1;
                    hit_max = true;
                }
            }
            if (lane < lim) {
                const int rank = k + acc_before;
                acc_s[UG_IDX(r, kSmaxCap)] = mine ? rank : -1;
                gid_s[UG_IDX(r, kSmaxCap)] = mine ? (int32_t)(n_slots + rank) : -1;
            }
            const int taken = __popc(accm & (lim >= 32 ? 0xffffffffu : ((1u << lim) - 1u)));
            k += taken;
            n_unique += taken;
        } else {
            // Group rounds: each lane first gathers what its survivor's list says of earlier
            // windows -- the one group its contacts (and the pre-round test) name, or that
            // there are two -- and the mask of earlier lanes it touches.  The 32 are then
            // decided in index order from registers (a lane's contacts within the window by
            // its mask), some 70 cycles each instead of a list walk of 450.
            const int r = r0 + lane;
            const bool over = cnt0 > kConflictCap;  // the list holds only kConflictCap contacts
            const int n = over ? kConflictCap : cnt0;
            int32_t eg = g00, my_acc = -1, my_gid = -1;
            bool two = false;
            uint32_t dep = 0;
            const int4* list = reinterpret_cast<const int4*>(win + lane * kListPitch);
            for (int i = 0; i < n; i += 4) {
                const int4 l4 = list[i >> 2];
                const int r4[4] = {l4.x, l4.y, l4.z, l4.w};
                int32_t g4[4];
#pragma unroll
                for (int q = 0; q < 4; q++)  // a rejected survivor's group is -1
                    g4[q] = i + q < n && r4[q] < r0 ? gid_s[UG_IDX(r4[q], kSmaxCap)] : -1;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    if (i + q < n && r4[q] >= r0) dep |= 1u << (r4[q] - r0);
                    if (g4[q] == -1) continue;
                    two |= eg != -1 && g4[q] != eg;
                    if (eg == -1) eg = g4[q];
                }
            }
            const uint32_t m_two = __ballot_sync(0xffffffffu, two), m_over = __ballot_sync(0xffffffffu, over);
            for (int j = 0; j < nvalid; j++) {
                if (k >= room) {
                    lim = j;
                    grow = stopped = true;
                    break;
                }
                // union of the lane's group and those of admitted contacts in the window
                const uint32_t dj = __shfl_sync(0xffffffffu, dep, j);
                int32_t first = __shfl_sync(0xffffffffu, eg, j);
                const int32_t mine = ((dj >> lane) & 1u) && my_acc >= 0 ? my_gid : -1;
                const uint32_t has = __ballot_sync(0xffffffffu, mine != -1);
                if (first == -1 && has) first = __shfl_sync(0xffffffffu, mine, __ffs(has) - 1);
                const bool both = ((m_two >> j) & 1u) || (has && __any_sync(0xffffffffu, mine != -1 && mine != first));
                if (!both && ((m_over >> j) & 1u)) {  // unlisted contacts might add a group: decide next round
                    lim = j;
                    undecided = stopped = true;
                    break;
                }
                // two groups touched: rejected; none: founds one, or (subpath) rejected
                const bool founds = !both && first == -1;
                const bool accept = !both && (first != -1 || unique_group);
                if (lane == j && accept) {
                    my_acc = k;
                    my_gid = founds ? (int32_t)(n_slots + k) : first;
                }
                if (accept) {
                    k++;
                    if (founds)
                        n_unique++;
                    else
                        n_sub++;
                    if (max_n > 0 && n_unique >= max_n) {
                        lim = j + 1;
                        hit_max = stopped = true;
                        break;
                    }
                }
            }
            if (lane < lim) {
                acc_s[UG_IDX(r, kSmaxCap)] = my_acc;
                gid_s[UG_IDX(r, kSmaxCap)] = my_gid;
            }
        }
        __syncwarp();
        if (r0 + lane < S) {
            const bool in = lane < lim;
            d.acc_rank[UG_IDX(r0 + lane, d.S_max)] = in ? acc_s[UG_IDX(r0 + lane, kSmaxCap)] : -1;
            d.sgid[UG_IDX(r0 + lane, d.S_max)] = in ? gid_s[UG_IDX(r0 + lane, kSmaxCap)] : -1;
        }
        if (stopped) stop_at = r0 + lim;
        cnt0 = cnt1;
        cnt1 = cnt2;
        g00 = g01;
        g01 = g02;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // survivors beyond the last window are not decided this round
    for (int r = (stop_at + 31) / 32 * 32 + lane; r < S; r += 32) {
        d.acc_rank[UG_IDX(r, d.S_max)] = -1;
        d.sgid[UG_IDX(r, d.S_max)] = -1;
    }
    if (lane != 0) return;
    int64_t next;
    if (hit_max)
        next = c.round_base + d.surv_off[UG_IDX(stop_at - 1, d.S_max + 1)] + 1;
    else if (stop_at < c.S_raw)
        next = c.round_base + d.surv_off[UG_IDX(stop_at, d.S_max + 1)];
    else
        next = c.round_base + c.B;
    const int64_t used = next - c.round_base;
    c.stop_at = stop_at;
    c.n_slots_prev = c.n_slots;
    c.n_slots += k;
    c.n_unique = n_unique;
    c.n_sub = n_sub;
    c.accepted_round = k;
    c.next_cand = next;
    c.attempts = next;
    c.last_used = used;
    c.rounds++;
    if (grow) c.state = ST_GROW;
    // round-size adaptation (the reference steers toward 64..512 survivors for
    // its serial host admission, braid_cuda.cu:921-924; the device resolver
    // takes up to S_max, so steer toward the survivor capacity instead).
    // Admission results do not depend on it.
    if (undecided && c.round_B > kTile)  // crowded in-round contacts: smaller rounds
        c.round_B = max(c.round_B >> 1, kTile);
    else if (c.S_raw > d.S_max && c.round_B > c.B_min)
        c.round_B = max(c.round_B >> 1, c.B_min);
    else if (c.S_raw < d.S_max / 4 && c.round_B < c.B_cap)
        c.round_B = min(c.round_B << 1, c.B_cap);
}

// ---------------------------------------------------------------- commit

// Appends slot to the chain of cell lin at timestep t; *old_head gets the
// previous head.  *new_key is set when the insert claimed a new hash key (the
// caller counts them into UniCtl::hash_used).
__device__ __forceinline__ void grid_insert(const UniDev& d, UniCtl& c, int t, int64_t lin, uint32_t fbit,
                                            int64_t cpt, int32_t slot, int32_t* old_head, bool* new_key,
                                            bool* new_cell) {
    if (d.grid_kind == GRID_DENSE) {
        *old_head = atomicExch(d.heads + UG_IDX((int64_t)t * cpt + lin, d.dense_cells), slot);
        *new_cell = *old_head < 0;
        return;
    }
    const uint64_t key = ((uint64_t)t << 40) | (uint64_t)lin;
    uint64_t h = mix64(key) & d.hmask;
    for (uint64_t probe = 0; probe <= d.hmask; probe++) {
        unsigned long long* kp = &d.hslot[h].x;
        const ulonglong2 sv = __ldcg(&d.hslot[h]);  // key and y in one load
        uint64_t k = sv.x;
        if (k == kEmptyKey) {
            const uint64_t prev = atomicCAS(kp, kEmptyKey, key);
            if (prev == kEmptyKey) {
                *new_key = true;
                k = key;
            } else {
                k = prev;
            }
        }
        if (k == key) {
            // y: chain head (low half), complemented cell mask of a coarse key (high half)
            if (!fbit) {
                *old_head = (int32_t)atomicExch(reinterpret_cast<unsigned int*>(&d.hslot[h].y), (unsigned int)slot);
                *new_cell = *old_head < 0;
                return;
            }
            // coarse key: the new head and the cell's bit in one compare-and-swap of y
            // (a failed swap means another insert into this coarse cell went first)
            unsigned long long* yp = &d.hslot[h].y;
            unsigned long long cur = sv.y;
            for (int it = 0; it < (1 << 20); it++) {
                const unsigned long long nv = (((cur >> 32) & ~(unsigned long long)fbit) << 32) | (uint32_t)slot;
                const unsigned long long prev = atomicCAS(yp, cur, nv);
                if (prev == cur) {
                    *old_head = (int32_t)(uint32_t)cur;
                    *new_cell = ((cur >> 32) & fbit) != 0ull;
                    return;
                }
                cur = prev;
            }
            break;
        }
        h = (h + 1) & d.hmask;
    }
    *old_head = -1;
    *new_cell = false;
    c.err_code = 3;  // hash full (host keeps the load factor below 1/2), or no progress
    c.state = ST_ERROR;
}

// Sets bits of an occupancy bitmap.  Bits are only ever set during a run, so a word that
// holds them needs no atomic (most do: an unconditional atomicOr took k_commit from 56 to
// 63 ms in the 256-universe batch).  A round of few points (blind) does not read first: its
// time is the chain of those reads, and an atomic without a result is not waited for
// (2+1 T = 64, 20 survivors 16.4 -> 12.6 us a round; 3+1 T = 128, 1800 60 -> 50 us).
__device__ __forceinline__ void occ_set_mask(uint32_t* words, int64_t w, uint32_t m, int64_t nwords, bool blind) {
    uint32_t* p = words + UG_IDX(w, nwords);
    if (blind || (__ldcg(p) & m) != m) atomicOr(p, m);
}
__device__ __forceinline__ void occ_set(uint32_t* words, int64_t bit, int64_t nwords, bool blind) {
    occ_set_mask(words, bit >> 5, 1u << (bit & 31), nwords, blind);
}

// Dilated filter: marks every block holding a cell that meets the cube of
// half-width occ1_reach around the committed point x (cells wrap around the
// torus; per axis at most 5 cells, so at most 5 blocks).
__device__ __forceinline__ void occ1_mark(const UniDev& d, int t, const double* x, bool blind) {
    int bk[3][5], nb[3] = {1, 1, 1};
#pragma unroll
    for (int ax = 0; ax < 3; ax++) {
        bk[ax][0] = 0;
        if (ax >= d.dim) continue;
        const int c0 = (int)floor((x[ax] - d.occ1_reach + 1.0) / d.cell);
        const int c1 = (int)floor((x[ax] + d.occ1_reach + 1.0) / d.cell);
        int n = 0;
        for (int c = c0; c <= c1 && n < 5; c++) {
            int w = c % d.gw;
            w += w < 0 ? d.gw : 0;
            const int b = w >> d.occ1_shift;
            bool seen = false;
            for (int k = 0; k < n; k++) seen |= bk[ax][k] == b;
            if (!seen) bk[ax][n++] = b;
        }
        nb[ax] = n;
    }
    // along the last axis the blocks are neighbouring bits: one masked update per word
    const int L = d.dim - 1;
    const int64_t t0 = (int64_t)t * d.occ1_per_t;
    for (int i0 = 0; i0 < (L > 0 ? nb[0] : 1); i0++)
        for (int i1 = 0; i1 < (L > 1 ? nb[1] : 1); i1++) {
            int64_t row = 0;
            if (L > 0) row = bk[0][i0];
            if (L > 1) row = row * d.occ1_gw + bk[1][i1];
            row = t0 + row * d.occ1_gw;
            int64_t wcur = -1;
            uint32_t m = 0;
            for (int i = 0; i < nb[L]; i++) {
                const int64_t bit = row + bk[L][i];
                if ((bit >> 5) != wcur) {
                    if (m) occ_set_mask(d.occ1, wcur, m, d.occ1_words, blind);
                    wcur = bit >> 5;
                    m = 0;
                }
                m |= 1u << (bit & 31);
            }
            occ_set_mask(d.occ1, wcur, m, d.occ1_words, blind);
        }
}

__global__ void __launch_bounds__(256) k_commit(const UniDev* __restrict__ U, UniCtl* ctl,
                                                RoundInfo* info) {
    const int n_uni = info->n_uni, total = info->total_spt;
    const int lane = threadIdx.x & 31;
    const bool blind = total <= (int)(gridDim.x * blockDim.x);  // a point per thread at most
    // items: (survivor, timestep) pairs, survivor-major per universe; the trip
    // count is uniform over the block so the warp-level counting below converges
    for (int w0 = blockIdx.x * blockDim.x; w0 < total; w0 += gridDim.x * blockDim.x) {
        const int w = w0 + threadIdx.x;
        int u = -1;
        bool new_key = false, new_cell = false;
        if (w < total) {
            u = find_uni(info->spt_off, n_uni, w);
            const UniDev& d = U[u];
            UniCtl& c = ctl[u];
            const int local = w - info->spt_off[u];
            const int r = local / d.T, t = local - r * d.T;
            const int k = r < c.stop_at ? d.acc_rank[UG_IDX(r, d.S_max)] : -1;
            if (k >= 0) {
                const int64_t slot = UG_IDX(c.n_slots_prev + k, d.slot_cap);
                Pt64 q = d.spos[UG_IDX((int64_t)r * d.T + t, (int64_t)d.S_max * d.T)];
                int cc[3] = {0, 0, 0};
#pragma unroll
                for (int ax = 0; ax < 3; ax++)
                    if (ax < d.dim) cc[ax] = cell_of(q.c[ax], d.cell, d.gw);
                int32_t old;
                uint32_t fbit;
                const int64_t lin = grid_lin(d, cc, &fbit);
                occ_set(d.occ, occ_bit(d, t, cc), d.occ_words, blind);
                occ1_mark(d, t, q.c, blind);
                grid_insert(d, c, t, lin, fbit, cells_per_t(d), (int32_t)slot, &old, &new_key, &new_cell);
                q.next = old;
                q.gid = d.sgid[UG_IDX(r, d.S_max)];
                d.pts[UG_IDX(slot * d.T + t, d.slot_cap * d.T)] = q;
                Pt32 f;
                f.c[0] = (float)q.c[0];
                f.c[1] = (float)q.c[1];
                f.c[2] = (float)q.c[2];
                f.next = old;
                d.ptf[UG_IDX(slot * d.T + t, d.slot_cap * d.T)] = f;
                if (t == 0)
                    d.acc_idx[UG_IDX(slot, d.slot_cap)] = c.round_base + d.surv_off[UG_IDX(r, d.S_max + 1)];
            }
        }
        // new hash keys and newly occupied cells: one atomic per (warp, universe)
        const uint32_t nk = __ballot_sync(0xffffffffu, new_key);
        const uint32_t ncl = __ballot_sync(0xffffffffu, new_cell);
        if (nk | ncl) {
            const uint32_t peers = __match_any_sync(0xffffffffu, u);
            const uint32_t mine = nk & peers, minec = ncl & peers;
            if (new_key && lane == __ffs(mine) - 1)
                atomicAdd((unsigned long long*)&ctl[u].hash_used, (unsigned long long)__popc(mine));
            if (new_cell && lane == __ffs(minec) - 1)
                atomicAdd((unsigned long long*)&ctl[u].round_new, (unsigned long long)__popc(minec));
        }
    }
}

// Rebuild the main-grid hash of universe u from its committed points (after
// the host swapped in a larger, empty table).
__global__ void k_rehash(const UniDev* __restrict__ U, UniCtl* ctl, int u, int64_t n_slots) {
    const UniDev& d = U[u];
    UniCtl& c = ctl[u];
    const int64_t total = n_slots * d.T;
    for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < total;
         w += (int64_t)gridDim.x * blockDim.x) {
        const int64_t slot = w / d.T;
        const int t = (int)(w % d.T);
        Pt64* q = d.pts + slot * d.T + t;
        int cc[3] = {0, 0, 0};
#pragma unroll
        for (int ax = 0; ax < 3; ax++)
            if (ax < d.dim) cc[ax] = cell_of(q->c[ax], d.cell, d.gw);
        int32_t old;
        bool new_key = false, new_cell = false;
        uint32_t fbit;
        const int64_t lin = grid_lin(d, cc, &fbit);
        grid_insert(d, c, t, lin, fbit, cells_per_t(d), (int32_t)slot, &old, &new_key, &new_cell);
        if (new_key) atomicAdd((unsigned long long*)&c.hash_used, 1ull);
        q->next = old;
        d.ptf[slot * d.T + t].next = old;
    }
}

}  // namespace ug

namespace ug {

// Worldline parameters in term order (the --dump-params content).  The knot stream
// replays the reference draw sequence (cuda/braid_knot.cu:111-166) keeping each
// term, one thread per path (the stream is sequential); the counter stream lists
// term j = frequency j + 2 (k_params_philox).
__global__ void k_params(const UniDev* __restrict__ U, int u, int64_t n, double* a2o, double* ao,
                         int32_t* bo, double* fo) {
    const UniDev& d = U[u];
    const int D = d.dim, nw = d.nw;
    double wj[kMaxF];
    int32_t bj[kMaxF];
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < n;
         s += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t idx = (uint64_t)d.acc_idx[s];
        Xo r;
        r.seed(knot_seed(d.seed, idx));
        for (int ax = 0; ax < D; ax++) {
            const int64_t o = (s * D + ax) * nw;
            if ((uint32_t)nw == d.modmax) {
                for (int j = 0; j < nw; j++) bj[j] = j + 2;
                for (int j = nw - 1; j > 0; j--) {
                    const int k = (int)r.below((uint32_t)(j + 1));
                    const int32_t tmp = bj[j];
                    bj[j] = bj[k];
                    bj[k] = tmp;
                }
            } else {
                for (int j = 0; j < nw; j++) {
                    int bnew = 0;
                    bool dup = true;
                    for (int guard = 0; dup && guard < 64; guard++) {
                        bnew = (int)r.below(d.modmax) + 2;
                        dup = false;
                        for (int k = 0; k < j; k++)
                            if (bj[k] == bnew) dup = true;
                    }
                    bj[j] = bnew;
                }
            }
            double sum = 0.0;
            for (int j = 0; j < nw; j++) {
                wj[j] = -log(1.0 - r.f64());
                sum += wj[j];
            }
            for (int j = 0; j < nw; j++) wj[j] /= sum;
            for (int j = 0; j < nw; j++) {
                double amp = wj[j] / (double)bj[j];
                if (r.flip()) amp = -amp;
                ao[o + j] = amp;
                bo[o + j] = bj[j];
                fo[o + j] = (bj[j] % 2 == 0) ? r.f64() * kPi : 0.0;
            }
            a2o[s * D + ax] = d.pin ? 0.0 : (r.f64() * 2.0 - 1.0);
        }
    }
}

// The counter stream's parameters: one warp per (path, axis), blocks spread over the
// lanes, so every store is coalesced; the normalisation sums in ascending b as the
// candidate test does.  Bound by the FP64 logarithms and the 20 bytes written per term:
// 18 k paths x 2 axes x 255 terms in 0.11 ms (one thread per path, storing 5 KB apart from
// its neighbours: 2.75 ms).
__global__ void __launch_bounds__(128) k_params_philox(const UniDev* __restrict__ U, int u, int64_t n, double* a2o,
                                                       double* ao, int32_t* bo, double* fo) {
    __shared__ double s_e[4][kMaxF + 1];
    const UniDev& d = U[u];
    const int D = d.dim, nw = d.nw, F = d.F;
    const int lane = threadIdx.x & 31;
    double* e = s_e[threadIdx.x >> 5];
    const int64_t warps = (int64_t)gridDim.x * 4;
    for (int64_t i = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5); i < n * D; i += warps) {
        const int64_t s = i / D;
        const int ax = (int)(i - s * D);
        const uint64_t idx = (uint64_t)d.acc_idx[s];
        const int64_t o = i * nw - 2;  // term j = b - 2
        for (int p = lane; 2 * p <= F; p += 32) {
            const uint4 q = philox_block(d.seed, idx, ax, p);
            if (p == 0) {
                a2o[i] = d.pin ? 0.0 : (double)q.x * (1.0 / 2147483648.0) - 1.0;
                continue;
            }
            const int be = 2 * p, bo2 = 2 * p + 1;
            const double Ee = -log(((double)q.x + 0.5) * (1.0 / 4294967296.0));
            e[be] = (q.z & 1u) ? -Ee : Ee;
            fo[o + be] = (double)(q.z >> 1) * (1.0 / 2147483648.0) * kPi;
            if (bo2 <= F) {
                const double Eo = -log(((double)q.y + 0.5) * (1.0 / 4294967296.0));
                e[bo2] = (q.w & 1u) ? -Eo : Eo;
                fo[o + bo2] = 0.0;
            }
        }
        __syncwarp();
        double sum = 0.0;
        if (lane == 0)
            for (int b = 2; b <= F; b++) sum += fabs(e[b]);
        sum = __shfl_sync(0xffffffffu, sum, 0);
        for (int b = 2 + lane; b <= F; b += 32) {
            const double amp = fabs(e[b]) / sum / (double)b;
            ao[o + b] = e[b] < 0.0 ? -amp : amp;
            bo[o + b] = b;
        }
        __syncwarp();
    }
}

void launch_params(const UniDev* dU, int u, int rng, int dim, int64_t n, double* a2, double* a, int32_t* b,
                   double* f, cudaStream_t st) {
    if (rng == RNG_KNOT) {
        const int blocks = (int)std::min<int64_t>((n + 127) / 128, 4096);
        k_params<<<blocks, 128, 0, st>>>(dU, u, n, a2, a, b, f);
        return;
    }
    const int blocks = (int)std::min<int64_t>((n * dim + 3) / 4, 148 * 64);
    k_params_philox<<<blocks, 128, 0, st>>>(dU, u, n, a2, a, b, f);
}

// ------------------------------------------------------------- read-back

// Trajectories of the first n slots as [slot][axis][timestep] doubles: a warp reads 32
// points of a slot (32 bytes each) and writes each axis coalesced.  Bound by HBM; the whole
// read-back of 8000 3+1 paths at T = 128 (parameters and trajectories) went from 19.7 to 12.7
// ms against copying the points and transposing them on one host thread.
__global__ void __launch_bounds__(256) k_positions(const UniDev* __restrict__ U, int u, int64_t n,
                                                   double* __restrict__ out) {
    const UniDev& d = U[u];
    const int T = d.T, dim = d.dim;
    for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n * T; w += (int64_t)gridDim.x * blockDim.x) {
        const int64_t s = w / T;
        const int t = (int)(w - s * T);
        const Pt64 p = d.pts[UG_IDX(w, d.slot_cap * T)];
        double* o = out + s * dim * T + t;
#pragma unroll
        for (int ax = 0; ax < 3; ax++)
            if (ax < dim) o[(int64_t)ax * T] = p.c[ax];
    }
}

// Accepted candidate indices and group labels of every universe into one
// contiguous pair of arrays (universe u at [off[u], off[u+1])), so that a
// caller reads all of them back with one copy each.  One CTA per universe.
__global__ void k_gather_accepted(const UniDev* __restrict__ U, const int64_t* __restrict__ off,
                                  int64_t* __restrict__ idx, int32_t* __restrict__ gid) {
    const int u = blockIdx.x;
    const UniDev& d = U[u];
    const int64_t o = off[u], n = off[u + 1] - o;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        idx[o + i] = d.acc_idx[UG_IDX(i, d.slot_cap)];
        gid[o + i] = d.pts[UG_IDX(i * d.T, d.slot_cap * d.T)].gid;
    }
}

}  // namespace ug
