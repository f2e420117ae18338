// ug_frames.cu -- past-light-cone frame baking of a packed universe (2+1).
//
// For each instant z_obs and observer, the pulse centre is frozen at the
// observer's comoving position and the universe is rewound while a front
// expands (cuda/frame_bake.cu:1-40): front "speed" (conformal, speed c),
// "fit" (c = -1/eta(z_min)) or "budget" (wiggle-budget reach).  Every torus
// image (2nx, 2ny), |n| <= K, of every worldline is walked along the rewind
// grid for sign changes of dist(pos + shift - centre) - chi_front and each
// crossing is refined by 24 bisection steps with fresh evaluations
// (frame_bake.cu:281-371).  Hits are (src, dx, dy, chi, z_emit); optionally
// they are histogrammed into a bins x bins uint32 density grid per frame over
// [-chi_max, chi_max]^2 (no reference counterpart; the reference draws
// scatter plots, plots/render_frames.py:47-110).
//
// Evaluation: X(z) = [a2 sin z + sum_j a_j (sin(b_j z + f_j) - sin f_j)] / sin z
// (frame_bake.cu:201-212).  Full-band dumps evaluate sum_j a_j sin(b_j z + f_j)
// on the rewind grid as an FP64 tensor product over sin, cos(b z), and at single
// instants as Im P(e^{iz}) with P(w) = sum_b (a_b e^{i f_b}) w^b by complex
// Horner -- one sincos per evaluation instead of one per term; few-term dumps
// sum the terms directly.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "ug_dmma.cuh"
#include "ug_frames.cuh"

namespace ug {

int set_error(int code, const char* msg);

namespace {

constexpr int kGridRows = 420;     // rewind grid (frame_bake.cu:71)
constexpr int kBisect = 24;        // bisection steps (frame_bake.cu:72)
constexpr int kBudgetCap = 4000;   // budget rewind-grid cap (frame_bake.cu:73)
constexpr double kPiF = 3.14159265358979323846;

struct FPaths {
    int n, nw, bmax;
    int horner;            // 1: complex Horner over b = 0..bmax; 0: per-term sums
    const double* a2;      // [n][2]
    const double* s0;      // [n][2]  sum_j a_j sin f_j
    const double* a;       // [n][2][nw]
    const double* b;       // [n][2][nw]
    const double* f;       // [n][2][nw]
    const double2* coef;   // [n][2][bmax+1] a_b e^{i f_b} (Horner form)
    const double* amp;     // [n] largest sum_j |a_j| of the axes
};

struct FFront {
    int budget, cheb, M, bMax;
    double spd, zObs, etaObs, chiMax;
    const double2* reach;  // budget: terms of frequency b at z_obs (k_fb_reach)
};

__host__ __device__ inline double wiggle_direct(const double* a, const double* b, const double* f, int nw,
                                                double z) {
    double s = 0.0;
    for (int j = 0; j < nw; j++) s += a[j] * sin(b[j] * z + f[j]);
    return s;
}

__device__ inline double wiggle_horner(const double2* c, int bmax, double z) {
    double sz, cz;
    sincos(z, &sz, &cz);
    double pr = c[bmax].x, pi = c[bmax].y;
    for (int k = bmax - 1; k >= 0; k--) {
        const double nr = fma(pr, cz, fma(-pi, sz, c[k].x));
        const double ni = fma(pr, sz, fma(pi, cz, c[k].y));
        pr = nr;
        pi = ni;
    }
    return pi;
}

__device__ inline void comov(const FPaths& P, int p, double z, double* X, double* Y) {
    const double s = sin(z);
    double w[2];
    for (int ax = 0; ax < 2; ax++) {
        const size_t o = ((size_t)p * 2 + ax);
        w[ax] = P.horner ? wiggle_horner(P.coef + o * (P.bmax + 1), P.bmax, z)
                         : wiggle_direct(P.a + o * P.nw, P.b + o * P.nw, P.f + o * P.nw, P.nw, z);
    }
    *X = (P.a2[(size_t)p * 2] * s + w[0] - P.s0[(size_t)p * 2]) / s;
    *Y = (P.a2[(size_t)p * 2 + 1] * s + w[1] - P.s0[(size_t)p * 2 + 1]) / s;
}

// Wiggle-budget reach of the front (frame_bake.cu:236-251).
inline double reach_of(double z, double zObs, int bMax) {
    const double s = sin(z), sObs = sin(zObs);
    double best = 0.0;
    for (int b = 2; b <= bMax; b++) {
        const double da = (cos(b * z) - 1.0) / (b * s) - (cos(b * zObs) - 1.0) / (b * sObs);
        const double db = sin(b * z) / (b * s) - sin(b * zObs) / (b * sObs);
        const double d = (b % 2 == 0) ? sqrt(da * da + db * db) : fabs(db);
        best = d > best ? d : best;
    }
    return best;
}

// reach_of with its z_obs terms (x: cosine, y: sine) tabulated once per frame.
__device__ inline double reach_tab(const FFront& F, double z) {
    const double s = sin(z);
    double best = 0.0;
    for (int b = 2; b <= F.bMax; b++) {
        const double2 o = __ldg(F.reach + b);
        double sb, cb;
        sincos(b * z, &sb, &cb);
        const double da = (cb - 1.0) / (b * s) - o.x;
        const double db = sb / (b * s) - o.y;
        const double d = (b % 2 == 0) ? sqrt(da * da + db * db) : fabs(db);
        best = d > best ? d : best;
    }
    return best;
}

__global__ void k_fb_reach(int bMax, double zObs, double2* reach) {
    const double sObs = sin(zObs);
    for (int b = 2 + blockIdx.x * blockDim.x + threadIdx.x; b <= bMax; b += gridDim.x * blockDim.x)
        reach[b] = make_double2((cos(b * zObs) - 1.0) / (b * sObs), sin(b * zObs) / (b * sObs));
}

__device__ inline double metric(double dx, double dy, int cheb) {
    return cheb ? fmax(fabs(dx), fabs(dy)) : sqrt(dx * dx + dy * dy);
}

// Rewind-grid positions of few-term dumps, one thread per (path, row): a sine per term.
__global__ void k_fb_grid(FPaths P, int M, const double* zg, double* px, double* py) {
    const int R = M + 1;
    const int64_t total = (int64_t)P.n * R;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        comov(P, (int)(i / R), zg[i % R], px + i, py + i);
    }
}

// The rewind grid as an FP64 product for full-band dumps: wiggle[row (p, ax)][i] =
// sum_b re_b sin(b z_i) + im_b cos(b z_i), half the multiplications of evaluating the
// polynomial at every (path, row).  The basis of a frame is laid out by k_fb_basis.
constexpr int kGbRows = 64;    // (path, axis) rows of a tile, 16 per warp
constexpr int kGbCols = 72;    // rewind rows of a tile: 421 rows are 6 tiles, 2.6 % padding
constexpr int kGbB = 8;        // frequencies per chunk (16 terms)
constexpr int kGbStages = 3;
constexpr int kGbPitch = kGbCols + 2;  // two rows are 4 mod 16 apart: operand reads touch every bank once

// basis[2 b][c], basis[2 b + 1][c] = sin, cos of b z_c, zero beyond the last row.  The
// rounding of b z is carried into the result, so the phase is good to an ulp of z.
__global__ void k_fb_basis(int bmax, int R, int Rp, const double* __restrict__ zg, double* __restrict__ basis) {
    const int64_t total = (int64_t)(bmax + 1) * Rp;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int b = (int)(i / Rp), c = (int)(i % Rp);
        double s = 0.0, co = 0.0;
        if (c < R) {
            const double z = zg[c], x = b * z, e = fma((double)b, z, -x);
            double s0, c0;
            sincos(x, &s0, &c0);
            s = fma(e, c0, s0);
            co = fma(-e, s0, c0);
        }
        basis[(int64_t)(2 * b) * Rp + c] = s;
        basis[(int64_t)(2 * b + 1) * Rp + c] = co;
    }
}

// One CTA per 64 x 72 tile, a warp per 16 rows (9 products of 16 x 8 a step of four
// frequencies).  A step's terms are ordered sin of its four frequencies, then cos, so a
// lane's A operands are the (re, im) pairs of its own frequency, read straight from
// global memory two steps ahead; the basis chunks come in by cp.async, two in flight.
// Bound by the FP64 tensor rate: 18 k paths x 421 rows at b_max 256 take 0.58 ms, 0.45 ms
// at 37 TFLOP/s.  The same product on FP64 FMAs waited for its shared-memory operands
// (0.90 ms); the polynomial at every (path, row) took 1.53 ms.
__global__ void __launch_bounds__(128) k_fb_grid_mm(FPaths P, int R, int Rp, const double* __restrict__ zg,
                                                    const double* __restrict__ basis, double* __restrict__ px,
                                                    double* __restrict__ py) {
    __shared__ __align__(16) double Bs[kGbStages][2 * kGbB][kGbPitch];
    constexpr int kN = kGbCols / 8;
    const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int64_t nrows = (int64_t)P.n * 2;
    // the column tiles of a row tile are neighbours: its coefficients are read from DRAM once
    const int ct = Rp / kGbCols;
    const int64_t row0 = (int64_t)(blockIdx.x / ct) * kGbRows + (tid >> 5) * 16;
    const int col0 = (int)(blockIdx.x % ct) * kGbCols;
    const int nb = P.bmax + 1;
    const int nch = (nb + kGbB - 1) / kGbB;
    auto stage = [&](int ch) {
        const int terms = min(2 * kGbB, 2 * (nb - ch * kGbB));  // none past the last chunk
        for (int e = tid; e < 2 * kGbB * (kGbCols / 2); e += 128) {
            const int k = e / (kGbCols / 2), cc = (e % (kGbCols / 2)) * 2;
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&Bs[ch % kGbStages][k][cc]);
            const double* src = basis + (k < terms ? (int64_t)(2 * ch * kGbB + k) * Rp : 0) + col0 + cc;
            // terms beyond the last frequency: zeros
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(k < terms ? 16 : 0)
                         : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const double2* ar[2] = {P.coef + min(row0 + g, nrows - 1) * nb, P.coef + min(row0 + g + 8, nrows - 1) * nb};
    double2 a[3][2];  // this step's and the next two steps' (re, im) of rows g, g + 8
    auto fetch = [&](int step, double2* v) {
        const int b = 4 * step + t;
#pragma unroll
        for (int q = 0; q < 2; q++) v[q] = b < nb ? __ldg(ar[q] + b) : make_double2(0.0, 0.0);
    };
    double acc[kN][4];
#pragma unroll
    for (int j = 0; j < kN; j++)
#pragma unroll
        for (int q = 0; q < 4; q++) acc[j][q] = 0.0;
    stage(0);
    stage(1);
    fetch(0, a[0]);
    fetch(1, a[1]);
    for (int ch = 0; ch < nch; ch++) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();  // chunk ch has landed, chunk ch - 1 has been read
        stage(ch + 2);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            fetch(2 * ch + h + 2, a[2]);
            const double av[4] = {a[0][0].x, a[0][1].x, a[0][0].y, a[0][1].y};
            // basis row 2 b: sin, 2 b + 1: cos
            const double* bs = &Bs[ch % kGbStages][8 * h + 2 * t][g];
#pragma unroll
            for (int j = 0; j < kN; j++) {
                const double bv[2] = {bs[8 * j], bs[kGbPitch + 8 * j]};
                dmma_16x8x8(acc[j], av, bv);
            }
#pragma unroll
            for (int q = 0; q < 2; q++) {
                a[0][q] = a[1][q];
                a[1][q] = a[2][q];
            }
        }
    }
    double a2[2], s0[2];
    double* out[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int64_t row = min(row0 + g + 8 * q, nrows - 1);
        a2[q] = P.a2[row];
        s0[q] = P.s0[row];
        out[q] = row0 + g + 8 * q < nrows ? (row & 1 ? py : px) + (row >> 1) * R : nullptr;
    }
#pragma unroll
    for (int j = 0; j < kN; j++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int c = col0 + 8 * j + 2 * t + e;
            if (c >= R) continue;
            const double s = __ldg(basis + 2 * (int64_t)Rp + c);  // sin z
#pragma unroll
            for (int q = 0; q < 2; q++)
                if (out[q]) out[q][c] = (a2[q] * s + acc[j][2 * q + e] - s0[q]) / s;
        }
}

// A sign change of dist(image) - chi_front between rewind rows i-1 and i.
struct FCross {
    int32_t p;
    int16_t nx, ny;
    int32_t i;
    int32_t inside;  // the image was inside the front at row i-1
};

// First rewind row the front can reach an image of ring s = max(|nx|, |ny|) at (comoving
// coordinates stay within +-2), M + 1 when it never does.
__device__ __forceinline__ int first_row(const FFront& F, int s) {
    if (s <= 2) return F.chiMax > 0.0 ? 1 : F.M + 1;
    const double dmin = 2.0 * s - 4.0;
    if (dmin >= F.chiMax) return F.M + 1;
    return F.budget ? 1 : max(1, (int)ceil(dmin * F.M / F.chiMax));
}

// Nearest |n| to zero of n0 .. n0 + w - 1.
__device__ __forceinline__ int nearest_ring(int n0, int w) { return n0 > 0 ? n0 : (n0 + w > 0 ? 0 : 1 - n0 - w); }

// One warp per path and 32 x 32 of its (2K + 1)^2 torus images.  A lane holds a rewind row
// (chunks of 32 rows, the first of which is the last of the chunk before), a ballot the
// signs of dist(image) - chi_front at all of them; neighbouring bits that differ are the
// crossings, which k_fb_refine bisects.  The square metric is separable: max(|dx|, |dy|) <
// chi is |dx| < chi and |dy| < chi, so 2 x 32 ballots serve the 32 x 32 images and the
// lanes combine one image each.  Chunks before the front reaches an image are left out.
// Bound by issue: 0.11 ms for 18 k paths of 49 images (one thread per (path, image)
// walking the 421 rows: 0.36 ms).  A warp for all images of a path, with a ballot each
// beyond 32 a side, left a view of few paths and many images to few warps (one path, 301
// images a side: 840 ms).
__global__ void __launch_bounds__(128) k_fb_cross(FPaths P, FFront F, double ox, double oy, int K, int obsIdx,
                                                  const double* __restrict__ chig, const double* __restrict__ px,
                                                  const double* __restrict__ py, FCross* cross,
                                                  unsigned long long* count, unsigned long long cap) {
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * (blockDim.x >> 5);
    const int R = F.M + 1, side = (2 * K + 32) / 32, tiles = side * side;  // tiles a side, in all
    const int64_t items = (int64_t)P.n * tiles;
    for (int64_t item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); item < items; item += warps) {
        const int p = (int)(item / tiles), tile = (int)(item % tiles);
        const int x0 = tile % side * 32 - K, y0 = tile / side * 32 - K;
        const int wx = min(32, K + 1 - x0), wy = min(32, K + 1 - y0), images = wx * wy;
        const int first = first_row(F, max(nearest_ring(x0, wx), nearest_ring(y0, wy)));
        const double* X = px + (int64_t)p * R;
        const double* Y = py + (int64_t)p * R;
        for (int c0 = (first - 1) / 31 * 31; c0 + 1 < R; c0 += 31) {
            const int i = c0 + lane;
            const double x = i < R ? X[i] : 0.0, y = i < R ? Y[i] : 0.0, chi = i < R ? chig[i] : 0.0;
            // rows that a crossing may end at: all of the chunk's but its first
            const uint32_t rows = (R - c0 >= 32 ? 0xffffffffu : (1u << (R - c0)) - 1u) & ~1u;
            // the observer sits on the front at chi = 0: keep its own image inside
            const bool own = p == obsIdx && c0 == 0 && fabs(metric(x + (0.0 - ox), y + (0.0 - oy), F.cheb) - chi) < 1e-9;
            const bool own0 = __shfl_sync(0xffffffffu, (int)own, 0) != 0;
            uint32_t mx = 0, my = 0;
            if (F.cheb) {
                for (int k = 0; k < wx; k++) {
                    const uint32_t b = __ballot_sync(0xffffffffu, i < R && fabs(x + (2.0 * (x0 + k) - ox)) < chi);
                    if (lane == k) mx = b;
                }
                for (int k = 0; k < wy; k++) {
                    const uint32_t b = __ballot_sync(0xffffffffu, i < R && fabs(y + (2.0 * (y0 + k) - oy)) < chi);
                    if (lane == k) my = b;
                }
            }
            for (int m0 = 0; m0 < images; m0 += 32) {
                // this lane's image and the signs of its rows, from the first that counts on
                const int m = m0 + lane;
                const int xi = m % wx, yi = m / wx, nx = x0 + xi, ny = y0 + yi;
                const int i0 = m < images ? first_row(F, max(abs(nx), abs(ny))) : R;
                const uint32_t on = __ballot_sync(0xffffffffu, i0 < c0 + 32 && i0 < R);
                if (!on) continue;
                uint32_t sg = 0;
                if (F.cheb) {
                    sg = __shfl_sync(0xffffffffu, mx, xi) & __shfl_sync(0xffffffffu, my, yi & 31);
                } else {
                    for (uint32_t w = on; w; w &= w - 1) {
                        const int q = __ffs(w) - 1, qx = x0 + (m0 + q) % wx, qy = y0 + (m0 + q) / wx;
                        const uint32_t b = __ballot_sync(
                            0xffffffffu,
                            i < R && metric(x + (2.0 * qx - ox), y + (2.0 * qy - oy), F.cheb) - chi < 0.0);
                        if (lane == q) sg = b;
                    }
                }
                uint32_t cr = 0;
                if ((on >> lane) & 1u) {
                    if (own0 && nx == 0 && ny == 0 && i0 == 1) sg |= 1u;
                    cr = (sg ^ (sg << 1)) & rows;
                    if (i0 > c0) cr &= ~((1u << (i0 - c0)) - 1u);  // rows from i0 on
                }
                const uint32_t any = __ballot_sync(0xffffffffu, cr != 0u);
                if (!any) continue;
                int incl = __popc(cr);
                const int mine = incl;
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += v;
                }
                unsigned long long base = 0;
                if (lane == 31) base = atomicAdd(count, (unsigned long long)incl);
                base = __shfl_sync(0xffffffffu, base, 31) + (unsigned long long)(incl - mine);
                for (; cr; cr &= cr - 1, base++) {
                    const int bit = __ffs(cr) - 1;
                    if (base < cap)
                        cross[base] = FCross{p, (int16_t)nx, (int16_t)ny, c0 + bit, (int32_t)((sg >> (bit - 1)) & 1u)};
                }
            }
        }
    }
}

// Refinement of a crossing: 24 bisection steps over its row interval
// (frame_bake.cu:281-371).
//
// Over one rewind row the wiggle of each axis is, to well below 1e-12, the polynomial
// through its values at 16 Chebyshev nodes: sin(b z + f) on an interval of half-width h
// is interpolated to 4 (b h / 2)^16 / 16! (Jacobi-Anger: its Chebyshev coefficients are
// at most 2 J_k(b h)), and the rounding of the nodes' values (2 b_max ulps of the summed
// amplitudes) grows at most threefold.  So the path's coefficients are read once, for the 16 nodes, and
// the steps evaluate the interpolant.  A step whose distance to the front is below
// kSure, where the interpolant might give the other sign, evaluates the path itself;
// intervals too wide for the bound (kWide), and few-term dumps, always do.  Every step
// therefore takes the side that a fresh evaluation gives, and the offsets of the hit
// come from a fresh evaluation at the end.
constexpr int kNodes = 16;
constexpr double kSure = 1e-12;   // |g| above this: the interpolant's sign is the path's
constexpr double kWide = 5e-13;   // largest error of an interpolated position

// Wiggles of both axes of a few-term dump's path.
__device__ __forceinline__ void wiggles(const FPaths& P, int p, double z, double (*w)[1]) {
    const size_t o = (size_t)p * 2;
#pragma unroll
    for (int ax = 0; ax < 2; ax++)
        w[ax][0] = wiggle_direct(P.a + (o + ax) * P.nw, P.b + (o + ax) * P.nw, P.f + (o + ax) * P.nw, P.nw, z);
}

// Terms of a path that its eight lanes stage at a time, a buffer being read, one coming in.
constexpr int kFbTerms = 16;
struct FbStage {
    double2 c[2][2][kFbTerms];  // [buffer][axis][terms k, descending from b_max]
    double2 pad;                // a warp's four paths in different banks
};

// Wiggles of a path (wiggle_horner's operations) by the eight lanes (mask oct, lane j) that
// hold it: of both axes at the lane's own kQ instants (kAx = 2), or of axis j & 1 (kAx = 1).  The terms come in by cp.async,
// so their way from memory runs behind the products.
template <int kQ, int kAx>
__device__ __forceinline__ void oct_wiggles(const FPaths& P, int p, const double* z, double (*w)[kQ], FbStage& S,
                                            uint32_t oct, int j) {
    const int nt = P.bmax + 1, nst = (nt + kFbTerms - 1) / kFbTerms;
    const double2* src = P.coef + (size_t)p * 2 * nt;
    auto stage = [&](int ch) {
        if (ch < nst)
#pragma unroll
            for (int h = 0; h < 2 * kFbTerms / 8; h++) {
                const int e = j + 8 * h, ax = e / kFbTerms, q = e % kFbTerms, k = P.bmax - (ch * kFbTerms + q);
                const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&S.c[ch & 1][ax][q]);
                asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst),
                             "l"(src + (size_t)ax * nt + max(k, 0)), "r"(k >= 0 ? 16 : 0)
                             : "memory");
            }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    double sz[kQ], cz[kQ], pr[kAx][kQ], pi[kAx][kQ];
    __syncwarp(oct);  // the buffers' last readers
    stage(0);
#pragma unroll
    for (int q = 0; q < kQ; q++) {
        sincos(z[q], &sz[q], &cz[q]);
#pragma unroll
        for (int ax = 0; ax < kAx; ax++) pr[ax][q] = pi[ax][q] = 0.0;
    }
    for (int ch = 0; ch < nst; ch++) {
        stage(ch + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp(oct);  // chunk ch has landed
        const double2(*cs)[kFbTerms] = S.c[ch & 1];
        const int n = min(kFbTerms, nt - ch * kFbTerms);
        auto term = [&](int e) {
#pragma unroll
            for (int ax = 0; ax < kAx; ax++) {
                const double2 ck = cs[kAx == 2 ? ax : j & 1][e];
#pragma unroll
                for (int q = 0; q < kQ; q++) {
                    const double nr = fma(pr[ax][q], cz[q], fma(-pi[ax][q], sz[q], ck.x));
                    const double ni = fma(pr[ax][q], sz[q], fma(pi[ax][q], cz[q], ck.y));
                    pr[ax][q] = nr;
                    pi[ax][q] = ni;
                }
            }
        };
        if (n == kFbTerms) {
#pragma unroll 4
            for (int e = 0; e < kFbTerms; e++) term(e);
        } else {
            for (int e = 0; e < n; e++) term(e);
        }
        __syncwarp(oct);  // before chunk ch + 2 replaces it
    }
#pragma unroll
    for (int ax = 0; ax < kAx; ax++)
#pragma unroll
        for (int q = 0; q < kQ; q++) w[ax][q] = pi[ax][q];
}

// Eight lanes per crossing; a pass takes three bisection steps: the seven midpoints they
// can reach (one per lane) are evaluated, then the steps follow from the signs -- the same
// midpoints, from the same operations, as one step at a time.  Bound by FP64
// issue (40 % of it busy) and a last wave that is not full: 0.20 ms for 26 k crossings at b_max
// 256, 80 registers and six blocks an SM (eight with 64 registers: the same).  Four lanes, two
// points each and the terms loaded where they are used took 162 registers, and 15 % of the
// warps waited for memory: 0.31 ms; one thread per crossing 2.06 ms for 18 k.
constexpr int kFbThreads = 128;
__global__ void __launch_bounds__(kFbThreads, 6) k_fb_refine(FPaths P, FFront F, double ox, double oy, const double* zg,
                                                   const double* chig, const FCross* cross,
                                                   const unsigned long long* count, unsigned long long cap,
                                                   ug_hit* hits) {
    static_assert(kBisect % 3 == 0, "three bisection steps a pass");
    __shared__ double s_cos[kNodes][kNodes + 1];               // cos(k theta_i) / 8 (row 0: 1 / 16)
    __shared__ double s_w[kFbThreads / 8][2][kNodes + 1];      // samples, then coefficients, of each crossing
    __shared__ __align__(16) FbStage s_st[kFbThreads / 8];
    const unsigned long long c = *count;
    const int64_t n = (int64_t)(c < cap ? c : cap);
    for (int e = threadIdx.x; e < kNodes * kNodes; e += blockDim.x) {
        const int k = e / kNodes, i = e % kNodes;
        s_cos[k][i] = k == 0 ? 1.0 / kNodes : cospi((double)(k * (2 * i + 1)) / (2 * kNodes)) * (2.0 / kNodes);
    }
    __syncthreads();
    const int j = threadIdx.x & 7;                       // lane of the crossing's eight
    const int sh = threadIdx.x & 24;                     // its first lane of the warp
    double(*ws)[kNodes + 1] = s_w[threadIdx.x >> 3];
    FbStage& S = s_st[threadIdx.x >> 3];
    const uint32_t oct = 0xffu << sh;  // the eight lanes share all of their crossing's branches
    const int64_t stride = (int64_t)gridDim.x * blockDim.x >> 3;
    for (int64_t k = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3; k < n; k += stride) {
        const FCross x = cross[k];
        const int p = x.p, i = x.i;
        const bool inside = x.inside != 0;
        const size_t o = (size_t)p * 2;
        const double a2x = P.a2[o], a2y = P.a2[o + 1], s0x = P.s0[o], s0y = P.s0[o + 1];
        const double bx = 2.0 * x.nx - ox, by = 2.0 * x.ny - oy;
        // the bracket in z (budget front) or chi (the others)
        double lo = F.budget ? zg[i - 1] : chig[i - 1], hi = F.budget ? zg[i] : chig[i];
        // emission times run down as the front grows
        const double zc = 0.5 * (zg[i - 1] + zg[i]), zh = 0.5 * fabs(zg[i - 1] - zg[i]) * (1.0 + 1e-12) + 1e-15;
        bool smooth = false;
        if (P.horner) {
            double u = 0.5 * P.bmax * zh;
            u *= u;
            u *= u;
            u *= u;
            u *= u;  // (b h / 2)^16, over 16!
            smooth = P.amp[p] * (4.0 / 2.0922789888e13 * u + 1e-15 * P.bmax) < kWide * fmin(sin(zc - zh), sin(zc + zh));
        }
        if (smooth) {
            double z[2], w[2][2];
#pragma unroll
            for (int q = 0; q < 2; q++) z[q] = fma(zh, cospi((2 * (2 * j + q) + 1) / (2.0 * kNodes)), zc);
            oct_wiggles<2, 2>(P, p, z, w, S, oct, j);
#pragma unroll
            for (int q = 0; q < 2; q++) {
                ws[0][2 * j + q] = w[0][q];
                ws[1][2 * j + q] = w[1][q];
            }
            __syncwarp(oct);
#pragma unroll
            for (int q = 0; q < 2; q++) w[0][q] = w[1][q] = 0.0;
            for (int e = 0; e < kNodes; e++)
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    w[0][q] = fma(s_cos[2 * j + q][e], ws[0][e], w[0][q]);
                    w[1][q] = fma(s_cos[2 * j + q][e], ws[1][e], w[1][q]);
                }
            __syncwarp(oct);
#pragma unroll
            for (int q = 0; q < 2; q++) {
                ws[0][2 * j + q] = w[0][q];
                ws[1][2 * j + q] = w[1][q];
            }
            __syncwarp(oct);
        }
        const double izh = 1.0 / zh;
        for (int it = 0; it < kBisect; it += 3) {
            // nodes of the pass's tree: 1 the midpoint, 2 and 3 those of its halves, 4..7
            // of its quarters; lane j evaluates node j (lane 0 node 1 as well)
            const int mine = max(j, 1);
            double l = lo, h = hi, m = (l + h) / 2.0;
            for (int lev = mine >= 4 ? 1 : (mine >= 2 ? 0 : -1); lev >= 0; lev--) {
                if ((mine >> lev) & 1)
                    l = m;
                else
                    h = m;
                m = (l + h) / 2.0;
            }
            const double z = F.budget ? m : 2.0 * atan(exp(F.etaObs - m / F.spd));
            double w[2][1];
            if (smooth) {  // Clenshaw, both axes together
                const double t2 = 2.0 * (z - zc) * izh;
                double b1[2] = {0.0, 0.0}, b2[2] = {0.0, 0.0};
                for (int e = kNodes - 1; e > 0; e--)
#pragma unroll
                    for (int ax = 0; ax < 2; ax++) {
                        const double b0 = fma(t2, b1[ax], ws[ax][e] - b2[ax]);
                        b2[ax] = b1[ax];
                        b1[ax] = b0;
                    }
#pragma unroll
                for (int ax = 0; ax < 2; ax++) w[ax][0] = fma(0.5 * t2, b1[ax], ws[ax][0] - b2[ax]);
            } else if (P.horner) {
                oct_wiggles<1, 2>(P, p, &z, w, S, oct, j);
            } else {
                wiggles(P, p, z, w);
            }
            const double s = sin(z);
            const double gm = metric((a2x * s + w[0][0] - s0x) / s + bx, (a2y * s + w[1][0] - s0y) / s + by, F.cheb) -
                              (F.budget ? reach_tab(F, m) : m);
            // bit of each node: the crossing lies above its midpoint; its sign is certain
            const uint32_t up = __ballot_sync(oct, (gm < 0.0) == inside) >> sh;
            const uint32_t sure = __ballot_sync(oct, !smooth || fabs(gm) > kSure) >> sh;
            int node = 1;
#pragma unroll
            for (int lev = 0; lev < 3; lev++) {
                const double mid = (lo + hi) / 2.0;
                int u = (up >> node) & 1;
                if (!((sure >> node) & 1)) {  // the path itself
                    const double z1 = F.budget ? mid : 2.0 * atan(exp(F.etaObs - mid / F.spd));
                    double w1[2][1];
                    oct_wiggles<1, 2>(P, p, &z1, w1, S, oct, j);
                    const double s1 = sin(z1);
                    const double g1 =
                        metric((a2x * s1 + w1[0][0] - s0x) / s1 + bx, (a2y * s1 + w1[1][0] - s0y) / s1 + by, F.cheb) -
                        (F.budget ? reach_tab(F, mid) : mid);
                    u = (g1 < 0.0) == inside;
                }
                if (u)
                    lo = mid;
                else
                    hi = mid;
                node = 2 * node + u;
            }
        }
        double chi, z1;
        if (F.budget) {
            z1 = (lo + hi) / 2.0;
            chi = reach_tab(F, z1);
        } else {
            chi = (lo + hi) / 2.0;
            z1 = 2.0 * atan(exp(F.etaObs - chi / F.spd));
        }
        double w[2][1];
        if (P.horner) {  // lane 0 the first axis, lane 1 the second
            oct_wiggles<1, 1>(P, p, &z1, w, S, oct, j);
            w[1][0] = __shfl_sync(oct, w[0][0], sh + 1);
        } else {
            wiggles(P, p, z1, w);
        }
        __syncwarp(oct);  // the next crossing's samples replace the coefficients
        if (j != 0) continue;
        const double s = sin(z1);
        ug_hit h;
        h.src = (uint32_t)p;
        h.dx = (float)((a2x * s + w[0][0] - s0x) / s + bx);
        h.dy = (float)((a2y * s + w[1][0] - s0y) / s + by);
        h.chi = (float)chi;
        h.z_emit = (float)z1;
        hits[k] = h;
    }
}

// Density scatter: hit offsets binned over the closed square [-chi_max, chi_max]^2.
// Every hit lies on a front of radius chi <= chi_max, so every hit is counted:
// an offset that FP32 rounding puts a hair past an edge goes to the edge bin.
// Privatised by bands of rows: CTA b owns rows [b rows, (b+1) rows) of the grid in
// shared memory, streams all hits of the frame (coalesced, L2-resident), counts
// the ones in its band with shared-memory atomics and writes its band once,
// coalesced -- no global atomics and no separate clear of the grid.  The hit count
// is n, or *count (capped at cap) when count is given (read on the device).
__global__ void k_fb_density(const ug_hit* __restrict__ hits, int64_t n, const unsigned long long* count,
                             unsigned long long cap, double chiMax, int bins, int rows, uint32_t* grid) {
    extern __shared__ uint32_t band[];
    const int r0 = blockIdx.x * rows;
    const int nr = min(rows, bins - r0);
    const int cells = nr * bins;
    for (int i = threadIdx.x; i < cells; i += blockDim.x) band[i] = 0u;
    __syncthreads();
    if (count) {
        const unsigned long long c = *count;
        n = (int64_t)(c < cap ? c : cap);
    }
    const float inv = (float)(bins / (2.0 * chiMax));
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        const ug_hit h = hits[i];
        int cy = (int)floorf((h.dy + (float)chiMax) * inv);
        cy = cy < 0 ? 0 : (cy >= bins ? bins - 1 : cy);
        if (cy < r0 || cy >= r0 + nr) continue;
        int cx = (int)floorf((h.dx + (float)chiMax) * inv);
        cx = cx < 0 ? 0 : (cx >= bins ? bins - 1 : cx);
        atomicAdd(&band[(cy - r0) * bins + cx], 1u);
    }
    __syncthreads();
    uint32_t* out = grid + (size_t)r0 * bins;
    for (int i = threadIdx.x; i < cells; i += blockDim.x) out[i] = band[i];
}

// Rows per density band: bands of at most 48 KB of shared memory.
inline int density_rows(int bins) { return std::max(1, std::min(bins, 12288 / bins)); }

inline void launch_density(const ug_hit* hits, int64_t n, const unsigned long long* count,
                           unsigned long long cap, double chiMax, int bins, uint32_t* grid, cudaStream_t st) {
    const int rows = density_rows(bins);
    const int bands = (bins + rows - 1) / rows;
    k_fb_density<<<bands, 512, (size_t)rows * bins * 4, st>>>(hits, n, count, cap, chiMax, bins, rows, grid);
}

double h_eta(double z) { return log(tan(z / 2.0)); }

// Host comoving position and velocity of a path (frame_bake.cu:201-228).
void h_comov(const std::vector<double>& a2, const std::vector<double>& a, const std::vector<double>& b,
             const std::vector<double>& f, int nw, int p, double z, double* X, double* Y, double* VX,
             double* VY) {
    const double s = sin(z), c = cos(z);
    double xx[2], dd[2];
    for (int ax = 0; ax < 2; ax++) {
        xx[ax] = a2[(size_t)p * 2 + ax] * s;
        dd[ax] = a2[(size_t)p * 2 + ax] * c;
        for (int j = 0; j < nw; j++) {
            const size_t o = ((size_t)p * 2 + ax) * nw + j;
            xx[ax] += a[o] * (sin(b[o] * z + f[o]) - sin(f[o]));
            dd[ax] += a[o] * b[o] * cos(b[o] * z + f[o]);
        }
    }
    *X = xx[0] / s;
    *Y = xx[1] / s;
    *VX = (dd[0] * s - xx[0] * c) / (s * s);
    *VY = (dd[1] * s - xx[1] * c) / (s * s);
}

// Per (path, axis): s0 = sum_j a_j sin f_j, summed in term order, and the polynomial's
// coefficients a_b e^{i f_b} (coef zeroed by the caller; a frequency listed more than once
// adds up in term order).
// One warp per (path, axis): coalesced reads and the sines spread over the lanes (18 k
// paths of 255 terms: 0.55 -> 0.14 ms against a thread each).
__global__ void __launch_bounds__(128) k_fb_prep(int n, int nw, int bmax, int horner, const double* __restrict__ a,
                                                 const double* __restrict__ b, const double* __restrict__ f,
                                                 double* s0, double2* coef, double* amp) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < (int64_t)n * 2; i += warps) {
        double acc = 0.0, aa = 0.0;
        for (int j0 = 0; j0 < nw; j0 += 32) {
            const int j = j0 + lane;
            double term = 0.0, re = 0.0;
            int fb = -1 - lane;  // no term: unlike any other lane's
            if (j < nw) {
                const int64_t o = i * nw + j;
                double sf, cf;
                sincos(f[o], &sf, &cf);
                aa += fabs(a[o]);
                term = __dmul_rn(a[o], sf);
                re = __dmul_rn(a[o], cf);
                fb = (int)b[o];
            }
            if (horner) {  // the lanes of one frequency take turns: one turn where all differ
                const uint32_t same = __match_any_sync(0xffffffffu, fb);
                const int rank = __popc(same & ((1u << lane) - 1u));
                for (int turn = 0; __any_sync(0xffffffffu, rank >= turn); turn++) {
                    if (rank == turn && j < nw) {
                        double2* c = coef + i * (bmax + 1) + fb;
                        c->x += re;
                        c->y += term;
                    }
                    __syncwarp();
                }
            }
            const int m = min(32, nw - j0);
            for (int q = 0; q < m; q++) acc += __shfl_sync(0xffffffffu, term, q);
        }
        for (int q = 16; q > 0; q >>= 1) aa += __shfl_xor_sync(0xffffffffu, aa, q);
        if (lane == 0) {
            s0[i] = acc;
            // non-negative doubles order as their bits (amp zeroed by the caller)
            atomicMax((unsigned long long*)(amp + (i >> 1)), (unsigned long long)__double_as_longlong(aa));
        }
    }
}

// Dump-layout parameters from the packer (2+1): b as double for the direct sums.
__global__ void k_fb_from_params(int64_t m, const int32_t* bi, double* bd) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x)
        bd[i] = (double)bi[i];
}

// One observer path's parameters on the host (for its comoving position and velocity).
struct ObsPath {
    std::vector<double> a2, a, b, f;  // [2], [2][nw] x3
};

int check_cfg(const ug_frames_cfg* cfg, ug_frames_out* out, int n) {
    if (!cfg || !out || n < 1) return set_error(UG_EINVAL, "frame_bake: bad arguments");
    if (cfg->front < 0 || cfg->front > 2) return set_error(UG_EINVAL, "--front must be speed|fit|budget");
    if (cfg->n_frames < 1 || cfg->n_obs < 1) return set_error(UG_EINVAL, "need >= 1 frame and observer");
    for (int o = 0; o < cfg->n_obs; o++)
        if (cfg->obs_type[o] == 0 && (cfg->obs_path[o] < 0 || cfg->obs_path[o] >= n))
            return set_error(UG_EINVAL, "observer path out of range");
    return UG_OK;
}

// The frame loop over device-resident paths (dump layout, b as double).  With a hit
// buffer the hits of every (frame, observer) come back sorted by (chi, src); without
// one only counts and densities do, and no step waits for the host.
int bake_device(const ug_frames_cfg* cfg, int n, int nw, int bMax, const double* dA2, const double* dA,
                const double* dB, const double* dF, const std::vector<ObsPath>& obs, ug_frames_out* out,
                cudaStream_t st, CallScope& buf) {
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    // Horner when the band is dense enough that one polynomial beats nw sines
    const int horner = (bMax <= 4 * nw) ? 1 : 0;
    double* dS0 = buf.get<double>((size_t)n * 2);
    double2* dC = buf.get<double2>(horner ? (size_t)n * 2 * (bMax + 1) : 1);
    const int Mmax = std::min(kBudgetCap, std::max(kGridRows, 2 * bMax));
    const int NF = cfg->n_frames, NO = cfg->n_obs;
    double* dZg = buf.get<double>((size_t)NF * (Mmax + 1));
    double* dChig = buf.get<double>((size_t)NF * (Mmax + 1));
    const int RpMax = (Mmax + 1 + kGbCols - 1) / kGbCols * kGbCols;
    double* dAmp = buf.get<double>((size_t)n);
    double2* dReach = buf.get<double2>((size_t)bMax + 1);
    double* dBasis = buf.get<double>(horner ? (size_t)2 * (bMax + 1) * RpMax : 1);
    double* dPx = buf.get<double>((size_t)n * (Mmax + 1));
    double* dPy = buf.get<double>((size_t)n * (Mmax + 1));
    const bool want_hits = out->hits != nullptr;
    const bool want_density = cfg->density_bins > 0 && out->density;
    const size_t bins2 = want_density ? (size_t)cfg->density_bins * cfg->density_bins : 0;
    // densities: per (frame, observer) when hits come back one launch at a time,
    // all of them on the device otherwise (one copy at the end)
    uint32_t* dDen = want_density ? buf.get<uint32_t>(want_hits ? bins2 : bins2 * NF * NO) : nullptr;
    const unsigned long long hitCap = 1ull << 24;  // per (frame, observer) launch, frame_bake.cu:515
    unsigned long long* dCount = buf.get<unsigned long long>((size_t)NF * NO);
    if (!dS0 || !dC || !dZg || !dChig || !dBasis || !dReach || !dAmp || !dPx || !dPy || !dCount || (want_density && !dDen))
        return set_error(UG_ENOMEM, "frame_bake: device allocation failed");
    cudaMemsetAsync(dAmp, 0, (size_t)n * 8, st);
    // without hits no step waits for the host: the densities of finished frames are copied
    // on a second stream while the next ones are baked, into pages backed meanwhile
    const bool copies = want_density && !want_hits;
    const int group = (NF + 63) / 64;  // frames per copy
    struct Copies {
        cudaStream_t st = nullptr;
        std::vector<cudaEvent_t> ev;
        ~Copies() {
            if (st) cudaStreamSynchronize(st);  // an early return: none may outlive the call's buffers
            for (cudaEvent_t e : ev) cudaEventDestroy(e);
            if (st) cudaStreamDestroy(st);
        }
    } cp;
    PagesAhead pages;
    if (copies) {
        if (cudaStreamCreateWithFlags(&cp.st, cudaStreamNonBlocking) != cudaSuccess)
            return set_error(UG_ECUDA, "frame_bake: stream creation failed");
        pages.add(out->density, bins2 * NF * NO * 4);
    }
    if (horner) cudaMemsetAsync(dC, 0, (size_t)n * 2 * (bMax + 1) * sizeof(double2), st);
    k_fb_prep<<<(int)std::min<int64_t>(((int64_t)n * 2 + 3) / 4, nsm * 64), 128, 0, st>>>(n, nw, bMax, horner, dA, dB,
                                                                                        dF, dS0, dC, dAmp);
    cudaMemsetAsync(dCount, 0, (size_t)NF * NO * sizeof(unsigned long long), st);
    FPaths P{n, nw, bMax, horner, dA2, dS0, dA, dB, dF, dC, dAmp};
    const double zMin = std::max(2e-3, cfg->zmin_pi * kPiF);
    // fronts and rewind grids of every frame, uploaded once
    std::vector<FFront> fronts(NF);
    std::vector<int> Ks(NF);
    std::vector<double> zgAll((size_t)NF * (Mmax + 1)), chigAll((size_t)NF * (Mmax + 1));
    for (int fi = 0; fi < NF; fi++) {
        const double frac = NF == 1 ? 0.0 : (double)fi / (NF - 1);
        const double zObs = std::min((cfg->from_pi + (cfg->to_pi - cfg->from_pi) * frac) * kPiF, kPiF - 1e-3);
        if (zMin >= zObs) return set_error(UG_EINVAL, "rewind floor >= z_obs");
        FFront& F = fronts[fi];
        F = FFront{};
        F.budget = cfg->front == 2;
        F.reach = dReach;
        F.cheb = F.budget || cfg->cheb;
        F.zObs = zObs;
        F.etaObs = h_eta(zObs);
        F.spd = cfg->front == 0 ? std::max(1e-3, cfg->speed) : -1.0 / h_eta(zMin);
        F.bMax = bMax;
        F.M = F.budget ? std::min(kBudgetCap, std::max(kGridRows, 2 * bMax)) : kGridRows;
        double* zg = zgAll.data() + (size_t)fi * (Mmax + 1);
        double* chig = chigAll.data() + (size_t)fi * (Mmax + 1);
        if (F.budget) {
            F.chiMax = 0.0;
            for (int i = 0; i <= F.M; i++) {
                zg[i] = zObs - (zObs - zMin) * i / F.M;
                chig[i] = reach_of(zg[i], zObs, bMax);
                F.chiMax = std::max(F.chiMax, chig[i]);
            }
        } else {
            F.chiMax = F.spd * (F.etaObs - h_eta(zMin));
            for (int i = 0; i <= F.M; i++) {
                chig[i] = F.chiMax * i / F.M;
                zg[i] = 2.0 * atan(exp(F.etaObs - chig[i] / F.spd));
            }
        }
        Ks[fi] = cfg->wraps >= 0 ? cfg->wraps : (int)ceil((F.chiMax + 4.0) / 2.0);
        if (out->frame_meta) {
            out->frame_meta[fi * 3 + 0] = zObs;
            out->frame_meta[fi * 3 + 1] = F.chiMax;
            out->frame_meta[fi * 3 + 2] = Ks[fi];
        }
    }
    cudaMemcpyAsync(dZg, zgAll.data(), zgAll.size() * 8, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(dChig, chigAll.data(), chigAll.size() * 8, cudaMemcpyHostToDevice, st);
    // Room for the hits of a launch.  A path slower than the front meets it once per image, about
    // chi_max^2 times over the torus: four times that, and the search is repeated with the
    // room it needs where fast or wavering paths meet it more often.  (Room for hitCap
    // in every call is 600 MB.)
    double chiTop = 0.0;
    for (const FFront& F : fronts) chiTop = std::max(chiTop, F.chiMax);
    unsigned long long room = 0;
    ug_hit* dHits = nullptr;
    FCross* dCross = nullptr;
    auto make_room = [&](double want) {
        room = (unsigned long long)std::min<double>((double)hitCap, std::max<double>({1 << 16, 2.0 * room, want}));
        dHits = buf.get<ug_hit>(room);
        dCross = buf.get<FCross>(room);
        return dHits && dCross ? UG_OK : set_error(UG_ENOMEM, "frame_bake: device allocation failed");
    };
    if (const int rc = make_room(4.0 * n * (1.0 + chiTop) * (1.0 + chiTop))) return rc;
    int64_t written = 0;
    out->hits_total = 0;
    std::vector<ug_hit> hh;
    std::vector<unsigned long long> counts((size_t)NF * NO);
search_again:  // (without hits: with more room)
    for (int fi = 0; fi < NF; fi++) {
        const FFront& F = fronts[fi];
        // rings of images that the front reaches (as first_row says; further ones hold no hit)
        int K = std::min(Ks[fi], (int)std::min(32767.0, std::max(2.0, ceil(0.5 * F.chiMax + 2.0))));
        while (K > 2 && 2.0 * K - 4.0 >= F.chiMax) K--;
        const int tiles = ((2 * K + 32) / 32) * ((2 * K + 32) / 32);
        const double* zg = dZg + (size_t)fi * (Mmax + 1);
        const double* chig = dChig + (size_t)fi * (Mmax + 1);
        if (F.budget) k_fb_reach<<<(bMax + 127) / 128, 128, 0, st>>>(bMax, F.zObs, dReach);
        if (horner) {
            const int R = F.M + 1, Rp = (R + kGbCols - 1) / kGbCols * kGbCols;
            k_fb_basis<<<(int)std::min<int64_t>(((int64_t)(bMax + 1) * Rp + 127) / 128, nsm * 16), 128, 0, st>>>(
                bMax, R, Rp, zg, dBasis);
            const int64_t tiles = ((int64_t)n * 2 + kGbRows - 1) / kGbRows * (Rp / kGbCols);
            k_fb_grid_mm<<<(unsigned)tiles, 128, 0, st>>>(P, R, Rp, zg, dBasis, dPx, dPy);
        } else {
            const int64_t tot = (int64_t)n * (F.M + 1);
            k_fb_grid<<<(int)std::min<int64_t>((tot + 127) / 128, 65536), 128, 0, st>>>(P, F.M, zg, dPx, dPy);
        }
        for (int o = 0; o < NO; o++) {
            double ox, oy, bxv = 0.0, byv = 0.0;
            if (cfg->obs_type[o] == 0) {
                double vx, vy;
                const ObsPath& q = obs[o];
                h_comov(q.a2, q.a, q.b, q.f, nw, 0, F.zObs, &ox, &oy, &vx, &vy);
                bxv = sin(F.zObs) * vx / F.spd;
                byv = sin(F.zObs) * vy / F.spd;
            } else {
                ox = cfg->obs_xy[2 * o];
                oy = cfg->obs_xy[2 * o + 1];
            }
            if (out->obs_meta) {
                double* m = out->obs_meta + ((size_t)fi * NO + o) * 4;
                m[0] = ox;
                m[1] = oy;
                m[2] = bxv;
                m[3] = byv;
            }
            unsigned long long* cnt = dCount + (size_t)fi * NO + o;
            auto search = [&]() {
                k_fb_cross<<<(int)std::min<int64_t>(((int64_t)n * tiles + 3) / 4, nsm * 64), 128, 0, st>>>(
                    P, F, ox, oy, K, cfg->obs_type[o] == 0 ? cfg->obs_path[o] : -1, chig, dPx, dPy, dCross, cnt, room);
                k_fb_refine<<<nsm * 8, kFbThreads, 0, st>>>(P, F, ox, oy, zg, chig, dCross, cnt, room, dHits);
            };
            search();
            if (!want_hits) {
                if (want_density)
                    launch_density(dHits, 0, cnt, room, F.chiMax, cfg->density_bins,
                                   dDen + ((size_t)fi * NO + o) * bins2, st);
                continue;
            }
            unsigned long long nh = 0;
            for (;;) {
                cudaError_t e = cudaMemcpyAsync(&nh, cnt, 8, cudaMemcpyDeviceToHost, st);
                if (e == cudaSuccess) e = cudaStreamSynchronize(st);
                if (e != cudaSuccess) {
                    std::string m = std::string("frame_bake: ") + cudaGetErrorString(e);
                    return set_error(UG_ECUDA, m.c_str());
                }
                if (nh <= room || nh > hitCap) break;
                if (const int rc = make_room((double)nh)) return rc;
                cudaMemsetAsync(cnt, 0, 8, st);
                search();
            }
            if (nh > hitCap) return set_error(UG_ECAP, "frame_bake: hit cap overflow (lower the wraps)");
            if (want_density) {
                launch_density(dHits, (int64_t)nh, nullptr, room, F.chiMax, cfg->density_bins, dDen, st);
                cudaMemcpyAsync(out->density + ((size_t)fi * NO + o) * bins2, dDen, bins2 * 4, cudaMemcpyDeviceToHost,
                                st);
            }
            if (out->hit_count) out->hit_count[(size_t)fi * NO + o] = (int64_t)nh;
            out->hits_total += (int64_t)nh;
            if (written + (int64_t)nh <= out->hit_cap) {
                hh.resize(nh);
                if (nh) cudaMemcpyAsync(hh.data(), dHits, nh * sizeof(ug_hit), cudaMemcpyDeviceToHost, st);
                if (cudaStreamSynchronize(st) != cudaSuccess) return set_error(UG_ECUDA, "frame_bake: hit copy failed");
                // device append order is scheduling-dependent: sort by (chi, src)
                std::sort(hh.begin(), hh.end(), [](const ug_hit& x, const ug_hit& y) {
                    return x.chi < y.chi || (x.chi == y.chi && x.src < y.src);
                });
                if (nh) memcpy(out->hits + written, hh.data(), nh * sizeof(ug_hit));
                written += (int64_t)nh;
            }
        }
        if (copies && ((fi + 1) % group == 0 || fi + 1 == NF)) {
            cudaEvent_t ev = nullptr;
            if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess)
                return set_error(UG_ECUDA, "frame_bake: event creation failed");
            cp.ev.push_back(ev);
            cudaEventRecord(ev, st);
        }
    }
    pages.wait();
    for (size_t k = 0; k < cp.ev.size(); k++) {
        const size_t all = bins2 * NO * NF, part = bins2 * NO * group, at = part * k;
        if (cudaStreamWaitEvent(cp.st, cp.ev[k], 0) != cudaSuccess ||
            cudaMemcpyAsync(out->density + at, dDen + at, std::min(part, all - at) * 4, cudaMemcpyDeviceToHost, cp.st) !=
                cudaSuccess)
            return set_error(UG_ECUDA, "frame_bake: density copy failed");
    }
    if (copies && cudaStreamSynchronize(cp.st) != cudaSuccess)
        return set_error(UG_ECUDA, "frame_bake: density copy failed");
    const cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        std::string m = std::string("frame_bake: ") + cudaGetErrorString(e);
        return set_error(UG_ECUDA, m.c_str());
    }
    if (!want_hits) {
        if (cudaMemcpyAsync(counts.data(), dCount, counts.size() * 8, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess)
            return set_error(UG_ECUDA, "frame_bake: count copy failed");
        const unsigned long long most = *std::max_element(counts.begin(), counts.end());
        if (most > hitCap) return set_error(UG_ECAP, "frame_bake: hit cap overflow (lower the wraps)");
        if (most > room) {
            if (const int rc = make_room((double)most)) return rc;
            cudaMemsetAsync(dCount, 0, counts.size() * 8, st);
            for (cudaEvent_t ev : cp.ev) cudaEventDestroy(ev);
            cp.ev.clear();
            goto search_again;
        }
        for (size_t i = 0; i < counts.size(); i++) {
            if (out->hit_count) out->hit_count[i] = (int64_t)counts[i];
            out->hits_total += (int64_t)counts[i];
        }
    }
    if (want_hits && out->hits_total > out->hit_cap) return set_error(UG_ECAP, "frame_bake: hit buffer too small");
    return UG_OK;
}

}  // namespace

__global__ void k_fb_maxb(int64_t m, const int32_t* b, int* out) {
    int mx = 2;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x)
        mx = max(mx, b[i]);
    atomicMax(out, mx);
}

// Largest frequency of device-resident dump parameters.
int max_b_device(const int32_t* b, int64_t m, int* out, cudaStream_t st, CallScope& buf) {
    int* d = buf.get<int>(1);
    if (!d) return set_error(UG_ENOMEM, "frame_bake: device allocation failed");
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaMemsetAsync(d, 0, 4, st);
    k_fb_maxb<<<nsm * 4, 256, 0, st>>>(m, b, d);
    cudaError_t e = cudaMemcpyAsync(out, d, 4, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    return e == cudaSuccess ? UG_OK : set_error(UG_ECUDA, "frame_bake: reduction failed");
}

// Frames of the accepted paths of a packer universe, straight from the device
// (the dump -> frame_bake pipeline without a CSV or host round trip).
int frames_from_params(const ug_frames_cfg* cfg, int n, int nw, int bMax, const double* dA2, const double* dA,
                       const int32_t* dBi, const double* dF, ug_frames_out* out, cudaStream_t st, CallScope& buf) {
    int rc = check_cfg(cfg, out, n);
    if (rc) return rc;
    double* dB = buf.get<double>((size_t)n * 2 * nw);
    if (!dB) return set_error(UG_ENOMEM, "frame_bake: device allocation failed");
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    k_fb_from_params<<<nsm * 8, 256, 0, st>>>((int64_t)n * 2 * nw, dBi, dB);
    std::vector<ObsPath> obs(cfg->n_obs);
    for (int o = 0; o < cfg->n_obs; o++) {
        if (cfg->obs_type[o] != 0) continue;
        const int p = cfg->obs_path[o];
        ObsPath& q = obs[o];
        q.a2.resize(2);
        q.a.resize(2 * nw);
        q.b.resize(2 * nw);
        q.f.resize(2 * nw);
        std::vector<int32_t> bi(2 * nw);
        if (cudaMemcpyAsync(q.a2.data(), dA2 + (size_t)p * 2, 16, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaMemcpyAsync(q.a.data(), dA + (size_t)p * 2 * nw, 16 * nw, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaMemcpyAsync(bi.data(), dBi + (size_t)p * 2 * nw, 8 * nw, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaMemcpyAsync(q.f.data(), dF + (size_t)p * 2 * nw, 16 * nw, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess)
            return set_error(UG_ECUDA, "frame_bake: observer copy failed");
        for (int j = 0; j < 2 * nw; j++) q.b[j] = bi[j];
    }
    return bake_device(cfg, n, nw, bMax, dA2, dA, dB, dF, obs, out, st, buf);
}

}  // namespace ug

using namespace ug;

extern "C" int ug_frame_bake(const ug_frames_cfg* cfg, int32_t n, int32_t nw, const double* a2,
                             const double* a, const double* b, const double* f, ug_frames_out* out) {
    if (nw < 1 || !a2 || !a || !b || !f) return set_error(UG_EINVAL, "frame_bake: bad arguments");
    int rc = check_cfg(cfg, out, n);
    if (rc) return rc;
    int bMax = 2;
    for (size_t i = 0; i < (size_t)n * 2 * nw; i++) bMax = std::max(bMax, (int)b[i]);
    CallScope buf;
    const size_t m = (size_t)n * 2 * nw;
    double* dA2 = buf.get<double>((size_t)n * 2);
    double* dA = buf.get<double>(m);
    double* dB = buf.get<double>(m);
    double* dF = buf.get<double>(m);
    if (!dA2 || !dA || !dB || !dF) return set_error(UG_ENOMEM, "frame_bake: device allocation failed");
    // the library's own stream for this call (host buffers in, host buffers out)
    cudaStream_t st = nullptr;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess)
        return set_error(UG_ECUDA, "frame_bake: stream creation failed");
    struct StreamGuard {
        cudaStream_t s;
        ~StreamGuard() { cudaStreamDestroy(s); }
    } guard{st};
    cudaMemcpyAsync(dA2, a2, (size_t)n * 2 * 8, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(dA, a, m * 8, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(dB, b, m * 8, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(dF, f, m * 8, cudaMemcpyHostToDevice, st);
    std::vector<ObsPath> obs(cfg->n_obs);
    for (int o = 0; o < cfg->n_obs; o++) {
        if (cfg->obs_type[o] != 0) continue;
        const size_t p = (size_t)cfg->obs_path[o];
        obs[o].a2.assign(a2 + p * 2, a2 + p * 2 + 2);
        obs[o].a.assign(a + p * 2 * nw, a + (p + 1) * 2 * nw);
        obs[o].b.assign(b + p * 2 * nw, b + (p + 1) * 2 * nw);
        obs[o].f.assign(f + p * 2 * nw, f + (p + 1) * 2 * nw);
    }
    return bake_device(cfg, n, nw, bMax, dA2, dA, dB, dF, obs, out, st, buf);
}

// ------------------------------------------------------- observer view remap

namespace ug {
namespace {

// The boost of one observer frame, set up on the host with the reference's
// operations in its order (braidlab/frames.py:164-174): cap, static threshold,
// gamma, unit vector, and the two scalar products it forms once.
struct ViewBoost {
    int moving, cheb;
    double bx, by, ux, uy, gamma, gm1, gbx, gby;
};

constexpr double kBetaCap = 0.995;  // FRAME_BETA_CAP (braidlab/frames.py:37)

ViewBoost view_boost(double beta_x, double beta_y, int mode, int cheb) {
    ViewBoost v{};
    v.cheb = cheb != 0;
    if (mode != UG_VIEW_MOVING) return v;
    double bx = beta_x, by = beta_y;
    double bm = std::hypot(bx, by);
    if (bm > kBetaCap) {
        const double s = kBetaCap / bm;
        bx *= s;
        by *= s;
        bm = kBetaCap;
    }
    if (bm <= 1e-6) return v;
    v.moving = 1;
    v.gamma = 1.0 / std::sqrt(1.0 - std::pow(bm, 2.0));
    v.ux = bx / bm;
    v.uy = by / bm;
    v.bx = bx;
    v.by = by;
    v.gbx = v.gamma * bx;
    v.gby = v.gamma * by;
    v.gm1 = v.gamma - 1.0;
    return v;
}

// One thread per hit, FP64, every product and sum rounded on its own (no
// contraction) in the order of braidlab/frames.py:175-188.
__global__ void k_apparent(const ug_hit* __restrict__ hits, int64_t n, ViewBoost v, double* __restrict__ ax,
                           double* __restrict__ ay, double* __restrict__ ld) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const ug_hit h = hits[i];
        const double dx = h.dx, dy = h.dy;
        if (!v.moving) {
            ax[i] = dx;
            ay[i] = dy;
            ld[i] = 0.0;
            continue;
        }
        const double eucl = hypot(dx, dy);
        const bool ok = eucl > 0.0;
        const double nx = ok ? dx / eucl : 0.0, ny = ok ? dy / eucl : 0.0;
        const double bdotn = __dadd_rn(__dmul_rn(v.bx, nx), __dmul_rn(v.by, ny));
        const double udotn = __dadd_rn(__dmul_rn(v.ux, nx), __dmul_rn(v.uy, ny));
        const double dfac = __dmul_rn(v.gamma, __dadd_rn(1.0, bdotn));
        const double gu = __dmul_rn(v.gm1, udotn);
        const double apx = __dadd_rn(__dadd_rn(nx, v.gbx), __dmul_rn(gu, v.ux)) / dfac;
        const double apy = __dadd_rn(__dadd_rn(ny, v.gby), __dmul_rn(gu, v.uy)) / dfac;
        const double chi = h.chi;
        const double norm = v.cheb ? fmax(fabs(apx), fabs(apy)) : 1.0;
        ax[i] = ok ? __dmul_rn(apx, chi) / norm : dx;
        ay[i] = ok ? __dmul_rn(apy, chi) / norm : dy;
        ld[i] = ok ? log(dfac) : 0.0;
    }
}

int check_view(int64_t n, int32_t mode) {
    if (n < 0) return set_error(UG_EINVAL, "apparent_positions: negative hit count");
    if (mode != UG_VIEW_STATIC && mode != UG_VIEW_MOVING)
        return set_error(UG_EINVAL, "apparent_positions: mode must be static|moving");
    return UG_OK;
}

}  // namespace
}  // namespace ug

extern "C" int ug_apparent_positions_async(const ug_hit* d_hits, int64_t n, double beta_x, double beta_y,
                                           int32_t mode, int32_t cheb, double* d_ax, double* d_ay,
                                           double* d_ln_dopp, void* stream) {
    int rc = check_view(n, mode);
    if (rc || n == 0) return rc;
    if (!d_hits || !d_ax || !d_ay || !d_ln_dopp) return set_error(UG_EINVAL, "apparent_positions: null buffer");
    int dev = 0, nsm = 148;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return set_error(UG_ECUDA, "apparent_positions: no CUDA device");
    const int64_t blocks = std::min<int64_t>((n + 255) / 256, (int64_t)nsm * 8);
    k_apparent<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(d_hits, n, view_boost(beta_x, beta_y, mode, cheb),
                                                                   d_ax, d_ay, d_ln_dopp);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return set_error(UG_ECUDA, cudaGetErrorString(e));
    return UG_OK;
}

extern "C" int ug_apparent_positions(const ug_hit* hits, int64_t n, double beta_x, double beta_y, int32_t mode,
                                     int32_t cheb, double* ax, double* ay, double* ln_dopp) {
    int rc = check_view(n, mode);
    if (rc || n == 0) return rc;
    if (!hits || !ax || !ay || !ln_dopp) return set_error(UG_EINVAL, "apparent_positions: null buffer");
    CallScope buf;
    ug_hit* dH = buf.get<ug_hit>((size_t)n);
    double* dO = buf.get<double>((size_t)n * 3);
    if (!dH || !dO) return set_error(UG_ENOMEM, "apparent_positions: device allocation failed");
    if (cudaMemcpy(dH, hits, (size_t)n * sizeof(ug_hit), cudaMemcpyHostToDevice) != cudaSuccess)
        return set_error(UG_ECUDA, "apparent_positions: hit copy failed");
    rc = ug_apparent_positions_async(dH, n, beta_x, beta_y, mode, cheb, dO, dO + n, dO + 2 * n, nullptr);
    if (rc) return rc;
    if (cudaMemcpy(ax, dO, (size_t)n * 8, cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaMemcpy(ay, dO + n, (size_t)n * 8, cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaMemcpy(ln_dopp, dO + 2 * n, (size_t)n * 8, cudaMemcpyDeviceToHost) != cudaSuccess)
        return set_error(UG_ECUDA, "apparent_positions: result copy failed");
    return UG_OK;
}
