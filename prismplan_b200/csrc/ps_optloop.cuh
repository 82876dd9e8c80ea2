// ps_optloop.cuh -- pieces shared by the batched trajectory optimisers
// (ps_chomp.cu, ps_stomp.cu): per-request loop state and the reference's
// bookkeeping, the banded factor of the smoothness metric, the densified
// validity check of an iterate, and the graph-chunk driver. Each translation
// unit that includes this header gets its own private copy of the kernels.
//
// Both reference solvers (CHOMP::solve_runtime_scene, chomp.cu:358-600;
// STOMP::solve_runtime_scene, stomp.cu:565-965) run the same host state
// machine around their updates: seed evaluation, best valid snapshot, a
// polish budget once valid, a two-iteration convergence streak, an iteration
// cap and a wall-clock limit. Here it runs per request on the device.
#pragma once

#include <algorithm>
#include <cfloat>
#include <cmath>

#include "ps_internal.h"
#include "ps_pathkern.cuh"

namespace ps {
namespace {

constexpr int kOptMaxT = 1024;   // longest trajectory of the optimisers
constexpr int kBand = 4;         // bandwidth of R (5-point stencil pair)

struct OptState {
    float best_total, prev_total, last_total, pad0;
    int best_valid, streak, polish_left, iters, step, pad1[3];
};

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// R (central T x T block of dt A^T A over the 6-padded 5-point acceleration
// stencil, chomp_precompute.cpp:20-37, stomp_precompute.cpp:24-42) + 1e-8 I,
// factored as L L^T with L lower-banded: L[i * 5 + k] = L(i, i - k) for
// k = 1..4 and L[i * 5] = 1 / L(i, i). FP64. One block: its threads compute
// the entries of R, kBandRows rows at a time in shared memory, and thread 0
// factors them with the last kBand rows of L in registers (T = 64: 127 us in
// one thread over global memory, now 13 us).
constexpr int kBandThreads = 128, kBandRows = 64;
__global__ void __launch_bounds__(kBandThreads) opt_band_kernel(int T, float dt_f, double* __restrict__ L) {
    __shared__ double rows[kBandRows * 5];
    const double dt = dt_f, inv_dt2 = 1.0 / (dt * dt);
    const double coeff[7] = {0.0, -1.0 / 12.0, 16.0 / 12.0, -30.0 / 12.0, 16.0 / 12.0, -1.0 / 12.0, 0.0};
    const int pad = 6, Np = T + 12;
    auto A = [&](int r, int c) -> double {   // padded stencil matrix entry
        const int j = c - r;
        return (j >= -3 && j <= 3) ? inv_dt2 * coeff[j + 3] : 0.0;
    };
    auto R = [&](int i, int j) -> double {   // central block entry
        const int ci = i + pad, cj = j + pad;
        double s = 0.0;
        for (int r = max(max(ci, cj) - 3, 0); r <= min(min(ci, cj) + 3, Np - 1); ++r) s += A(r, ci) * A(r, cj);
        return dt * s + (i == j ? 1.0e-8 : 0.0);
    };
    double w[kBand][5] = {};   // w[m]: row i - 1 - m of L (zero above the matrix)
    for (int i0 = 0; i0 < T; i0 += kBandRows) {
        const int n = min(kBandRows, T - i0);
        for (int e = threadIdx.x; e < n * 5; e += blockDim.x) {
            const int i = i0 + e / 5, k = e % 5;
            rows[e] = k <= i ? R(i, i - k) : 0.0;
        }
        __syncthreads();
        if (threadIdx.x == 0)
            for (int i = 0; i < n; ++i) {
                double c[5];   // L(i, i - k), k = 1..4, then 1 / L(i, i)
#pragma unroll
                for (int k = kBand; k >= 0; --k) {
                    double s = rows[i * 5 + k];
#pragma unroll
                    for (int m = kBand; m > k; --m) s -= c[m] * (k ? w[k - 1][m - k] : c[m]);
                    c[k] = k ? s * w[k - 1][0] : 1.0 / sqrt(s > 0.0 ? s : 1.0e-300);
                }
#pragma unroll
                for (int m = kBand - 1; m > 0; --m)
#pragma unroll
                    for (int k = 0; k < 5; ++k) w[m][k] = w[m - 1][k];
#pragma unroll
                for (int k = 0; k < 5; ++k) {
                    w[0][k] = c[k];
                    rows[i * 5 + k] = c[k];
                }
            }
        __syncthreads();
        for (int e = threadIdx.x; e < n * 5; e += blockDim.x)
            if (e % 5 <= i0 + e / 5) L[(size_t)i0 * 5 + e] = rows[e];
        __syncthreads();
    }
}

// The two triangular halves of the banded solve, serial in one thread. The
// last kBand results stay in registers, so a step's chain is its kBand
// multiply-subtracts (j ascending, as the textbook loop takes them) and no
// shared-memory round trip; the factor entries do not depend on the chain
// and load ahead of it.
static_assert(kBand == 4, "the register windows below hold kBand = 4 values");

// x <- L^-1 x
__device__ __forceinline__ void band_forward(const double* Ls, double* x, int T) {
    double w0 = 0.0, w1 = 0.0, w2 = 0.0, w3 = 0.0;   // y[i-4], y[i-3], y[i-2], y[i-1]
#pragma unroll 4
    for (int i = 0; i < T; ++i) {
        const double* l = Ls + i * 5;
        double s = x[i];
        if (i >= 4) s -= l[4] * w0;
        if (i >= 3) s -= l[3] * w1;
        if (i >= 2) s -= l[2] * w2;
        if (i >= 1) s -= l[1] * w3;
        const double y = s * l[0];
        x[i] = y;
        w0 = w1;
        w1 = w2;
        w2 = w3;
        w3 = y;
    }
}

// x <- L^-T x
__device__ __forceinline__ void band_backward(const double* Ls, double* x, int T) {
    double v0 = 0.0, v1 = 0.0, v2 = 0.0, v3 = 0.0;   // x[i+1], x[i+2], x[i+3], x[i+4]
#pragma unroll 4
    for (int i = T - 1; i >= 0; --i) {
        double s = x[i];
        if (i + 1 <= T - 1) s -= Ls[(i + 1) * 5 + 1] * v0;
        if (i + 2 <= T - 1) s -= Ls[(i + 2) * 5 + 2] * v1;
        if (i + 3 <= T - 1) s -= Ls[(i + 3) * 5 + 3] * v2;
        if (i + 4 <= T - 1) s -= Ls[(i + 4) * 5 + 4] * v3;
        const double xi = s * Ls[i * 5];
        x[i] = xi;
        v3 = v2;
        v2 = v1;
        v1 = v0;
        v0 = xi;
    }
}

// x <- (L L^T)^-1 x for the banded factor of opt_band_kernel (Ls: 5 T
// doubles, any memory). Serial, one thread.
__device__ __forceinline__ void band_solve(const double* Ls, double* x, int T) {
    band_forward(Ls, x, T);
    band_backward(Ls, x, T);
}

// Sizes of the lists that an iteration's validity check fills (opt_refine_kernel's
// and opt_rest_kernel's); emptied by the bookkeeping for the next one.
struct OptLists {
    int refine, rest, unit;   // unit: the longest rest_unit on the rest list
    __device__ __forceinline__ void empty() { refine = rest = unit = 0; }
};

__global__ void opt_init_kernel(OptState* __restrict__ st, uint8_t* __restrict__ done, int B, int polish,
                                int* __restrict__ n_done, unsigned long long* __restrict__ t0,
                                int* __restrict__ hit_step, OptLists* __restrict__ lists) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b == 0) {
        *n_done = 0;
        lists->empty();
        *t0 = now_ns();
    }
    if (b >= B) return;
    OptState s;
    s.best_total = INFINITY;
    s.prev_total = INFINITY;
    s.last_total = 0.0f;
    s.pad0 = 0.0f;
    s.best_valid = 0;
    s.streak = 0;
    s.polish_left = polish;
    s.iters = 0;
    s.step = 0;
    st[b] = s;
    done[b] = 0;
    hit_step[b] = 0;
}

// One block per request: its segments (theta_t -> theta_t+1) as edges with
// n_sub samples each; 0 samples once the request has finished or when one of
// its waypoints already collides (wp_hit, from the configuration check of the
// same iterate), since the trajectory is then invalid whatever its segments.
// n_sub = ceil(max segment L2 / check_step) as the host loops compute it
// (chomp.cu:459-474, stomp.cu:739-755): FP32, in order, no contraction.
__global__ void opt_segments_kernel(const float* __restrict__ theta, int T, int D, float check_step,
                                    const uint8_t* __restrict__ done, const uint8_t* __restrict__ wp_hit,
                                    float* __restrict__ from, float* __restrict__ to, int* __restrict__ G) {
    __shared__ float red[256];
    const int b = blockIdx.x;
    const float* th = theta + (size_t)b * T * D;
    bool any_hit = false;
    for (int t = threadIdx.x; t < T; t += blockDim.x) any_hit |= wp_hit[(size_t)b * T + t] != 0;
    any_hit = __syncthreads_or(any_hit) != 0;
    float mx = 0.0f;
    for (int t = threadIdx.x; t < T - 1; t += blockDim.x) {
        float d2 = 0.0f;
        for (int d = 0; d < D; ++d) {
            const float df = __fsub_rn(th[(t + 1) * D + d], th[t * D + d]);
            d2 = __fadd_rn(d2, __fmul_rn(df, df));
        }
        mx = fmaxf(mx, __fsqrt_rn(d2));
    }
    red[threadIdx.x] = mx;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] = fmaxf(red[threadIdx.x], red[threadIdx.x + o]);
        __syncthreads();
    }
    const float max_seg = red[0];
    int n_sub = 1;   // capped so that the cast stays defined
    if (check_step > 0.0f && max_seg > check_step)
        n_sub = (int)fminf(ceilf(__fdiv_rn(max_seg, check_step)), 1048576.0f);
    const int g = (done[b] || any_hit) ? 0 : n_sub;
    const size_t e0 = (size_t)b * (T - 1);
    for (int i = threadIdx.x; i < (T - 1) * D; i += blockDim.x) {
        from[e0 * D + i] = th[i];
        to[e0 * D + i] = th[D + i];
    }
    for (int t = threadIdx.x; t < T - 1; t += blockDim.x) G[e0 + t] = g;
}

// Validity of the iterates (opt_validity's usual path): a block takes a slice
// of 32 consecutive segments of a request, a group each. The swept check shows
// most segments clear, their first waypoints included; the other waypoints are
// checked, and the densified samples too when they are few. Else a segment
// goes on a list: of at most 32 samples, or by an ESDF layer without a self
// check (its box of voxels, which is all that the swept check tests, has to be
// far for an interval to be clear), for all warps (opt_rest_kernel), the
// others for a block each first (opt_refine_kernel; an iterate far from its
// goal has some 90 samples on each of 63 segments).
// All that stops when one of the request's slices has a hit: hit_step[b] = the
// request's step + 1 (so that nothing needs clearing between iterations).
// Together the same points as the waypoint and segment checks below (a
// waypoint is the start of its segment; the last one belongs to the last
// slice), so the request's validity is the same. Finished requests are skipped.
//
// Those checks took eight launches (scene and self check of the waypoints,
// segments, header, preparation, two queue passes, self pass, finalize) and
// 141 us of a 256-request CHOMP iteration; this kernel takes 40 us,
// opt_refine_kernel 21 us and opt_rest_kernel 4 us. With the segments' samples
// finished in their own blocks refining took 28 us there, and by an ESDF layer
// 510 us an iteration (64 requests of 200 waypoints; now 144 us on the list).
template <bool kEsdf>
__global__ void __launch_bounds__(kPathThreads, 4) opt_check_kernel(ModelDev md, ps_scene_view sv,
                                                                    const float* __restrict__ theta, int T,
                                                                    float check_step, float margin, int check_self,
                                                                    const uint8_t* __restrict__ done,
                                                                    const OptState* __restrict__ state,
                                                                    int* hit_step, OptLists* lists,
                                                                    int2* __restrict__ refine,
                                                                    RestItem* __restrict__ rest) {
    const int b = blockIdx.y;
    if (done[b]) return;   // uniform over the block
    const int now = state[b].step + 1;
    volatile int* hit_at = hit_step + b;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ int counters[4];
    __shared__ float bmax;
    __shared__ PathBlock blk;
    __shared__ int max_seg_bits;
    PathSmem ps;
    SceneSmem sc;
    if (!path_stage(md, sv, smem, &mbar, counters, &bmax, check_self != 0, false, ps, sc)) {   // fail closed
        if (threadIdx.x == 0) *hit_at = now;
        return;
    }
    const ModelSmem M = model_view(smem);
    const int D = M.H->n_dof;
    const bool self = check_self != 0;
    const float* th = theta + (size_t)b * T * D;
    if (threadIdx.x == 0) blk.hit = max_seg_bits = 0;
    __syncthreads();
    // n_sub of the whole request, as opt_segments_kernel computes it
    float mx = 0.0f;
    for (int t = threadIdx.x; t < T - 1; t += blockDim.x) {
        float d2 = 0.0f;
        for (int d = 0; d < D; ++d) {
            const float df = __fsub_rn(th[(t + 1) * D + d], th[t * D + d]);
            d2 = __fadd_rn(d2, __fmul_rn(df, df));
        }
        mx = fmaxf(mx, __fsqrt_rn(d2));
    }
    atomicMax(&max_seg_bits, __float_as_int(mx));   // non-negative floats order as ints
    __syncthreads();
    const float max_seg = __int_as_float(max_seg_bits);
    int G = 1;   // n_sub, capped so that the cast stays defined
    if (check_step > 0.0f && max_seg > check_step)
        G = (int)fminf(ceilf(__fdiv_rn(max_seg, check_step)), 1048576.0f);
    // the slice's segments, the waypoint and samples 1 .. G, and on the last one its end
    const int seg0 = blockIdx.x * kPathGroups, n = min(kPathGroups, T - 1 - seg0), x = threadIdx.x;
    const bool last = seg0 + n == T - 1;
    if (x < n) blk.item[x] = PathItem{seg0 + x, 0, last && x == n - 1 ? G + 1 : G, self ? 3 : 1};
    path_run<kEsdf>(
        M, md, sc, sv, ps, margin, self, blk, n, G, true, 0,
        [&](int sg, int i, float& a, float& b) {
            a = th[sg * D + i];
            b = th[(sg + 1) * D + i];
        },
        [&]() { return *hit_at == now; },
        [&](const PathItem& it) {
            if (G <= 32 || (kEsdf && !(it.what & 2))) {
                const unsigned bits = rest_bits(1, G, G);
                rest[atomicAdd(&lists->rest, 1)] =
                    RestItem{b * T + it.seg, G, it.what & 1 ? bits : 0u, it.what & 2 ? bits : 0u};
                atomicMax(&lists->unit, rest_unit(G));
            } else {
                refine[atomicAdd(&lists->refine, 1)] = make_int2(b * (T - 1) + it.seg, G << 2 | it.what);
            }
        });
    if (threadIdx.x == 0 && blk.hit) *hit_at = now;
}

// The long segments that opt_check_kernel left, a block each.
template <bool kEsdf>
__global__ void __launch_bounds__(kPathThreads, 4) opt_refine_kernel(ModelDev md, ps_scene_view sv,
                                                                     const float* __restrict__ theta, int T,
                                                                     float margin, int check_self,
                                                                     const OptState* __restrict__ state,
                                                                     int* hit_step, OptLists* lists,
                                                                     const int2* __restrict__ refine,
                                                                     RestItem* __restrict__ rest) {
    const int total = lists->refine;
    if ((int)blockIdx.x >= total) return;   // uniform over the block
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ int counters[4];
    __shared__ float bmax;
    __shared__ PathBlock blk;
    PathSmem ps;
    SceneSmem sc;
    const bool staged = path_stage(md, sv, smem, &mbar, counters, &bmax, check_self != 0, false, ps, sc);
    const ModelSmem M = model_view(smem);
    const bool self = check_self != 0;
    for (int k = blockIdx.x; k < total; k += gridDim.x) {
        const int2 item = refine[k];
        const int b = item.x / (T - 1), sg = item.x - b * (T - 1), G = item.y >> 2;
        const int now = state[b].step + 1;
        volatile int* hit_at = hit_step + b;
        if (!staged) {   // fail closed
            if (threadIdx.x == 0) *hit_at = now;
            continue;
        }
        if (__syncthreads_or(*hit_at == now)) continue;   // the request is known to collide (also: blk's readers are done)
        const float* a = theta + ((size_t)b * T + sg) * M.H->n_dof;
        const float* c = a + M.H->n_dof;
        // samples 1 .. G in up to 32 intervals (opt_check_kernel has the ends)
        const int m = (G - 1) / kPathGroups + 1, n = (G - 1) / m + 1, x = threadIdx.x;
        if (x == 0) blk.hit = blk.left[0] = blk.left[1] = 0;
        if (x < n) blk.item[x] = PathItem{sg, x * m + 1, min((x + 1) * m, G), item.y & 3};
        path_run<kEsdf>(
            M, md, sc, sv, ps, margin, self, blk, n, G, false, 1,
            [&](int, int i, float& ai, float& ci) {
                ai = a[i];
                ci = c[i];
            },
            [&]() { return *hit_at == now; }, [&](const PathItem& it) { path_left(blk, it, G); });
        if (threadIdx.x == 0) {
            if (blk.hit) *hit_at = now;
            if (blk.left[0] | blk.left[1]) {
                rest[atomicAdd(&lists->rest, 1)] = RestItem{b * T + sg, G, blk.left[0], blk.left[1]};
                atomicMax(&lists->unit, rest_unit(G));
            }
        }
    }
}

// The samples that those two left, all warps over all of them.
template <bool kEsdf>
__global__ void __launch_bounds__(kPathThreads, 4) opt_rest_kernel(ModelDev md, ps_scene_view sv,
                                                                   const float* __restrict__ theta, int T,
                                                                   float margin, int check_self,
                                                                   const OptState* __restrict__ state, int* hit_step,
                                                                   const OptLists* lists,
                                                                   const RestItem* __restrict__ rest) {
    const int n = lists->rest;
    if (n == 0) return;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ int counters[4];
    __shared__ float bmax;
    PathSmem ps;
    SceneSmem sc;
    volatile int* hit_at = hit_step;
    auto report = [&](int row) { hit_at[row / T] = state[row / T].step + 1; };
    if (!path_stage(md, sv, smem, &mbar, counters, &bmax, check_self != 0, true, ps, sc)) {   // fail closed
        for (int k = threadIdx.x; k < n; k += blockDim.x) report(rest[k].row);
        return;
    }
    const ModelSmem M = model_view(smem);
    rest_run<kEsdf>(
        M, md, sc, sv, ps, margin, check_self != 0, theta, theta + M.H->n_dof, n, lists->unit,
        [&](int k) { return rest[k]; }, [&](int row) { return hit_at[row / T] == state[row / T].step + 1; }, report);
}

// What opt_bookkeep_block reads an iterate's validity from: hit_step
// (opt_check_kernel) when given, else the segments' and waypoints' verdicts.
struct OptVerdict {
    const uint8_t *seg_valid, *wp_hit;
    const int* hit_step;
    OptLists* lists;   // emptied for the next iteration
};

// Block-level part of the bookkeeping for request b (call from every thread
// of a one-block-per-request kernel; `total` valid in thread 0): validity =
// every segment and every waypoint free; then the reference's state machine
// (chomp.cu:486-555, stomp.cu:764-889) for the request's step k (k = 0 is the
// seed evaluation before the loop, k >= 1 follows the k-th update); theta is
// copied into best when it improved. The reference checks its stop
// conditions at the top of the next iteration; here they are checked at the
// end of this one, which stops at the same iterate.
__device__ void opt_bookkeep_block(int b, const float* __restrict__ th, float total, const OptVerdict v, int T, int D, int n_iter, float conv_eps,
                                   float time_limit_ms, const unsigned long long* __restrict__ t0,
                                   OptState* __restrict__ state, uint8_t* __restrict__ done, float* __restrict__ best,
                                   int* __restrict__ n_done) {
    __shared__ int s_improved;
    bool bad = false;
    if (v.hit_step) {
        bad = v.hit_step[b] == state[b].step + 1;   // every thread, before thread 0 advances the step
    } else {
        for (int t = threadIdx.x; t < T - 1; t += blockDim.x) bad |= v.seg_valid[(size_t)b * (T - 1) + t] == 0;
        for (int t = threadIdx.x; t < T; t += blockDim.x) bad |= v.wp_hit[(size_t)b * T + t] != 0;
    }
    const bool valid = __syncthreads_or(bad) == 0;
    if (threadIdx.x == 0) {
        OptState s = state[b];
        const int k = s.step++;
        bool improved = false, fin = false;
        s.last_total = total;
        if (k == 0) {
            if (valid) {
                s.best_total = total;
                s.best_valid = 1;
                improved = true;
            }
        } else {
            s.iters += 1;
            if (valid && total < s.best_total) {
                s.best_total = total;
                s.best_valid = 1;
                improved = true;
            }
            if (s.best_valid) {
                const float impr = s.prev_total - s.best_total;
                s.streak = (impr >= 0.0f && impr < conv_eps) ? s.streak + 1 : 0;
                s.prev_total = s.best_total;
                s.polish_left -= 1;
                if (s.streak >= 2) fin = true;
            }
        }
        if (k >= n_iter || (s.best_valid && s.polish_left <= 0)) fin = true;
        if (time_limit_ms > 0.0f && (double)(now_ns() - *t0) > (double)time_limit_ms * 1.0e6) fin = true;
        state[b] = s;
        if (fin) {
            done[b] = 1;
            atomicAdd(n_done, 1);
        }
        s_improved = improved;
    }
    __syncthreads();
    if (s_improved)
        for (int i = threadIdx.x; i < T * D; i += blockDim.x) best[(size_t)b * T * D + i] = th[i];
}

// Requests that never became valid return their last iterate and its cost.
__global__ void opt_finalize_kernel(const float* __restrict__ theta, int B, int T, int D,
                                    const OptState* __restrict__ state, float* __restrict__ best,
                                    uint8_t* __restrict__ solved, int* __restrict__ iterations,
                                    float* __restrict__ best_cost) {
    const int b = blockIdx.x;
    if (b >= B) return;
    const OptState s = state[b];
    if (threadIdx.x == 0) {
        solved[b] = s.best_valid ? 1 : 0;
        iterations[b] = s.iters;
        best_cost[b] = s.best_valid ? s.best_total : s.last_total;
    }
    if (!s.best_valid)
        for (int i = threadIdx.x; i < T * D; i += blockDim.x) best[(size_t)b * T * D + i] = theta[(size_t)b * T * D + i];
}

inline size_t a256(size_t x) { return (x + 255) & ~size_t(255); }

// Bump allocator over a caller's workspace (or a dry run for its size).
struct Carver {
    unsigned char* base;
    size_t off = 0;
    template <class P>
    P* take(size_t bytes) {
        P* p = base ? reinterpret_cast<P*>(base + off) : nullptr;
        off += a256(bytes);
        return p;
    }
};

// Loop state, validity scratch and the edge workspace of B requests of T
// waypoints (the part both optimisers share).
struct OptBufs {
    OptState* state;
    uint8_t *done, *evalid, *hit;
    int *G, *n_done, *hit_step;
    OptLists* lists;
    int2* refine;
    RestItem* rest;
    unsigned long long* t0;
    float *from, *to, *ecost;
    double* band;   // 5 T, opt_band_kernel
    void* ews;
    size_t ews_bytes;
};

inline void opt_carve(Carver& c, int B, int T, int D, OptBufs& o) {
    const size_t Bq = (size_t)std::max(B, 1), BT = Bq * std::max(T, 1), E = Bq * std::max(T - 1, 1);
    o.state = c.take<OptState>(sizeof(OptState) * Bq);
    o.done = c.take<uint8_t>(Bq);
    o.evalid = c.take<uint8_t>(E);
    o.hit = c.take<uint8_t>(BT);
    o.G = c.take<int>(4 * E);
    o.n_done = c.take<int>(sizeof(int));
    o.hit_step = c.take<int>(4 * Bq);
    o.lists = c.take<OptLists>(sizeof(OptLists));
    o.refine = c.take<int2>(sizeof(int2) * E);
    o.rest = c.take<RestItem>(sizeof(RestItem) * E);
    o.t0 = c.take<unsigned long long>(sizeof(unsigned long long));
    o.from = c.take<float>(4 * E * D);
    o.to = c.take<float>(4 * E * D);
    o.ecost = c.take<float>(4 * E);
    o.band = c.take<double>(sizeof(double) * 5 * std::max(T, 1));
    o.ews_bytes = ps_edges_workspace_bytes((int)E);
    o.ews = c.take<unsigned char>(o.ews_bytes);
}

// Densified validity of the B iterates theta [B][T][D]: every waypoint and
// every segment sample (G = n_sub), self check as asked; `v` says where the
// bookkeeping finds it. Models and scenes that opt_check_kernel does not serve
// go through the configuration kernel and the persistent edge kernel.
inline int opt_validity(const ps_model* m, const ps_scene_view* scene, const float* theta, int B, int T, int D,
                        float collision_margin, int check_self, float check_step, const OptBufs& o, OptVerdict& v,
                        cudaStream_t q) {
    const int slices = (T - 1 + kPathGroups - 1) / kPathGroups;
    v = OptVerdict{o.evalid, o.hit, nullptr, o.lists};
    if (m->rigid && !g_stats && B <= 65535 && path_serves(m, scene, collision_margin, check_self != 0)) {
        const bool esdf = scene->n_voxel_layers > 0;
        auto k = esdf ? opt_check_kernel<true> : opt_check_kernel<false>;
        auto k2 = esdf ? opt_refine_kernel<true> : opt_refine_kernel<false>;
        auto k3 = esdf ? opt_rest_kernel<true> : opt_rest_kernel<false>;
        const size_t smem = path_smem_bytes(m, scene, check_self != 0), smem3 = rest_smem_bytes(m, scene, check_self != 0);
        PS_TRY_CUDA(allow_smem((const void*)k, smem));
        PS_TRY_CUDA(allow_smem((const void*)k2, smem));
        int grid3 = 1;
        if (int rc = rest_grid(k3, smem3, grid3)) return rc;
        v = OptVerdict{nullptr, nullptr, o.hit_step, o.lists};
        k<<<dim3(slices, B), kPathThreads, smem, q>>>(m->dev, *scene, theta, T, check_step, collision_margin, check_self,
                                                      o.done, o.state, o.hit_step, o.lists, o.refine, o.rest);
        k2<<<(unsigned)std::min<long long>((long long)B * (T - 1), sm_count() * 4ll), kPathThreads, smem, q>>>(
            m->dev, *scene, theta, T, collision_margin, check_self, o.state, o.hit_step, o.lists, o.refine, o.rest);
        k3<<<grid3, kPathThreads, smem3, q>>>(m->dev, *scene, theta, T, collision_margin, check_self, o.state, o.hit_step,
                                              o.lists, o.rest);
        PS_TRY_CUDA(cudaGetLastError());
        return PS_OK;
    }
    ps_edge_params ep{};
    ep.granularity = 1;
    ep.collision_margin = collision_margin;
    ep.check_self = check_self;
    if (int rc = ps_check_configs(m, scene, theta, B * T, collision_margin, check_self ? PS_CHECK_SELF : 0u, o.hit,
                                  nullptr, q))
        return rc;
    opt_segments_kernel<<<B, 256, 0, q>>>(theta, T, D, check_step, o.done, o.hit, o.from, o.to, o.G);
    PS_TRY_CUDA(cudaGetLastError());
    return ps_check_edges(m, scene, o.from, o.to, o.G, B * (T - 1), &ep, o.evalid, o.ecost, nullptr, o.ews,
                          o.ews_bytes, q);
}

// Owns the capture stream and graph of one optimiser call.
struct GraphGuard {
    cudaStream_t cap = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    ~GraphGuard() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        if (cap) cudaStreamDestroy(cap);
    }
};

// Captures kChunk calls of iteration(stream, i) (i = 0..kChunk-1, the
// position inside the chunk) once into a graph on a private stream, then
// replays it on s until n_evals iterations have run or every request has
// finished (read between replays). Every request finishes by its last
// evaluation and finished ones are skipped, so replays past that point are
// never needed.
template <class Iter>
int opt_run_chunks(Iter&& iteration, int n_evals, int B, const int* n_done_dev, cudaStream_t s) {
    constexpr int kChunk = 8;
    cudaStreamCaptureStatus cap_status = cudaStreamCaptureStatusNone;
    PS_TRY_CUDA(cudaStreamIsCapturing(s, &cap_status));
    if (cap_status != cudaStreamCaptureStatusNone)
        return set_error(PS_EINVAL, "the optimiser synchronises and cannot be captured");
    GraphGuard g;
    PS_TRY_CUDA(cudaStreamCreateWithFlags(&g.cap, cudaStreamNonBlocking));
    PS_TRY_CUDA(cudaStreamBeginCapture(g.cap, cudaStreamCaptureModeThreadLocal));
    int rc = PS_OK;
    for (int i = 0; i < kChunk && rc == PS_OK; ++i) rc = iteration(g.cap, i);
    const cudaError_t end_err = cudaStreamEndCapture(g.cap, &g.graph);
    if (rc != PS_OK) return rc;
    if (end_err != cudaSuccess) return cuda_error(end_err, "cudaStreamEndCapture (optimiser iterations)");
    PS_TRY_CUDA(cudaGraphInstantiate(&g.exec, g.graph, 0));
    const int n_chunks = (n_evals + kChunk - 1) / kChunk;
    for (int c = 0; c < n_chunks; ++c) {
        PS_TRY_CUDA(cudaGraphLaunch(g.exec, s));
        if (c + 1 == n_chunks) break;
        int nd = 0;
        PS_TRY_CUDA(cudaMemcpyAsync(&nd, n_done_dev, sizeof(int), cudaMemcpyDeviceToHost, s));
        PS_TRY_CUDA(cudaStreamSynchronize(s));
        if (nd >= B) break;
    }
    return PS_OK;
}

}  // namespace
}  // namespace ps
