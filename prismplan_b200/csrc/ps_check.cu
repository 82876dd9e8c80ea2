// ps_check.cu -- batched configuration check (1, 4 or 16 lanes per
// configuration), sphere FK diagnostics and the FP32 throughput probe.
//
// Replaces check_collision_scene_kernel (code/gpu_planning/cpp/src/planning/
// pRRTC.cu:2337-2389, one 4-thread block per configuration, 1/8 of a warp
// busy) with full warps: lane = configuration, the 3x4 joint frames live in
// registers, the model core arrives in shared memory through one bulk async
// copy, and the obstacle table is staged once per block as prepared 3x3
// boxes. Clearance (PS_CLEARANCE_OBB) is the min over spheres of the
// sphere-vs-box SDF, the OBB counterpart of scene_min_clearance_runtime
// (scene_collision.cuh:339-384, which covers ESDF only).
#include <algorithm>

#include "ps_internal.h"
#include "ps_group.cuh"
#include "ps_verdict.cuh"

namespace ps {

namespace {

constexpr int kCfgThreads = 128;

// SDF of a point from its min outside d^2 over the boxes (as
// sphere_obb_min_sdf): sqrt when outside every box, else the most negative
// max(q) over the boxes that contain it.
__device__ __forceinline__ float sdf_from_min(const SceneSmem& sc, float px, float py, float pz, float mn) {
    if (mn > 0.0f) return sqrtf(mn);
    float inside = 0.0f;
    for (int o = 0; o < sc.n_obbs; ++o) {
        float qx, qy, qz;
        if (fast_box_dsq(sc.obbs[o], px, py, pz, qx, qy, qz) == 0.0f) inside = fminf(inside, fmaxf(qx, fmaxf(qy, qz)));
    }
    return inside;
}

// Fail-closed outputs of a configuration kernel whose model staging gave up:
// this block's configurations (c = block * threads + thread, grid-strided)
// are reported in collision with a NaN clearance.
__device__ __forceinline__ void configs_fail_closed(int n, int threads, uint8_t* hit_out, float* clr_out) {
    if ((int)threadIdx.x >= threads) return;
    for (long long c = (long long)blockIdx.x * threads + threadIdx.x; c < n; c += (long long)gridDim.x * threads) {
        hit_out[c] = 1;
        if (clr_out) clr_out[c] = __int_as_float(0x7fc00000);
    }
}

template <bool kClr, bool kStats>
__global__ void __launch_bounds__(kCfgThreads) check_configs_kernel(ModelDev md, ps_scene_view sv, const float* __restrict__ q,
                                                                   int n, float margin, unsigned flags,
                                                                   uint8_t* __restrict__ hit_out,
                                                                   float* __restrict__ clr_out,
                                                                   unsigned long long* stats) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ int counters[4];
    __shared__ float bmax;
    unsigned char* blob = smem;
    ObbPrep* obbs = reinterpret_cast<ObbPrep*>(smem + md.bytes_core);
    const int nob = max(sv.n_obbs, 1);
    int* orig = reinterpret_cast<int*>(obbs + nob);
    LayerPrep* layers = reinterpret_cast<LayerPrep*>(orig + ((nob + 3) & ~3));
    float* qtile = reinterpret_cast<float*>(layers + PS_MAX_LAYERS);

    if (!stage_model(md, blob, &mbar)) return configs_fail_closed(n, kCfgThreads, hit_out, clr_out);
    SceneSmem sc;
    stage_scene(sv, obbs, orig, layers, counters, &bmax, sc);
    const ModelSmem M = model_view(blob);
    const int D = M.H->n_dof, NJ = M.H->n_joints;
    const bool no_gate = (flags & PS_NO_GATE) != 0;
    const bool want_obb_clr = (flags & PS_CLEARANCE_OBB) != 0;
    const bool want_esdf_clr = (flags & PS_CLEARANCE_ESDF) != 0;
    LaneStats st;
    st.zero();

    for (int base = blockIdx.x * kCfgThreads; base < n; base += gridDim.x * kCfgThreads) {
        // Coalesced load of this block's configurations into shared memory.
        const int cnt = min(kCfgThreads, n - base);
        __syncthreads();
        for (int k = threadIdx.x; k < cnt * D; k += kCfgThreads) qtile[k] = q[(size_t)base * D + k];
        __syncthreads();
        const int c = base + threadIdx.x;
        const bool active = threadIdx.x < cnt;
        const float* qc = qtile + threadIdx.x * D;

        Affine s0, s1, T, a0, a1, TA;
        affine_identity(s0);
        affine_identity(s1);
        affine_identity(a0);
        affine_identity(a1);
        bool hit = false;
        float clr = 1000.0f;
        if (active) {
            if (kStats) st.v[ST_SAMPLES] += 1;
            const bool shares = M.H->approx_shares_chain != 0;
            for (int p = 0; p < NJ; ++p) {
                const JointRec& jr = M.J[p];
                fk_step<true>(jr, p, qc, s0, s1, T);
                if (kStats) st.v[ST_JOINTS] += (p > 0);
                if (!shares) fk_step<true>(M.JA[p], p, qc, a0, a1, TA);
                // ---- approximate gate for this joint ----
                bool flagged = no_gate;
                for (int a = jr.apx_beg; a < jr.apx_end && !flagged; ++a) {
                    const float4 sa = M.A[a];
                    float px, py, pz;
                    sphere_world(shares ? T : TA, sa.x, sa.y, sa.z, px, py, pz);
                    if (kStats) st.v[ST_SPHERES] += 1;
                    const float sr = __fadd_rn(sa.w, margin);
                    // no mask in the approximate pass: the reference passes
                    // sphere index -1 (scene_collision.cuh:584-606), which
                    // turns both the OBB and the ESDF mask lookups off
                    flagged = (sc.n_obbs && sphere_obb_any(sc, nullptr, 0, px, py, pz, sr, nullptr, st)) ||
                              (sc.n_layers && sphere_esdf_any(sc, sv, px, py, pz, sr, nullptr, st));
                }
                // ---- exact spheres of this joint ----
                const int s_first = jr.sph_beg;
                const int s_end = (kClr || (flagged && !hit)) ? jr.sph_end : jr.sph_beg;
                for (int s_i = s_first; s_i < s_end; ++s_i) {
                    const float4 sp = M.S[s_i];
                    float px, py, pz;
                    sphere_world(T, sp.x, sp.y, sp.z, px, py, pz);
                    if (kStats) st.v[ST_SPHERES] += 1;
                    const float sr = __fadd_rn(sp.w, margin);
                    const int so = M.SO[s_i];
                    const uint8_t* acm =
                        sv.sphere_obb_acm_mask ? sv.sphere_obb_acm_mask + (size_t)so * sv.n_obbs : nullptr;
                    const uint8_t* eacm =
                        sv.sphere_acm_mask ? sv.sphere_acm_mask + (size_t)so * sv.n_voxel_layers : nullptr;
                    const bool decide = flagged && !hit;
                    if (kClr) {
                        if (sc.n_obbs && (want_obb_clr || decide)) {
                            float min_dsq;
                            bool any_box;
                            float sdf = sphere_obb_min_sdf(sc, px, py, pz, acm, min_dsq, any_box, st);
                            // sphere_obb_clearance: 1000 sentinel when no box applies
                            if (want_obb_clr && any_box) clr = fminf(clr, __fadd_rn(sdf, -sr));
                            if (decide && any_box) hit = decide_from_min(sc, px, py, pz, sr, min_dsq, acm, st);
                        }
                        if (want_esdf_clr && sc.n_layers)
                            clr = fminf(clr, sphere_esdf_clearance(sc, sv, px, py, pz, sr, eacm, st));
                        if (flagged && !hit && sc.n_layers) hit = sphere_esdf_any(sc, sv, px, py, pz, sr, eacm, st);
                    } else {
                        hit = (sc.n_obbs && sphere_obb_any(sc, nullptr, 0, px, py, pz, sr, acm, st)) ||
                              (sc.n_layers && sphere_esdf_any(sc, sv, px, py, pz, sr, eacm, st));
                        if (hit) break;
                    }
                }
                if (!kClr && __all_sync(__activemask(), hit)) break;
            }
        }
        if (active) {
            hit_out[c] = hit ? 1 : 0;
            if (clr_out) clr_out[c] = clr;
        }
    }
    if (kStats) flush_stats(stats, st);
}

// Fast variant for the common model and scene: the root is the only slot-0
// frame (one 3x4 frame in registers), the approximate chain is the full
// chain, no ACM masks. Same decisions and clearance as check_configs_kernel;
// in clearance mode the exact spheres of a joint are tested 4 per box load.
// Clearance and decision of one exact sphere from its min d^2 over the boxes
// (the per-sphere tail of the fast kernel, kept out of line so that the
// unrolled pair loop stays small in the instruction cache).
__device__ __noinline__ void sphere_tail(const SceneSmem& sc, const ps_scene_view& sv, float px, float py, float pz,
                                         float sr, float mn, bool want_obb_clr, bool want_esdf_clr, bool flagged,
                                         bool& hit, float& clr, unsigned& exact) {
    LaneStats st;
    st.zero();
    if (sc.n_obbs) {
        if (want_obb_clr) clr = fminf(clr, __fadd_rn(sdf_from_min(sc, px, py, pz, mn), -sr));
        if (flagged && !hit) hit = decide_from_min(sc, px, py, pz, sr, mn, nullptr, st);
    }
    if (want_esdf_clr && sc.n_layers) clr = fminf(clr, sphere_esdf_clearance(sc, sv, px, py, pz, sr, nullptr, st));
    if (flagged && !hit && sc.n_layers) hit = sphere_esdf_any(sc, sv, px, py, pz, sr, nullptr, st);
    exact += st.v[ST_EXACT];
}

// Clearance in a scene with ESDF layers (every sphere then needs its lookups,
// so there is little to cull; without layers configs_group_kernel runs).
// Residency, measured: 6 blocks per SM (short per-sphere work, latency-bound).
template <bool kStats>
__global__ void __launch_bounds__(kCfgThreads, 6) check_configs_fast_kernel(ModelDev md, ps_scene_view sv,
                                                                        const float* __restrict__ q, int n,
                                                                        float margin, unsigned flags,
                                                                        uint8_t* __restrict__ hit_out,
                                                                        float* __restrict__ clr_out,
                                                                        unsigned long long* stats) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ int counters[4];
    __shared__ float bmax;
    unsigned char* blob = smem;
    ObbPrep* obbs = reinterpret_cast<ObbPrep*>(smem + md.bytes_core);
    const int nob = max(sv.n_obbs, 1);
    int* orig = reinterpret_cast<int*>(obbs + nob);
    LayerPrep* layers = reinterpret_cast<LayerPrep*>(orig + ((nob + 3) & ~3));
    float* qtile = reinterpret_cast<float*>(layers + PS_MAX_LAYERS);

    if (!stage_model(md, blob, &mbar)) return configs_fail_closed(n, kCfgThreads, hit_out, clr_out);
    SceneSmem sc;
    stage_scene(sv, obbs, orig, layers, counters, &bmax, sc);
    const ModelSmem M = model_view(blob);
    const int D = M.H->n_dof, NJ = M.H->n_joints;
    // the clearance loop's box pairs, after the configuration tiles
    ObbPair* pairs = reinterpret_cast<ObbPair*>(
        reinterpret_cast<unsigned char*>(qtile) + (((size_t)kCfgThreads * D * 4 + 15) & ~size_t(15)));
    const int n_pairs = (sc.n_obbs + 1) / 2;
    __syncthreads();   // the staged boxes are visible
    stage_obb_pairs(sc, pairs);
    __syncthreads();
    const bool no_gate = (flags & PS_NO_GATE) != 0;
    const bool want_obb_clr = (flags & PS_CLEARANCE_OBB) != 0;
    const bool want_esdf_clr = (flags & PS_CLEARANCE_ESDF) != 0;
    LaneStats st;
    st.zero();

    // each warp stages its own 32 configurations: no block-wide barrier
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* wq = qtile + warp * 32 * D;
    for (int base = (blockIdx.x * (kCfgThreads / 32) + warp) * 32; base < n; base += gridDim.x * kCfgThreads) {
        const int cnt = min(32, n - base);
        __syncwarp();
        for (int k = lane; k < cnt * D; k += 32) wq[k] = q[(size_t)base * D + k];
        __syncwarp();
        const int c = base + lane;
        if (lane >= cnt) continue;   // no warp-wide sync below
        const float* qc = wq + lane * D;
        if (kStats) st.v[ST_SAMPLES] += 1;
        Affine T;
        affine_identity(T);
        bool hit = false;
        float clr = 1000.0f;
        for (int p = 0; p < NJ; ++p) {
            const JointRec& jr = M.J[p];
            if (p > 0) {
                const float qi = jr.dof >= 0 ? qc[jr.dof] : 0.0f;
                if (jr.parent_slot == 0) {
                    Affine I;
                    affine_identity(I);
                    joint_compose<true>(jr, qi, I, T);
                } else {
                    joint_compose<true>(jr, qi, T, T);   // rows are read before they are written
                }
                if (kStats) st.v[ST_JOINTS] += 1;
            }
            // ---- approximate gate ----
            bool flagged = no_gate;
            for (int a = jr.apx_beg; a < jr.apx_end && !flagged; ++a) {
                const float4 sa = M.A[a];
                float px, py, pz;
                sphere_world(T, sa.x, sa.y, sa.z, px, py, pz);
                if (kStats) st.v[ST_SPHERES] += 1;
                const float sr = __fadd_rn(sa.w, margin);
                flagged = (sc.n_obbs && sphere_obb_any(sc, nullptr, 0, px, py, pz, sr, nullptr, st)) ||
                          (sc.n_layers && sphere_esdf_any(sc, sv, px, py, pz, sr, nullptr, st));
            }
            // ---- exact spheres: 4 per box load, then singles ----
            int k = jr.sph_beg;
            for (; k + 4 <= jr.sph_end; k += 4) {
                float px[4], py[4], pz[4], mn[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 sp = M.S[k + i];
                    sphere_world(T, sp.x, sp.y, sp.z, px[i], py[i], pz[i]);
                }
                if (kStats) st.v[ST_SPHERES] += 4;
                if (sc.n_obbs) {
                    spheres_min_dsq_pairs<4>(pairs, n_pairs, px, py, pz, mn);
                    if (kStats) st.v[ST_PAIRS] += 4 * sc.n_obbs;
                }
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    sphere_tail(sc, sv, px[i], py[i], pz[i], __fadd_rn(M.S[k + i].w, margin), mn[i], want_obb_clr,
                                want_esdf_clr, flagged, hit, clr, st.v[ST_EXACT]);
            }
            for (; k < jr.sph_end; ++k) {
                const float4 sp = M.S[k];
                float px, py, pz;
                sphere_world(T, sp.x, sp.y, sp.z, px, py, pz);
                if (kStats) st.v[ST_SPHERES] += 1;
                const float sr = __fadd_rn(sp.w, margin);
                float mn = 3.0e38f;
                if (sc.n_obbs) {
                    spheres_min_dsq<1>(sc, &px, &py, &pz, &mn);
                    if (kStats) st.v[ST_PAIRS] += sc.n_obbs;
                }
                sphere_tail(sc, sv, px, py, pz, sr, mn, want_obb_clr, want_esdf_clr, flagged, hit, clr, st.v[ST_EXACT]);
            }
        }
        hit_out[c] = hit ? 1 : 0;
        if (clr_out) clr_out[c] = clr;
    }
    if (kStats) flush_stats(stats, st);
}

// The common configurations: see ps_group.cuh. A warp takes 32 / kSub
// consecutive configurations at a time.
template <int kSub, bool kClr, bool kEsdf, bool kStats>
__global__ void __launch_bounds__(kCfgThreads, 5) configs_group_kernel(ModelDev md, ps_scene_view sv,
                                                                       const float* __restrict__ q, int n,
                                                                       float margin, unsigned flags,
                                                                       uint8_t* __restrict__ hit_out,
                                                                       float* __restrict__ clr_out,
                                                                       unsigned long long* stats) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ int counters[4];
    __shared__ float bmax;
    ObbPrep* obbs = reinterpret_cast<ObbPrep*>(smem + md.bytes_core);
    const int nob = max(sv.n_obbs, 1);
    int* orig = reinterpret_cast<int*>(obbs + nob);
    LayerPrep* layers = reinterpret_cast<LayerPrep*>(orig + ((nob + 3) & ~3));
    float4* obs = reinterpret_cast<float4*>(layers + PS_MAX_LAYERS);
    constexpr int kPer = 32 / kSub;                       // configurations per warp
    constexpr int kTile = kCfgThreads / kSub;             // per block
    if (!stage_model(md, smem, &mbar)) return configs_fail_closed(n, kTile, hit_out, clr_out);
    SceneSmem sc;
    stage_scene(sv, obbs, orig, layers, counters, &bmax, sc);
    box_spheres(sc, obs);
    __syncthreads();
    box_limits(sc, obs);
    __syncthreads();
    const ModelSmem M = model_view(smem);
    const int D = M.H->n_dof;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* wq = reinterpret_cast<float*>(obs + nob) + warp * kPer * D;
    LaneStats st;
    st.zero();
    for (int base = (blockIdx.x * (kCfgThreads / 32) + warp) * kPer; base < n; base += gridDim.x * kTile) {
        const int cnt = min(kPer, n - base);
        __syncwarp();
        for (int k = lane; k < cnt * D; k += 32) wq[k] = q[(size_t)base * D + k];
        __syncwarp();
        const int slot = lane / kSub;
        const bool live = slot < cnt;   // a group past the end repeats the last configuration
        bool hit;
        float clr;
        LaneStats ls;
        ls.zero();
        group_verdict<kSub, kClr, kEsdf, kStats>(M, sc, sv, obs, wq + min(slot, cnt - 1) * D, margin,
                                                 (flags & PS_NO_GATE) != 0, hit, clr, ls);
        if (live && (lane & (kSub - 1)) == 0) {
            hit_out[base + slot] = hit ? 1 : 0;
            if (clr_out) clr_out[base + slot] = clr;
        }
        if (kStats && live) {
            if ((lane & (kSub - 1)) == 0) st.v[ST_SAMPLES] += 1;
            for (int k = 0; k < ST_COUNT; ++k) st.v[k] += ls.v[k];
        }
    }
    if (kStats) flush_stats(stats, st);
}

// Self-collision two-phase check, a group of kSelfSub lanes per
// configuration (group_self_hit), for the configurations without a scene hit.
__global__ void __launch_bounds__(kSelfBlock, 3) self_check_kernel(ModelDev md, const float* __restrict__ q, int n,
                                                                   uint8_t* __restrict__ hit_out,
                                                                   unsigned long long* stats) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ __align__(8) uint64_t mbar;
    unsigned char* blob = smem;
    if (!stage_model(md, blob, &mbar)) return configs_fail_closed(n, kSelfBlock, hit_out, nullptr);
    const ModelSmem M = model_view(blob);
    const int D = M.H->n_dof, NS = M.H->n_spheres, NA = M.H->n_approx, NJ = M.H->n_joints;
    const SelfSmem sm = carve_self<kSelfThreads>(smem + md.bytes_core, NS, NA, NJ, md.bound_from_apx != 0);
    float* qtile = sm.end;
    LaneStats st;
    st.zero();
    const int slot = threadIdx.x / kSelfSub, u = threadIdx.x % kSelfSub;
    for (int base = blockIdx.x * kSelfThreads; base < n; base += gridDim.x * kSelfThreads) {
        const int cnt = min(kSelfThreads, n - base);
        __syncthreads();
        for (int k = threadIdx.x; k < cnt * D; k += kSelfBlock) qtile[k] = q[(size_t)base * D + k];
        __syncthreads();
        if (slot >= cnt) continue;                // uniform over the group
        if (hit_out[base + slot]) continue;       // already in collision with the scene (uniform over the group)
        if (group_self_hit<kSelfThreads>(M, md, qtile + slot * D, sm, slot, u, st) && u == 0)
            hit_out[base + slot] = 1;
    }
    flush_stats(stats, st);
}

// World sphere centres in descriptor order (diagnostics / parity).
__global__ void __launch_bounds__(kCfgThreads) fk_spheres_kernel(ModelDev md, const float* __restrict__ q, int n,
                                                                float* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ __align__(8) uint64_t mbar;
    if (!stage_model(md, smem, &mbar)) {   // fail closed: NaN centres (sizes from the blob in global memory)
        const long long total = (long long)n * reinterpret_cast<const BlobHeader*>(md.blob)->n_spheres * 3;
        for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < total;
             k += (long long)gridDim.x * blockDim.x)
            out[k] = __int_as_float(0x7fc00000);
        return;
    }
    const ModelSmem M = model_view(smem);
    const int D = M.H->n_dof, NJ = M.H->n_joints, NS = M.H->n_spheres;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        float qc[PS_MAX_DOF];
        for (int d = 0; d < D; ++d) qc[d] = q[(size_t)c * D + d];
        Affine s0, s1, T;
        affine_identity(s0);
        affine_identity(s1);
        for (int p = 0; p < NJ; ++p) {
            const JointRec& jr = M.J[p];
            fk_step<true>(jr, p, qc, s0, s1, T);
            for (int k = jr.sph_beg; k < jr.sph_end; ++k) {
                const float4 s = M.S[k];
                float px, py, pz;
                sphere_world(T, s.x, s.y, s.z, px, py, pz);
                float* o = out + ((size_t)c * NS + M.SO[k]) * 3;
                o[0] = px;
                o[1] = py;
                o[2] = pz;
            }
        }
    }
}

// One sphere-vs-box pair per thread, decided as every kernel decides it:
// prepared box (prep_box), 3x3 fast squared distance, definite outside the
// guard band of this pair (the narrowest any kernel uses: S = |p|inf and
// B = this box's |t|inf + |h|inf), the reference sequence inside it. Also the
// exact-sequence local coordinates (ref_to_local). Diagnostics.
__global__ void obb_pairs_kernel(const float4* __restrict__ dims, const float4* __restrict__ pose,
                                 const float4* __restrict__ sph, int n, uint8_t* __restrict__ decision,
                                 float* __restrict__ local) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const ObbPrep o = prep_box(dims[i], pose[2 * i], pose[2 * i + 1]);
        const float4 sp = sph[i];
        float lo, hi;
        guard_thresholds(sp.x, sp.y, sp.z, sp.w, o.h.w, lo, hi);
        float qx, qy, qz;
        const float d = fast_box_dsq(o, sp.x, sp.y, sp.z, qx, qy, qz);
        const bool band = d >= lo && d < hi;
        const bool hit = d < lo ? true : (d >= hi ? false : ref_obb_hit(o, sp.x, sp.y, sp.z, sp.w));
        decision[i] = (uint8_t)((hit ? 1 : 0) | (band ? 2 : 0));
        if (local) {
            float lx, ly, lz;
            ref_to_local(o.q.x, o.q.y, o.q.z, o.q.w, o.r0.w, o.r1.w, o.r2.w, sp.x, sp.y, sp.z, lx, ly, lz);
            local[3 * i] = lx;
            local[3 * i + 1] = ly;
            local[3 * i + 2] = lz;
        }
    }
}

// FP32 FMA throughput probe: 8 independent FMA chains per thread.
__global__ void __launch_bounds__(256) fma_probe_kernel(float* out, int iters, float a, float b) {
    float x0 = threadIdx.x * 1e-7f, x1 = x0 + 1e-7f, x2 = x0 + 2e-7f, x3 = x0 + 3e-7f;
    float x4 = x0 + 4e-7f, x5 = x0 + 5e-7f, x6 = x0 + 6e-7f, x7 = x0 + 7e-7f;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            x0 = fmaf(x0, a, b); x1 = fmaf(x1, a, b); x2 = fmaf(x2, a, b); x3 = fmaf(x3, a, b);
            x4 = fmaf(x4, a, b); x5 = fmaf(x5, a, b); x6 = fmaf(x6, a, b); x7 = fmaf(x7, a, b);
        }
    }
    float s = ((x0 + x1) + (x2 + x3)) + ((x4 + x5) + (x6 + x7));
    if (s == 12345.678f) out[0] = s;   // keeps the chains live
}

}  // namespace

unsigned long long* g_stats = nullptr;
cudaEvent_t g_ev_start = nullptr, g_ev_stop = nullptr;

}  // namespace ps

using namespace ps;

extern "C" int ps_set_stats(unsigned long long* dev_counters) {
    ps::g_stats = dev_counters;
    return PS_OK;
}

extern "C" int ps_set_timing_events(void* start, void* stop) {
    ps::g_ev_start = (cudaEvent_t)start;
    ps::g_ev_stop = (cudaEvent_t)stop;
    return PS_OK;
}

namespace {

using ConfigKernel = void (*)(ModelDev, ps_scene_view, const float*, int, float, unsigned, uint8_t*, float*,
                              unsigned long long*);

template <bool kClr, bool kEsdf, bool kStats>
ConfigKernel pick_lanes(int sub) {
    return sub == 1 ? configs_group_kernel<1, kClr, kEsdf, kStats>
                    : (sub == 4 ? configs_group_kernel<4, kClr, kEsdf, kStats>
                                : configs_group_kernel<16, kClr, kEsdf, kStats>);
}

ConfigKernel pick_group(int sub, bool clr, bool esdf, bool stats) {
    if (clr) return stats ? pick_lanes<true, false, true>(sub) : pick_lanes<true, false, false>(sub);
    if (esdf) return stats ? pick_lanes<false, true, true>(sub) : pick_lanes<false, true, false>(sub);
    return stats ? pick_lanes<false, false, true>(sub) : pick_lanes<false, false, false>(sub);
}

}  // namespace

extern "C" int ps_check_configs(const ps_model* m, const ps_scene_view* scene, const float* q, int n,
                                float margin, unsigned flags, uint8_t* hit, float* clearance, void* stream) {
    PS_NVTX("ps_check_configs");
    clear_error();
    if (!m) return set_error(PS_EINVAL, "model is NULL");
    if (n < 0) return set_error(PS_EINVAL, "n < 0");
    if (n == 0) return PS_OK;
    if (!q || !hit) return set_error(PS_EINVAL, "q / hit is NULL");
    if (int rc = validate_scene(m, scene)) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    // Without a clearance source the output (if any) is the 1000 sentinel.
    const bool clr = clearance != nullptr &&
                     ((flags & PS_CLEARANCE_OBB) || ((flags & PS_CLEARANCE_ESDF) && scene->n_voxel_layers > 0));
    const bool fast = m->root_slot_only && m->info.approx_shares_chain && !scene->sphere_obb_acm_mask &&
                      !scene->sphere_acm_mask;
    void (*k)(ModelDev, ps_scene_view, const float*, int, float, unsigned, uint8_t*, float*, unsigned long long*);
    const size_t tables = (size_t)m->dev.bytes_core + scene_smem_bytes(scene);
    size_t smem;
    int tile = kCfgThreads, per_sm = 8;
    // (sphere_obb_acm_mask_approx changes no result: the approximate gate applies no mask)
    if (fast && !(clr && scene->n_voxel_layers > 0)) {
        const int sub = config_lanes(n);
        k = pick_group(sub, clr, scene->n_voxel_layers > 0, g_stats != nullptr);
        tile = kCfgThreads / sub;
        smem = tables + (size_t)16 * std::max(scene->n_obbs, 1) + (size_t)tile * m->info.n_dof * 4;
    } else {
        smem = tables + (size_t)kCfgThreads * m->info.n_dof * 4;
        smem = ((smem + 15) & ~size_t(15)) + (size_t)((scene->n_obbs + 1) / 2) * sizeof(ObbPair);   // box pairs
        if (fast) k = g_stats ? check_configs_fast_kernel<true> : check_configs_fast_kernel<false>;
        else k = clr ? (g_stats ? check_configs_kernel<true, true> : check_configs_kernel<true, false>)
                     : (g_stats ? check_configs_kernel<false, true> : check_configs_kernel<false, false>);
    }
    if ((flags >> 8) & 15u) per_sm = (int)((flags >> 8) & 15u);   // PS_CONFIG_BLOCKS_PER_SM
    const int blocks_needed = (n + tile - 1) / tile;
    const int grid = std::max(1, std::min(blocks_needed, sm_count() * per_sm));
    PS_TRY_CUDA(allow_smem((const void*)k, smem));
    mark_start(s);
    k<<<grid, kCfgThreads, smem, s>>>(m->dev, *scene, q, n, margin, flags, hit, clearance, g_stats);
    mark_stop(s);
    PS_TRY_CUDA(cudaGetLastError());
    if (flags & PS_CHECK_SELF) {
        if (int rc = check_self_fits(m)) return rc;
        const size_t ss = self_smem_bytes(m);
        PS_TRY_CUDA(allow_smem((const void*)self_check_kernel, ss));
        const int g2 = std::max(1, std::min((n + kSelfThreads - 1) / kSelfThreads, sm_count() * 8));
        self_check_kernel<<<g2, kSelfBlock, ss, s>>>(m->dev, q, n, hit, g_stats);
        PS_TRY_CUDA(cudaGetLastError());
    }
    return PS_OK;
}

extern "C" int ps_fk_spheres(const ps_model* m, const float* q, int n, float* out, void* stream) {
    PS_NVTX("ps_fk_spheres");
    clear_error();
    if (!m || (n > 0 && (!q || !out))) return set_error(PS_EINVAL, "NULL argument");
    if (int rc = check_model_device(m)) return rc;
    if (n <= 0) return PS_OK;
    cudaStream_t s = (cudaStream_t)stream;
    size_t smem = (size_t)m->dev.bytes_core;
    PS_TRY_CUDA(allow_smem((const void*)fk_spheres_kernel, smem));
    const int grid = std::max(1, std::min((n + kCfgThreads - 1) / kCfgThreads, sm_count() * 8));
    fk_spheres_kernel<<<grid, kCfgThreads, smem, s>>>(m->dev, q, n, out);
    PS_TRY_CUDA(cudaGetLastError());
    return PS_OK;
}

extern "C" int ps_debug_obb_pairs(const float* obb_dims, const float* obb_pose, const float* spheres, int n,
                                  uint8_t* decision, float* local_xyz, void* stream) {
    PS_NVTX("ps_debug_obb_pairs");
    clear_error();
    if (n < 0) return set_error(PS_EINVAL, "n < 0");
    if (n == 0) return PS_OK;
    if (!obb_dims || !obb_pose || !spheres || !decision) return set_error(PS_EINVAL, "NULL argument");
    if (((reinterpret_cast<uintptr_t>(obb_dims) | reinterpret_cast<uintptr_t>(obb_pose) |
          reinterpret_cast<uintptr_t>(spheres)) & 15) != 0)
        return set_error(PS_EINVAL, "inputs must be 16-byte aligned");
    const int grid = std::max(1, std::min((n + 255) / 256, sm_count() * 8));
    obb_pairs_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(
        reinterpret_cast<const float4*>(obb_dims), reinterpret_cast<const float4*>(obb_pose),
        reinterpret_cast<const float4*>(spheres), n, decision, local_xyz);
    PS_TRY_CUDA(cudaGetLastError());
    return PS_OK;
}

extern "C" int ps_probe_fp32_peak(double* flops_per_s, void* stream) {
    clear_error();
    if (!flops_per_s) return set_error(PS_EINVAL, "NULL output");
    cudaStream_t s = (cudaStream_t)stream;
    float* d = nullptr;
    PS_TRY_CUDA(cudaMalloc(&d, sizeof(float)));
    const int blocks = sm_count() * 8, threads = 256, iters = 4096;
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    fma_probe_kernel<<<blocks, threads, 0, s>>>(d, 64, 1.0000001f, 1e-7f);   // warm-up
    cudaEventRecord(a, s);
    fma_probe_kernel<<<blocks, threads, 0, s>>>(d, iters, 1.0000001f, 1e-7f);
    cudaEventRecord(b, s);
    cudaError_t e = cudaEventSynchronize(b);
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFree(d);
    if (e != cudaSuccess) return cuda_error(e, "fma probe");
    const double flops = 2.0 * 8 * 16 * (double)iters * blocks * threads;
    *flops_per_s = flops / (ms * 1e-3);
    return PS_OK;
}

extern "C" int ps_tune_configs(const ps_model* m, const ps_scene_view* scene, const float* q, int n, float margin,
                               unsigned flags, uint8_t* hit, float* clearance, void* stream, ps_config_tuning* out,
                               unsigned* tuned_flags) {
    PS_NVTX("ps_tune_configs");
    clear_error();
    if (!tuned_flags) return set_error(PS_EINVAL, "tuned_flags is NULL");
    cudaStream_t s = (cudaStream_t)stream;
    const unsigned base = flags & ~(15u << 8);
    cudaEvent_t a = nullptr, z = nullptr;
    PS_TRY_CUDA(cudaEventCreate(&a));
    if (cudaEventCreate(&z) != cudaSuccess) {
        cudaEventDestroy(a);
        return cuda_error(cudaGetLastError(), "tuning events");
    }
    float best = 3.0e38f, def_ms = 0.0f;
    int best_k = 8, n_cand = 0, rc = PS_OK;
    for (int k : {8, 1, 2, 3, 4, 6, 12}) {
        const unsigned f = base | PS_CONFIG_BLOCKS_PER_SM(k);
        rc = ps_check_configs(m, scene, q, n, margin, f, hit, clearance, stream);   // warm-up
        float ms[3];
        for (int r = 0; r < 3 && rc == PS_OK; ++r) {
            cudaEventRecord(a, s);
            rc = ps_check_configs(m, scene, q, n, margin, f, hit, clearance, stream);
            cudaEventRecord(z, s);
            if (rc == PS_OK && cudaEventSynchronize(z) != cudaSuccess) rc = cuda_error(cudaGetLastError(), "tuning run");
            ms[r] = 0.0f;
            cudaEventElapsedTime(&ms[r], a, z);
        }
        if (rc) break;
        std::sort(ms, ms + 3);
        ++n_cand;
        if (k == 8) def_ms = ms[1];
        if (ms[1] < best) {
            best = ms[1];
            best_k = k;
        }
    }
    cudaEventDestroy(a);
    cudaEventDestroy(z);
    if (rc) return rc;
    *tuned_flags = base | PS_CONFIG_BLOCKS_PER_SM(best_k);
    if (out) *out = ps_config_tuning{best_k, best, def_ms, n_cand};
    return PS_OK;
}
