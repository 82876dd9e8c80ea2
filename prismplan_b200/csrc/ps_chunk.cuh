// ps_chunk.cuh -- verdict of 32 consecutive samples of an edge, one lane each:
// the scene check of the edge queue (ps_edgekern.cuh) and of the samples that
// the one-block-per-path kernels leave (ps_pathkern.cuh).
#pragma once

#include "ps_internal.h"
#include "ps_verdict.cuh"

namespace ps {
namespace {

constexpr unsigned kFull = 0xffffffffu;

struct WarpScratch {
    float* q;          // [32 * D]
    uint16_t* cand;    // [n_obbs]
    const float4* obs; // [n_obbs] box centre, .w its part of the broad-phase limit (block-wide)
};

// Fast path of process_chunk for the common scene: the approximate chain is
// the full chain, no ACM masks, no ESDF layers, no clearance. Same verdict;
// fewer live registers and a per-joint guard band. Exact spheres are tested 4
// at a time (2 with ESDF layers) against each surviving box (one box load per
// group), then decided from their min d^2 with the exact re-decision inside
// the guard band.
//
// Code size matters here: the kernel issues about 3 of every 4 cycles, and
// instruction fetch stalls were the third largest stall reason. The box loops
// are kept rolled and the rare band re-decision is out of line, which took
// 7 % (boxes only) and 15 % (boxes and ESDF) off the kernel time.

// Exact re-decision of one sphere whose min d^2 fell inside the guard band
// (lo, hi): the band's boxes are decided one by one with the reference test.
__device__ __noinline__ bool band_redecide(const SceneSmem& sc, const uint16_t* cand, int ncand, float px, float py,
                                           float pz, float sr, float lo, float hi, LaneStats& st) {
    for (int k = 0; k < ncand; ++k) {
        const ObbPrep& o = sc.obbs[cand[k]];
        float qx, qy, qz;
        const float d = fast_box_dsq(o, px, py, pz, qx, qy, qz);
        if (d < lo) return true;
        if (d < hi) {
            st.v[ST_EXACT] += 1;
            if (ref_obb_hit(o, px, py, pz, sr)) return true;
        }
    }
    return false;
}

// Decide one sphere from its min d^2 over the candidate boxes: definite
// outside the guard band, exact re-decision of the band's boxes otherwise.
__device__ __forceinline__ bool decide_band(const SceneSmem& sc, const uint16_t* cand, int ncand, float px, float py,
                                            float pz, float sr, float g, float mn, LaneStats& st) {
    const float a = fmaxf(sr - g, 0.0f), b = sr + g;
    const float lo = a * a * (1.0f - 1.0e-6f), hi = b * b * (1.0f + 1.0e-6f);
    if (mn < lo) return true;
    if (mn >= hi) return false;
    return band_redecide(sc, cand, ncand, px, py, pz, sr, lo, hi, st);
}

// kN spheres (positions in registers) against every candidate box: one box
// load per kN pair tests. Returns whether any of them hits.
template <int kN, bool kStats>
__device__ __forceinline__ bool spheres_hit(const SceneSmem& sc, const uint16_t* cand, int ncand, const float* px,
                                            const float* py, const float* pz, const float* sr, float g,
                                            LaneStats& st) {
    float mn[kN];
#pragma unroll
    for (int i = 0; i < kN; ++i) mn[i] = 3.0e38f;
#pragma unroll 1
    for (int k = 0; k < ncand; ++k) {
        const ObbPrep& o = sc.obbs[cand[k]];
        const float4 r0 = o.r0, r1 = o.r1, r2 = o.r2, h = o.h;
#pragma unroll
        for (int i = 0; i < kN; ++i) {
            const float lx = fmaf(r0.z, pz[i], fmaf(r0.y, py[i], fmaf(r0.x, px[i], r0.w)));
            const float ly = fmaf(r1.z, pz[i], fmaf(r1.y, py[i], fmaf(r1.x, px[i], r1.w)));
            const float lz = fmaf(r2.z, pz[i], fmaf(r2.y, py[i], fmaf(r2.x, px[i], r2.w)));
            const float cx = fmaxf(fabsf(lx) - h.x, 0.0f), cy = fmaxf(fabsf(ly) - h.y, 0.0f),
                        cz = fmaxf(fabsf(lz) - h.z, 0.0f);
            mn[i] = fminf(mn[i], fmaf(cz, cz, fmaf(cy, cy, cx * cx)));
        }
    }
    if (kStats) st.v[ST_PAIRS] += ncand * kN;
    bool hit = false;
#pragma unroll
    for (int i = 0; i < kN; ++i)
        if (!hit) hit = decide_band(sc, cand, ncand, px[i], py[i], pz[i], sr[i], g, mn[i], st);
    return hit;
}

// Approximate gate of one joint for this lane: any approximate sphere hits a
// candidate box (or an ESDF layer).
template <bool kStats, bool kEsdf>
__device__ __forceinline__ bool joint_gate(const ModelSmem& M, const SceneSmem& sc, const ps_scene_view& sv,
                                           const JointRec& jr, const Affine& T, float margin, const WarpScratch& ws,
                                           int ncand, float g, LaneStats& st) {
    bool flagged = false;
    for (int a = jr.apx_beg; a < jr.apx_end && !flagged; ++a) {
        const float4 sa = M.A[a];
        float px, py, pz;
        sphere_world(T, sa.x, sa.y, sa.z, px, py, pz);
        const float sr = __fadd_rn(sa.w, margin);
        if (kStats) st.v[ST_SPHERES] += 1;
        flagged = spheres_hit<1, kStats>(sc, ws.cand, ncand, &px, &py, &pz, &sr, g, st) ||
                  (kEsdf && sphere_esdf_any(sc, sv, px, py, pz, sr, nullptr, st));
    }
    return flagged;
}

template <bool kStats, bool kEsdf>
__device__ bool process_chunk_fast(const ModelSmem& M, const SceneSmem& sc, const ps_scene_view& sv,
                                   float margin, const float* __restrict__ from, const float* __restrict__ to, int e,
                                   int G, int before, WarpScratch ws, LaneStats& st_out) {
    const int lane = threadIdx.x & 31;
    LaneStats st;
    st.zero();
    const int D = M.H->n_dof, NJ = M.H->n_joints;
    // samples before + 1 .. before + 32 of the edge; sampling rule as in
    // process_chunk (edge_eval.cuh:110-121)
    const int j_raw = before + lane + 1;
    const bool in_range = j_raw <= G;
    const bool start_lane = !in_range && (G % 16) != 0 && j_raw == G + 1;
    const bool real = in_range || start_lane;
    const int j = in_range ? j_raw : (start_lane ? 0 : G);
    const float t = __fdiv_rn((float)j, (float)G);
    const float* a = from + (size_t)e * D;
    const float* b = to + (size_t)e * D;
    float* qc = ws.q + lane * D;
    for (int i = 0; i < D; ++i) {
        const float ai = __ldg(a + i), bi = __ldg(b + i);
        qc[i] = __fmaf_rn(t, __fadd_rn(bi, -ai), ai);
    }
    __syncwarp();
    if (kStats && real) st.v[ST_SAMPLES] += 1;
    // Slot 0 holds only the root's identity frame (checked on the host), so a
    // joint's parent frame is the identity or the current frame: one 3x4
    // frame in registers. Composing with the identity reproduces the step
    // exactly, as the reference's slot walk does.
    Affine T;
    affine_identity(T);
    bool hit = false;
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
        if (jr.bound.w < 0.0f || (sc.n_obbs == 0 && !kEsdf)) continue;   // nothing to test (uniform)
        // ---- warp broad phase: one sphere around the joint's bound spheres of
        //      all 32 samples, centred on the middle sample's ----
        float cx, cy, cz;
        sphere_world(T, jr.bound.x, jr.bound.y, jr.bound.z, cx, cy, cz);
        const float mx = __shfl_sync(kFull, cx, 16), my = __shfl_sync(kFull, cy, 16),
                    mz = __shfl_sync(kFull, cz, 16);
        const float dx = cx - mx, dy = cy - my, dz = cz - mz;
        // max over lanes in one warp reduction: non-negative floats order as their bits
        const float r2 = __uint_as_float(__reduce_max_sync(kFull, __float_as_uint(fmaf(dz, dz, fmaf(dy, dy, dx * dx)))));
        const float Sm = fmaxf(fabsf(mx), fmaxf(fabsf(my), fabsf(mz)));
        // the square root only widens a conservative bound: the approximate
        // one, raised by 1e-6 relative (far above its error), is enough
        const float r2c = fmaxf(r2, 1.0e-30f);
        float Rc = r2c * rsqrtf(r2c) * (1.0f + 1.0e-6f) + jr.bound.w + fmaxf(margin, 0.0f);
        Rc += 4.0f * (Sm + Rc + sc.Bmax + 1.0f) * PS_GUARD_K;
        const float Rcl = Rc * sc.Mscale;   // world radius -> box-frame radius (map stretch)
        const float Rc2 = Rcl * Rcl;
        const float Rj = (Rc * (1.0f + 4.0f * PS_GUARD_K) + 4.0f * PS_GUARD_K * (Sm + 1.0f)) * (1.0f + 1.0e-6f);
        int ncand = 0;
        __syncwarp();
#pragma unroll 1
        for (int base = 0; base < sc.n_obbs; base += 32) {
            const int o = base + lane;
            bool keep = false;
            if (o < sc.n_obbs) {
                // circumscribed-sphere test first, the box distance only if it passes
                const float4 ob = ws.obs[o];
                const float ex = ob.x - mx, ey = ob.y - my, ez = ob.z - mz;
                const float lim = Rj + ob.w;   // see box_limits
                if (fmaf(ez, ez, fmaf(ey, ey, ex * ex)) < lim * lim) {
                    float qx, qy, qz;
                    keep = fast_box_dsq(sc.obbs[o], mx, my, mz, qx, qy, qz) < Rc2;
                }
                if (kStats) st.v[ST_CULL] += 1;
            }
            const unsigned bal = __ballot_sync(kFull, keep);
            if (keep) ws.cand[ncand + __popc(bal & ((1u << lane) - 1u))] = (uint16_t)o;
            ncand += __popc(bal);
        }
        __syncwarp();
        // ESDF layers within reach of any sphere of the joint over the chunk (uniform)
        const bool esdf = kEsdf && esdf_reachable(sc, mx, my, mz, Rc);
        if (ncand == 0 && !esdf) continue;   // nothing reachable from any lane (uniform)
        // Per-joint guard: every sphere of the joint lies within bound.w of c.
        const float S = fmaxf(fabsf(cx), fmaxf(fabsf(cy), fabsf(cz))) + jr.bound.w;
        const float g = (S + sc.Bmax + 1.0f) * PS_GUARD_K;
        // ---- the joint's verdict is gate && exact (two_phase_cc.cuh:57-138).
        //      Boxes only: exact spheres first, the approximate gate only for a
        //      lane whose exact spheres hit. With an ESDF layer in reach the
        //      gate comes first, so unflagged joints skip the exact spheres'
        //      ESDF lookups. ----
        if (!hit) {
            bool flagged = false;
            if (esdf) flagged = joint_gate<kStats, true>(M, sc, sv, jr, T, margin, ws, ncand, g, st);
            bool ex = false;
            if (!esdf || flagged) {
                int k = jr.sph_beg;
                // spheres per box load: 4 with boxes only, 2 when the ESDF
                // lookups share the registers (measured best for each)
                constexpr int kG = kEsdf ? 2 : 4;
                for (; k + kG <= jr.sph_end && !ex; k += kG) {
                    float px[kG], py[kG], pz[kG], sr[kG];
#pragma unroll
                    for (int i = 0; i < kG; ++i) {
                        const float4 sp = M.S[k + i];
                        sphere_world(T, sp.x, sp.y, sp.z, px[i], py[i], pz[i]);
                        sr[i] = __fadd_rn(sp.w, margin);
                    }
                    if (kStats) st.v[ST_SPHERES] += kG;
                    ex = spheres_hit<kG, kStats>(sc, ws.cand, ncand, px, py, pz, sr, g, st);
                    if (esdf)
#pragma unroll
                        for (int i = 0; i < kG; ++i)
                            if (!ex) ex = sphere_esdf_any(sc, sv, px[i], py[i], pz[i], sr[i], nullptr, st);
                }
                for (; k < jr.sph_end && !ex; ++k) {
                    const float4 sp = M.S[k];
                    float px, py, pz;
                    sphere_world(T, sp.x, sp.y, sp.z, px, py, pz);
                    const float sr = __fadd_rn(sp.w, margin);
                    if (kStats) st.v[ST_SPHERES] += 1;
                    ex = spheres_hit<1, kStats>(sc, ws.cand, ncand, &px, &py, &pz, &sr, g, st) ||
                         (esdf && sphere_esdf_any(sc, sv, px, py, pz, sr, nullptr, st));
                }
            }
            if (!esdf && ex) flagged = joint_gate<kStats, false>(M, sc, sv, jr, T, margin, ws, ncand, g, st);
            hit = ex && flagged;
        }
        if (__any_sync(kFull, hit && real)) break;   // warp-uniform early exit
    }
    if (kStats && real)
        for (int k = 0; k < ST_COUNT; ++k) st_out.v[k] += st.v[k];
    return __any_sync(kFull, hit && real);
}

}  // namespace
}  // namespace ps
