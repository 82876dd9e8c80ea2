// ps_group.cuh -- verdict and clearance of configurations, kSub consecutive
// lanes of a warp per configuration (kSub a power of two, 1 to 32).
//
// Same decisions and clearance as the generic kernel (check_configs_kernel):
// the two-phase verdict of two_phase_cc.cuh:57-138 and the min over spheres
// and boxes of sdf - (r + margin). It serves models whose root is the only
// slot-0 frame (one 3x4 frame in registers) and whose approximate chain is
// the full chain, without ACM masks.
//
// What bounds these checks is the sphere-box pairs, and most of them cannot
// matter: per joint, the boxes beyond the reach of the joint's spheres (their
// bound centre c and JointRec::reach) hit nothing, and, for the clearance, a
// box farther from c than reach + the smallest clearance found so far cannot
// lower it. So each joint first tests the boxes against c (circumscribed
// sphere, then box distance; a group's lanes split the boxes), 32 at a time
// into a bit mask, and only the boxes of the mask meet the joint's spheres (a
// group's lanes split the spheres). Every test keeps a superset (guard band
// and map stretch as in the edge kernels), each kept pair is computed as
// before, and minimum and OR do not depend on the order: same bits.
//
// Measured on 1,048,576 configurations (7 joints, 59 spheres, 16 boxes, with
// clearance): 1.09 ms with every pair computed, 0.56 ms; 20,011 verdicts of a
// 14-joint robot among 128 boxes and an ESDF: 419 us, 118 us (4 lanes each).
// What bounds it now is the issue rate (62 to 68 % of the issue slots, 20 of
// 32 lanes: a warp runs each joint's loops to its busiest lane's count).
//
// The approximate gate runs only where an exact sphere hits (the verdict is
// gate && exact) or, with ESDF layers, where the joint reaches a voxel box.
#pragma once

#include "ps_internal.h"
#include "ps_verdict.cuh"

namespace ps {
namespace {

constexpr unsigned kGrpFull = 0xffffffffu;

template <int kV>
struct IntC {
    static constexpr int value = kV;
};

// The group's bits of a warp ballot, lane u of the group in bit u.
template <int kSub>
__device__ __forceinline__ unsigned group_bits(unsigned bal) {
    if (kSub == 32) return bal;
    return (bal >> ((threadIdx.x & 31) & ~(kSub - 1))) & ((1u << (kSub & 31)) - 1u);
}

// OR / minimum over the group (every lane of the warp calls them).
template <int kSub>
__device__ __forceinline__ bool group_any(bool v) {
    return kSub == 1 ? v : group_bits<kSub>(__ballot_sync(kGrpFull, v)) != 0;
}
template <int kSub>
__device__ __forceinline__ float group_min(float v) {
#pragma unroll
    for (int o = 1; o < kSub; o <<= 1) v = fminf(v, __shfl_xor_sync(kGrpFull, v, o));
    return v;
}

// Exact re-decision of a sphere over the mask's boxes inside the guard band.
__device__ __noinline__ bool mask_redecide(const SceneSmem& sc, int base, unsigned mask, float px, float py, float pz,
                                           float sr, float lo, float hi, LaneStats& st) {
    while (mask) {
        const ObbPrep& o = sc.obbs[base + __ffs(mask) - 1];
        mask &= mask - 1;
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

// The most negative max(q) over the mask's boxes that contain the point.
__device__ __noinline__ float mask_inside(const SceneSmem& sc, int base, unsigned mask, float px, float py, float pz) {
    float inside = 0.0f;
    while (mask) {
        const ObbPrep& o = sc.obbs[base + __ffs(mask) - 1];
        mask &= mask - 1;
        float qx, qy, qz;
        if (fast_box_dsq(o, px, py, pz, qx, qy, qz) == 0.0f) inside = fminf(inside, fmaxf(qx, fmaxf(qy, qz)));
    }
    return inside;
}

// This lane's share of a joint's approximate gate against the boxes (boxes u,
// u + kSub, ...): whether any approximate sphere hits one of them.
template <int kSub>
__device__ __noinline__ bool lane_gate_boxes(const ModelSmem& M, const SceneSmem& sc, const JointRec& jr,
                                             const Affine& T, float margin, int u, LaneStats& st) {
    for (int a = jr.apx_beg; a < jr.apx_end; ++a) {
        const float4 sa = M.A[a];
        float px, py, pz;
        sphere_world(T, sa.x, sa.y, sa.z, px, py, pz);
        const float sr = __fadd_rn(sa.w, margin);
        float lo, hi;
        guard_thresholds(px, py, pz, sr, sc.Bmax, lo, hi);
        for (int o = u; o < sc.n_obbs; o += kSub) {
            float qx, qy, qz;
            const float d = fast_box_dsq(sc.obbs[o], px, py, pz, qx, qy, qz);
            if (d < lo) return true;
            if (d < hi && ref_obb_hit(sc.obbs[o], px, py, pz, sr)) return true;
        }
    }
    return false;
}

// OR over the group (every lane of the warp calls it).
template <int kSub>
__device__ __forceinline__ unsigned group_or(unsigned v) {
#pragma unroll
    for (int o = 1; o < kSub; o <<= 1) v |= __shfl_xor_sync(kGrpFull, v, o);
    return v;
}

// Boxes base .. base + 31 within reach of the joint: Rj the joint part of the
// circumscribed-sphere limit (box_limits), Rc2 the squared box-frame radius.
// Lane u of the group tests boxes base + u, + kSub, ..., the circumscribed
// spheres 4 at a time (independent, so they overlap), the box distance of
// those that pass. near (kClr): the box distances also bound the clearance
// from above (near() lowers Rc2 as they come). Returns the group's mask. The
// tests are written so that a NaN centre culls nothing.
template <int kSub, bool kStats, class Near>
__device__ __forceinline__ unsigned reach_mask(const SceneSmem& sc, const float4* __restrict__ obs, int base, int u,
                                               float cx, float cy, float cz, float Rj, float& Rc2, bool on,
                                               Near&& near, LaneStats& st) {
    const int n = min(32, sc.n_obbs - base);
    unsigned mask = 0;
    if (on) {
        constexpr int kStep = 4 * kSub < 32 ? 4 * kSub : 32;
        unsigned pass = 0;
#pragma unroll 1
        for (int i = u; i < n; i += kStep) {
#pragma unroll
            for (int k = 0; k < kStep; k += kSub) {
                const float4 ob = obs[base + min(i + k, n - 1)];
                const float ex = ob.x - cx, ey = ob.y - cy, ez = ob.z - cz;
                const float lim = Rj + ob.w;
                if (!(fmaf(ez, ez, fmaf(ey, ey, ex * ex)) >= lim * lim) && i + k < n) pass |= 1u << (i + k);
            }
        }
        if (kStats) st.v[ST_CULL] += (n + kSub - 1 - u) / kSub;
        while (pass) {
            const int k = __ffs(pass) - 1;
            pass &= pass - 1;
            float qx, qy, qz;
            const float d = fast_box_dsq(sc.obbs[base + k], cx, cy, cz, qx, qy, qz);
            if (!(d >= Rc2)) {
                mask |= 1u << k;
                near(d);
            }
        }
    }
    return group_or<kSub>(mask);
}

// Verdict (and, with kClr, the box clearance) of the group's configuration
// qc. Every lane of the warp calls it; the result is the same on all lanes of
// a group. kEsdf: the scene has ESDF layers (verdict only).
template <int kSub, bool kClr, bool kEsdf, bool kStats>
__device__ __forceinline__ void group_verdict(const ModelSmem& M, const SceneSmem& sc, const ps_scene_view& sv,
                                              const float4* __restrict__ obs, const float* qc, float margin,
                                              bool no_gate, bool& hit_out, float& clr_out, LaneStats& st) {
    static_assert(!(kClr && kEsdf), "the clearance variant serves boxes only");
    // spheres a lane holds at once: 4 per box load where a lane has all of a
    // joint's spheres, fewer where the group's lanes share them
    constexpr int kG = kSub == 1 ? 4 : (kSub <= 4 ? 2 : 1);
    const int u = (threadIdx.x & 31) & (kSub - 1);
    const int NJ = M.H->n_joints;
    const float am = fabsf(margin);
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
            if (kStats && u == 0) st.v[ST_JOINTS] += 1;
        }
        if (jr.reach < 0.0f || (sc.n_obbs == 0 && !kEsdf)) continue;   // nothing to test (uniform)
        float cx, cy, cz;
        sphere_world(T, jr.bound.x, jr.bound.y, jr.bound.z, cx, cy, cz);
        const float Sm = fmaxf(fabsf(cx), fmaxf(fabsf(cy), fabsf(cz)));
        const float G4 = 4.0f * PS_GUARD_K;
        const float R0 = jr.reach + am;
        const float gq = (Sm + sc.Bmax + 1.0f) * G4;
        // cull radius for a pair that may come within `slack` of contact
        auto radius = [&](float slack) { return (R0 + slack) * (1.0f + G4) + gq; };
        float slack = kClr ? fmaxf(clr, 0.0f) : 0.0f;
        float Rc = radius(slack);
        float Rcl = Rc * sc.Mscale, Rc2 = Rcl * Rcl;
        // a box at squared distance d2 from c (or nearer) bounds the clearance from above:
        // some sphere of the joint has clearance <= d + stretch * near_d - r - margin
        auto near = [&](float d2) {
            if (!kClr) return;
            const float d2c = fmaxf(d2, 1.0e-30f);
            const float ub = d2c * rsqrtf(d2c) * (1.0f + 1.0e-6f) + jr.near_r + (sc.Mscale - 1.0f) * jr.near_d -
                             margin + gq;
            if (ub < slack) {
                slack = fmaxf(ub, 0.0f);
                Rcl = radius(slack) * sc.Mscale;
                Rc2 = Rcl * Rcl;
            }
        };
        if (kClr && (kSub > 1 ? __any_sync(kGrpFull, slack > 2.0f) : slack > 2.0f)) {
            // no clearance known yet (on some group of the warp: the minimum
            // below is warp-wide): the nearest box centre bounds it, so that the
            // first joint does not take every box
            float dc = 3.0e38f;
            for (int o = u; o < sc.n_obbs; o += kSub) {
                const float4 ob = obs[o];
                const float ex = ob.x - cx, ey = ob.y - cy, ez = ob.z - cz;
                if (ob.w < 1.0e29f) dc = fminf(dc, fmaf(ez, ez, fmaf(ey, ey, ex * ex)));   // a known centre
            }
            near(group_min<kSub>(dc) * sc.Mscale * sc.Mscale);
            Rc = radius(slack);
        }
        const float Rj = (Rc * (1.0f + G4) + G4 * (Sm + 1.0f)) * (1.0f + 1.0e-6f);
        const float g = (Sm + jr.reach + sc.Bmax + 1.0f) * PS_GUARD_K;
        // ESDF layers within reach (the same on every lane of a group)
        const bool reach = kEsdf && !hit && esdf_reachable(sc, cx, cy, cz, Rc);
        bool ex = false;         // this lane saw an exact sphere hit a box
        bool gate_box = false;   // this lane saw an approximate sphere hit a box (asked for with a layer in reach)
        // kN spheres k, k + kSub, ... of this lane against the mask's boxes
        auto spheres = [&](auto kN_, int k, int base, unsigned mask) {
            constexpr int kN = decltype(kN_)::value;
            float px[kN], py[kN], pz[kN], sr[kN], mn[kN];
#pragma unroll
            for (int i = 0; i < kN; ++i) {
                const float4 sp = M.S[k + kSub * i];
                sphere_world(T, sp.x, sp.y, sp.z, px[i], py[i], pz[i]);
                sr[i] = __fadd_rn(sp.w, margin);
                mn[i] = 3.0e38f;
            }
            if (kStats) {
                st.v[ST_SPHERES] += kN;
                st.v[ST_PAIRS] += kN * __popc(mask);
            }
#pragma unroll 1
            for (unsigned m = mask; m; m &= m - 1) {
                const ObbPrep& o = sc.obbs[base + __ffs(m) - 1];
                const float4 r0 = o.r0, r1 = o.r1, r2 = o.r2, h = o.h;
#pragma unroll
                for (int i = 0; i < kN; ++i) {
                    const float lx = fmaf(r0.z, pz[i], fmaf(r0.y, py[i], fmaf(r0.x, px[i], r0.w)));
                    const float ly = fmaf(r1.z, pz[i], fmaf(r1.y, py[i], fmaf(r1.x, px[i], r1.w)));
                    const float lz = fmaf(r2.z, pz[i], fmaf(r2.y, py[i], fmaf(r2.x, px[i], r2.w)));
                    const float bx = fmaxf(fabsf(lx) - h.x, 0.0f), by = fmaxf(fabsf(ly) - h.y, 0.0f),
                                bz = fmaxf(fabsf(lz) - h.z, 0.0f);
                    mn[i] = fminf(mn[i], fmaf(bz, bz, fmaf(by, by, bx * bx)));
                }
            }
#pragma unroll
            for (int i = 0; i < kN; ++i) {
                if (kClr) {
                    // the root is taken only where it can lower the minimum (16 ulps of slack)
                    const float lim = clr + sr[i] + 2.0e-6f * (fabsf(clr) + fabsf(sr[i]));
                    if (mn[i] == 0.0f || (lim > 0.0f && mn[i] < lim * lim)) {
                        const float sdf =
                            mn[i] > 0.0f ? sqrtf(mn[i]) : mask_inside(sc, base, mask, px[i], py[i], pz[i]);
                        clr = fminf(clr, __fadd_rn(sdf, -sr[i]));
                    }
                }
                const float b = fabsf(sr[i]) + g;   // no box of the mask at or beyond it can be hit
                if (!hit && !ex && mn[i] < b * b * (1.0f + 1.0e-6f)) {
                    float lo, hi;
                    guard_thresholds(px[i], py[i], pz[i], sr[i], sc.Bmax, lo, hi);
                    ex = mn[i] < lo ||
                         (mn[i] < hi && mask_redecide(sc, base, mask, px[i], py[i], pz[i], sr[i], lo, hi, st));
                }
            }
        };
#pragma unroll 1
        for (int base = 0; base < sc.n_obbs; base += 32) {
            const float was = Rc2;
            unsigned mask = reach_mask<kSub, kStats>(sc, obs, base, u, cx, cy, cz, Rj, Rc2, kClr || !hit, near, st);
            if (kClr && kSub == 1 && Rc2 < was && (mask & (mask - 1))) {
                // the radius shrank on the way: drop the boxes taken before it did
                unsigned m = mask;
                mask = 0;
                for (; m; m &= m - 1) {
                    float qx, qy, qz;
                    const float d = fast_box_dsq(sc.obbs[base + __ffs(m) - 1], cx, cy, cz, qx, qy, qz);
                    if (!(d >= Rc2)) mask |= m & (0u - m);
                }
            }
            if (!mask) continue;
            int k = jr.sph_beg + u;
#pragma unroll 1
            for (; k + (kG - 1) * kSub < jr.sph_end && (kClr || !ex); k += kSub * kG) spheres(IntC<kG>{}, k, base, mask);
            if (kG > 1)
#pragma unroll 1
                for (; k < jr.sph_end && (kClr || !ex); k += kSub) spheres(IntC<1>{}, k, base, mask);
            if (kEsdf && reach && !gate_box) {
                // the approximate gate against these boxes, split over the group's lanes
                for (int a = jr.apx_beg; a < jr.apx_end && !gate_box; ++a) {
                    const float4 sa = M.A[a];
                    float px, py, pz;
                    sphere_world(T, sa.x, sa.y, sa.z, px, py, pz);
                    const float sr = __fadd_rn(sa.w, margin);
                    unsigned mine = 0;
                    int i = 0;
                    for (unsigned m = mask; m; m &= m - 1, ++i)
                        if ((i & (kSub - 1)) == u) mine |= m & (0u - m);
                    float lo, hi;
                    guard_thresholds(px, py, pz, sr, sc.Bmax, lo, hi);
                    gate_box = mask_redecide(sc, base, mine, px, py, pz, sr, lo, hi, st);
                }
            }
        }
        const bool exg = group_any<kSub>(ex);
        const bool ask = !hit && (exg || reach);
        if (kSub > 1 ? __any_sync(kGrpFull, ask) : ask) {
            bool fl = false;
            if (ask) {
                fl = no_gate || gate_box;
                if (reach)
                    for (int a = jr.apx_beg; a < jr.apx_end && !fl; ++a) {
                        const float4 sa = M.A[a];
                        float px, py, pz;
                        sphere_world(T, sa.x, sa.y, sa.z, px, py, pz);
                        fl = sphere_esdf_any(sc, sv, px, py, pz, __fadd_rn(sa.w, margin), nullptr, st);
                    }
                if (!fl && !reach) fl = lane_gate_boxes<kSub>(M, sc, jr, T, margin, u, st);
            }
            const bool flagged = group_any<kSub>(fl);
            if (kEsdf) {
                bool exe = false;
                if (reach && flagged && !exg)
                    for (int k = jr.sph_beg + u; k < jr.sph_end && !exe; k += kSub) {
                        const float4 sp = M.S[k];
                        float px, py, pz;
                        sphere_world(T, sp.x, sp.y, sp.z, px, py, pz);
                        if (kStats) st.v[ST_SPHERES] += 1;
                        exe = sphere_esdf_any(sc, sv, px, py, pz, __fadd_rn(sp.w, margin), nullptr, st);
                    }
                const bool any_esdf = group_any<kSub>(exe);   // every lane of the warp: the vote is warp-wide
                hit = hit || (flagged && (exg || any_esdf));
            } else {
                hit = hit || (flagged && exg);
            }
        }
        if (kClr) clr = group_min<kSub>(clr);
        else if (__all_sync(kGrpFull, hit)) break;   // uniform
    }
    hit_out = hit;
    clr_out = clr;
}

// Lanes per configuration. Few configurations leave the chip idle one lane
// each, and a configuration's chain of joints is serial, so its boxes and
// spheres are split over 16 lanes while that makes at most 16 warps per SM,
// over 4 while that makes at most 28; beyond, the split's repeated kinematics
// cost more than the latency it hides. Measured (us, 1 / 4 / 16 lanes; 7
// joints, 59 spheres, 16 boxes with clearance): 1024 configurations 35.2 /
// 17.9 / 12.3, 4096 38.0 / 18.0 / 15.7, 8192 37.8 / 19.6 / 28.2, 32,768 41.1 /
// 40.5 / 83.9, 131,072 92.7 / 132 / 302; the verdict on 14 joints, 128 boxes
// and an ESDF crosses at the same counts.
inline int config_lanes(int n) {
    const long long per_warp = 32ll * sm_count();
    if ((long long)n * 16 <= 16 * per_warp) return 16;
    return (long long)n * 4 <= 28 * per_warp ? 4 : 1;
}

}  // namespace
}  // namespace ps
