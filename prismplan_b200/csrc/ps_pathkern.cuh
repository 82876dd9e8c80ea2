// ps_pathkern.cuh -- one block checks a short path: every sample of an edge
// (small edge batches, ps_edges.cu) or the waypoints and densified segments of
// a slice of a trajectory (the optimisers, ps_optloop.cuh), scene and self
// collision, in one launch.
//
// A small batch is bound by latency and launches: the queue path runs one warp
// per 32 samples through serial candidate loops, once for the scene and once
// more, one thread per sample, for the self check, with a preparation, a
// second queue pass and a finalize around them. Here a block of 32 groups of 4
// lanes holds one path.
//   1. Swept check: the path is cut into intervals of samples, one per group.
//      From one kinematic pass at an interval's middle, with bounds on how far
//      links move inside it, an interval is shown clear of every box (and out
//      of reach of every ESDF layer) and of self collision, or not. Skipped
//      when the samples themselves fit the groups.
//   2. The samples of the other intervals are checked, a group each
//      (group_verdict, group_self_hit), if they are few; else their middles.
//   3. What is left goes on a list that all warps of the device work through
//      (rest_run), as the queue does: 32 samples a warp for the scene, 8 for
//      the self check. A block's own work is bounded by that: a path that
//      slides along a box has no interval that step 1 can clear, and a block
//      alone took 0.24 ms for 600 of its samples, 3.3 ms for 20,000 (the queue
//      40 us).
// The verdict is the OR over the samples' verdicts, and step 1 only leaves out
// samples that cannot hit, so the result is the queue path's.
#pragma once

#include <algorithm>
#include <cfloat>

#include "ps_chunk.cuh"
#include "ps_group.cuh"
#include "ps_internal.h"
#include "ps_verdict.cuh"

namespace ps {
namespace {

constexpr int kPathThreads = 128;
constexpr int kPathWarps = kPathThreads / 32;
constexpr int kPathSub = kSelfSub;                       // lanes per group
constexpr int kPathGroups = kPathThreads / kPathSub;     // intervals (or samples) at a time
constexpr float kSweepMaxQ = 16.0f;                      // largest joint value that the swept check judges

__device__ __forceinline__ float len_up(float x, float y, float z) {   // |(x, y, z)|, never below it
    const float d2 = fmaxf(fmaf(z, z, fmaf(y, y, x * x)), 1.0e-30f);
    return d2 * rsqrtf(d2) * (1.0f + 1.0e-6f);
}

// What a block of these kernels holds in shared memory.
struct PathSmem {
    ObbPrep* obbs;
    int* orig;
    LayerPrep* layers;
    float4* obs;
    float* q;        // [groups][2 D]: a group's configuration, and an interval's half width; [32 D] a warp over the list
    uint16_t* cand;  // over the list: a warp's candidate boxes
    SelfSmem self;   // positions of the groups' configurations
};

__host__ __device__ inline size_t path_tables(int n_obbs) {   // boxes, their indices, layers, spheres
    const size_t n = n_obbs > 1 ? n_obbs : 1;
    return n * sizeof(ObbPrep) + ((n + 3) & ~size_t(3)) * 4 + sizeof(LayerPrep) * PS_MAX_LAYERS + n * 16;
}

inline size_t path_self_bytes(const ps_model* m) {   // positions of the groups' configurations
    const int nc = m->dev.bound_from_apx ? 0 : m->info.n_joints;
    return (size_t)(m->info.n_spheres + m->info.n_approx_spheres + nc) * 3 * kPathGroups * 4;
}

inline size_t path_smem_bytes(const ps_model* m, const ps_scene_view* sv, bool self) {
    return (size_t)m->dev.bytes_core + path_tables(sv->n_obbs) + (size_t)kPathGroups * 2 * m->info.n_dof * 4 +
           (self ? path_self_bytes(m) : 0) + 64;
}

// The same for the kernels over the list: a tile of 32 configurations and the
// candidate boxes of each warp.
__host__ __device__ inline int rest_cand(int n_obbs) { return ((n_obbs > 1 ? n_obbs : 1) + 7) & ~7; }

inline size_t rest_smem_bytes(const ps_model* m, const ps_scene_view* sv, bool self) {
    return (size_t)m->dev.bytes_core + path_tables(sv->n_obbs) + (size_t)kPathThreads * m->info.n_dof * 4 +
           (size_t)kPathWarps * rest_cand(sv->n_obbs) * 2 + (self ? path_self_bytes(m) : 0) + 64;
}

// Models and calls these kernels serve; the rest takes the queue path. (A
// negative effective radius would be decided by the guard band's lower edge,
// which the two paths take from different bounds.)
inline bool path_serves(const ps_model* m, const ps_scene_view* sv, float margin, bool self) {
    return m->root_slot_only && m->info.approx_shares_chain && !sv->sphere_obb_acm_mask && !sv->sphere_acm_mask &&
           m->min_radius + margin >= 0.0f && path_smem_bytes(m, sv, self) <= smem_optin() / 2 &&
           rest_smem_bytes(m, sv, self) <= smem_optin() / 2;
}

// rest: the layout of rest_smem_bytes, else path_smem_bytes'.
__device__ __forceinline__ PathSmem path_carve(unsigned char* smem, const ModelDev& md, const ps_scene_view& sv,
                                               bool rest) {
    const BlobHeader* H = reinterpret_cast<const BlobHeader*>(md.blob);
    const int nob = max(sv.n_obbs, 1), D = H->n_dof;
    PathSmem s;
    s.obbs = reinterpret_cast<ObbPrep*>(smem + md.bytes_core);
    s.orig = reinterpret_cast<int*>(s.obbs + nob);
    s.layers = reinterpret_cast<LayerPrep*>(s.orig + ((nob + 3) & ~3));
    s.obs = reinterpret_cast<float4*>(s.layers + PS_MAX_LAYERS);
    s.q = reinterpret_cast<float*>(s.obs + nob);
    s.cand = reinterpret_cast<uint16_t*>(s.q + kPathThreads * D);
    unsigned char* end = rest ? reinterpret_cast<unsigned char*>(s.cand + kPathWarps * rest_cand(nob))
                              : reinterpret_cast<unsigned char*>(s.q + kPathGroups * 2 * D);
    s.self = carve_self<kPathGroups>(end, H->n_spheres, H->n_approx, H->n_joints, md.bound_from_apx != 0);
    return s;
}

// Swept check of the group's segment qm + s d, s in [-1, 1]: bit 0 set when a
// sphere may meet a box (or a layer's voxel box) somewhere on it, bit 1 when a
// self pair may overlap (with kSelf). Zero means that no sample of the segment
// can hit.
//
// One kinematic pass at the midpoint carries each joint frame's angular
// velocity w and origin velocity v per unit s, and bounds W >= |w|, A >= |w'|
// and Ao >= |v'| that hold on the whole segment, so a point at distance r from
// the joint's origin moves at most |v + w x r| + (Ao + |r| (W^2 + A)) / 2. A
// joint whose reach, widened by its centre's motion, meets no box is clear;
// otherwise its spheres, each widened by its own motion, are tested against
// the boxes met. The distance of two links changes only with the joints
// between them, by at most sum |d_k| lever(k, link) (ModelDev::lever). The
// guard band covers the rounding of the kinematics on either side (__sinf /
// __cosf included, for |q| <= kSweepMaxQ).
//
// Every lane of the warp calls it (ok: the group's segment may be judged);
// the result is the same on all lanes of a group.
template <bool kEsdf>
__device__ __forceinline__ unsigned path_sweep(const ModelSmem& M, const ModelDev& md, const SceneSmem& sc,
                                               const float4* __restrict__ obs, const float* qm, const float* dq,
                                               float margin, bool ok, bool self, const SelfSmem& sm, int slot) {
    constexpr int kSub = kPathSub;
    const int u = (threadIdx.x & 31) & (kSub - 1);
    const int NJ = M.H->n_joints;
    const float am = fabsf(margin), G4 = 4.0f * PS_GUARD_K;
    Affine T;
    affine_identity(T);
    float wx = 0.f, wy = 0.f, wz = 0.f, vx = 0.f, vy = 0.f, vz = 0.f, W = 0.f, A = 0.f, Ao = 0.f;
    bool clear = ok;
    for (int p = 0; p < NJ; ++p) {
        const JointRec& jr = M.J[p];
        if (p > 0) {
            const float qi = jr.dof >= 0 ? qm[jr.dof] : 0.0f;
            const float di = jr.dof >= 0 && jr.type != PS_FIXED ? dq[jr.dof] : 0.0f;
            float ox, oy, oz;   // the parent's origin
            if (jr.parent_slot == 0) {
                Affine I;
                affine_identity(I);
                joint_compose<true>(jr, qi, I, T);
                ox = oy = oz = wx = wy = wz = vx = vy = vz = W = A = Ao = 0.0f;
            } else {
                ox = T.m[3], oy = T.m[7], oz = T.m[11];
                joint_compose<true>(jr, qi, T, T);
            }
            const float ex = T.m[3] - ox, ey = T.m[7] - oy, ez = T.m[11] - oz;
            vx += wy * ez - wz * ey;
            vy += wz * ex - wx * ez;
            vz += wx * ey - wy * ex;
            const float ad = fabsf(di), el = len_up(ex, ey, ez) + ad;   // a sliding joint's offset grows by ad at most
            Ao += el * fmaf(W, W, A);
            const int ax = jr.type >= PS_X_ROT ? jr.type - PS_X_ROT : max(jr.type, 0);
            const float ux = T.m[ax] * di, uy = T.m[4 + ax] * di, uz = T.m[8 + ax] * di;
            if (jr.type >= PS_X_ROT) {
                wx += ux;
                wy += uy;
                wz += uz;
                A += ad * W;
                W += ad;
            } else {
                vx += ux;
                vy += uy;
                vz += uz;
                Ao += 2.0f * W * ad;
                if (jr.type >= PS_X_PRISM) ok = ok && fabsf(qi) + ad <= md.slide_max;   // the levers' range
            }
        }
        if (self) {
            for (int k = jr.sph_beg + u; k < jr.sph_end; k += kSub) {
                const float4 s = M.S[k];
                float px, py, pz;
                sphere_world(T, s.x, s.y, s.z, px, py, pz);
                put3(sm.pos, k, kPathGroups, slot, px, py, pz);
            }
            for (int k = jr.apx_beg + u; k < jr.apx_end && md.bound_from_apx; k += kSub) {
                const float4 s = M.A[k];
                float px, py, pz;
                sphere_world(T, s.x, s.y, s.z, px, py, pz);
                put3(sm.apos, k, kPathGroups, slot, px, py, pz);
            }
        }
        if (jr.reach < 0.0f) continue;   // uniform
        float cx, cy, cz;
        sphere_world(T, jr.bound.x, jr.bound.y, jr.bound.z, cx, cy, cz);
        if (self && u == 0 && !md.bound_from_apx) put3(sm.cpos, p, kPathGroups, slot, cx, cy, cz);
        if (sc.n_obbs == 0 && !kEsdf) continue;   // uniform
        const float WA = 0.5f * fmaf(W, W, A), hAo = 0.5f * Ao;
        // how far a point of this frame can move from its midpoint position
        auto motion = [&](float x, float y, float z) {
            const float rx = x - T.m[3], ry = y - T.m[7], rz = z - T.m[11];
            const float sp = len_up(vx + wy * rz - wz * ry, vy + wz * rx - wx * rz, vz + wx * ry - wy * rx);
            return (sp + hAo + len_up(rx, ry, rz) * WA) * 1.001f;   // a rigid transform's rounding
        };
        const float Sm = fmaxf(fabsf(cx), fmaxf(fabsf(cy), fabsf(cz)));
        const float R0 = jr.reach + am + motion(cx, cy, cz);
        const float gq = (Sm + R0 + sc.Bmax + 1.0f) * G4;
        const float Rc = R0 * (1.0f + G4) + gq;
        const float Rcl = Rc * sc.Mscale;
        float Rc2 = Rcl * Rcl;
        const float Rj = (Rc * (1.0f + G4) + G4 * (Sm + 1.0f)) * (1.0f + 1.0e-6f);
        bool near = kEsdf && esdf_reachable(sc, cx, cy, cz, Rc);
        LaneStats st;
#pragma unroll 1
        for (int base = 0; base < sc.n_obbs; base += 32) {
            const unsigned mask = reach_mask<kSub, false>(sc, obs, base, u, cx, cy, cz, Rj, Rc2, clear, [](float) {}, st);
            if (!mask) continue;
#pragma unroll 1
            for (int k = jr.sph_beg + u; k < jr.sph_end && !near; k += kSub) {
                const float4 s = M.S[k];
                float px, py, pz;
                sphere_world(T, s.x, s.y, s.z, px, py, pz);
                const float lim = (fabsf(s.w) + am + motion(px, py, pz) + gq) * sc.Mscale;
                const float lim2 = lim * lim;
#pragma unroll 1
                for (unsigned m = mask; m && !near; m &= m - 1) {
                    float qx, qy, qz;
                    near = !(fast_box_dsq(sc.obbs[base + __ffs(m) - 1], px, py, pz, qx, qy, qz) >= lim2);
                }
            }
        }
        const bool any_near = group_any<kSub>(near);   // every lane of the warp: the vote is warp-wide
        clear = clear && !any_near;
        if (!self && __all_sync(kGrpFull, !clear)) break;   // uniform
    }
    bool close = !ok;
    if (self) {   // uniform
        __syncwarp();   // the groups' positions are written
        auto at = [&](const float* a, int k, int c) { return a[(k * 3 + c) * kPathGroups + slot]; };
        auto bc = [&](int p, int c) { return md.bound_from_apx ? at(sm.apos, M.J[p].apx_beg, c) : at(sm.cpos, p, c); };
        // the group's lanes test 4 joint pairs at a time, then share the runs of
        // those that pass (the shuffles take the whole warp, so the loops over
        // pairs are uniform)
        for (int jp0 = 0; jp0 < md.n_sjp; jp0 += kSub) {
            bool pass = false;
            float wide = 0.0f;   // motion and guard
            if (jp0 + u < md.n_sjp) {
                const uint4 e = __ldg(md.sjp + jp0 + u);
                const int a = (int)(e.x & 0xffffu), qj = (int)(e.x >> 16);
                // how much the distance of a point of a and one of q can change
                float m = 0.0f;
                for (int x = qj, y = a; x != y;) {
                    const bool up = x > y;
                    const int k = up ? x : y;   // the later one in DFS order is not an ancestor of the other
                    const JointRec& jk = M.J[k];
                    if (jk.dof >= 0 && jk.type != PS_FIXED)
                        m = fmaf(fabsf(dq[jk.dof]), __ldg(md.lever + k * NJ + (up ? qj : a)), m);
                    if (up) x = jk.parent_pos;
                    else y = jk.parent_pos;
                }
                m *= 1.001f;
                const float ax = bc(a, 0), ay = bc(a, 1), az = bc(a, 2);
                const float qx = bc(qj, 0), qy = bc(qj, 1), qz = bc(qj, 2);
                const float dx = ax - qx, dy = ay - qy, dz = az - qz;
                const float S = fmaxf(fmaxf(fabsf(ax), fmaxf(fabsf(ay), fabsf(az))),
                                      fmaxf(fabsf(qx), fmaxf(fabsf(qy), fabsf(qz))));
                const float R = M.J[a].reach + M.J[qj].reach;
                wide = m + 4.0f * (S + R + m + 1.0f) * PS_GUARD_K;
                const float lim = R + wide;
                pass = !(fmaf(dz, dz, fmaf(dy, dy, dx * dx)) >= lim * lim);
            }
            const unsigned bal = group_bits<kSub>(__ballot_sync(kGrpFull, pass));
            for (int v = 0; v < kSub && jp0 + v < md.n_sjp; ++v) {
                const float wv = __shfl_sync(kGrpFull, wide, (threadIdx.x & 31 & ~(kSub - 1)) + v);
                if (close || !((bal >> v) & 1u)) continue;   // no warp-wide call below
                const uint4 e = __ldg(md.sjp + jp0 + v);
                const int qj = (int)(e.x >> 16);
                const float qx = bc(qj, 0), qy = bc(qj, 1), qz = bc(qj, 2), Rq = M.J[qj].reach;
                for (int r = (int)e.y + u; r < (int)e.z && !close; r += kSub) {
                    const uint2 run = __ldg(md.sruns + r);
                    const int i = run.x & 0x1ff, len = run.x >> 14;
                    const float px = at(sm.pos, i, 0), py = at(sm.pos, i, 1), pz = at(sm.pos, i, 2);
                    const float ri = fabsf(M.S[i].w) + wv;
                    const float ex = px - qx, ey = py - qy, ez = pz - qz;
                    const float lim = ri + Rq;
                    if (fmaf(ez, ez, fmaf(ey, ey, ex * ex)) >= lim * lim) continue;
                    bool any = false;   // no branch in the loop: its loads go out together
#pragma unroll 4
                    for (int k = 0; k < len; ++k) {
                        const int j = (int)run.y + k;
                        const float fx = px - at(sm.pos, j, 0), fy = py - at(sm.pos, j, 1), fz = pz - at(sm.pos, j, 2);
                        const float lj = ri + fabsf(M.S[j].w);
                        any |= !(fmaf(fz, fz, fmaf(fy, fy, fx * fx)) >= lj * lj);
                    }
                    close = any;
                }
            }
        }
        const bool any_close = group_any<kSub>(close);   // every lane of the warp
        close = any_close;
        __syncwarp();   // the positions' readers are done
    }
    return (clear ? 0u : 1u) | (self && close ? 2u : 0u);
}

// An interval of a segment's samples, lo .. hi, and what to check it for
// (path_sweep's bits).
struct PathItem {
    int seg, lo, hi, what;
};
constexpr int kPathQuarter = 16;             // most intervals that a block starts over with in quarters
constexpr int kPathMost = 4 * kPathQuarter;  // intervals of a pass (33 on the first one)
struct PathBlock {
    int hit;              // a sample collides
    int n_list;           // intervals that the swept check left
    int n_samples;        // samples they hold (saturated)
    unsigned left[2];     // units of the path that go on the list: scene, self (path_left)
    PathItem item[kPathMost], list[kPathMost];
};

// Works through the n intervals blk.item: the swept check (skipped for single
// samples), then for the intervals that it leaves every sample if they are
// few, else one of each (the first one when `ends`, else the middle one). With
// no hit among those, half of them or fewer start over in quarters, `again` times
// at most (an edge near something on a part of its way: 400 edges without self
// check 273 -> 199 us among 128 boxes, where nothing is left after one more
// pass; with it a pass more costs an edge batch 4 to 10 %, as the list's warps
// share the pairs better), and else they go to defer(), a thread each. Stops
// early once a sample hits or stop() says that the answer no longer matters.
//
// point(seg, i, a, b): DoF i of a segment's ends; sample j is a + (j / G)
// (b - a), rounded as the edge kernels round it, and j = G + 1 is b itself
// (with `ends` j = 0 is a itself, also where b - a is not finite).
// Every thread of the block calls it after a block barrier; blk.hit and what
// defer() wrote are there after the barrier inside.
template <bool kEsdf, class Point, class Stop, class Defer>
__device__ __forceinline__ void path_run(const ModelSmem& M, const ModelDev& md, const SceneSmem& sc,
                                         const ps_scene_view& sv, const PathSmem& ps, float margin, bool self,
                                         PathBlock& blk, int n, int G, bool ends, int again, Point&& point, Stop&& stop,
                                         Defer&& defer) {
    constexpr int kSub = kPathSub;
    const int D = M.H->n_dof;
    const int lane = threadIdx.x & 31, slot = threadIdx.x / kSub, u = lane & (kSub - 1);
    const int first = (threadIdx.x & ~31) / kSub;   // the warp's first group
    float* qc = ps.q + slot * 2 * D;
    float* dq = qc + D;
    volatile int* hit_flag = &blk.hit;
    LaneStats st;
    st.zero();
    for (;; --again) {
        if (threadIdx.x == 0) blk.n_list = blk.n_samples = 0;
        __syncthreads();
        // ---- swept check, a group per interval ----
        for (int k0 = 0; k0 < n; k0 += kPathGroups) {
            const PathItem it = blk.item[min(k0 + slot, n - 1)];   // a group past the end repeats the last one
            const bool single = it.lo == it.hi;
            unsigned bits = (unsigned)it.what;
            if (!__all_sync(kGrpFull, single)) {   // uniform
                const int lo = min(it.lo, G), hi = min(it.hi, G);
                const float tm = __fdiv_rn((float)lo + (float)hi, 2.0f * (float)G),
                            th = __fdiv_rn((float)hi - (float)lo, 2.0f * (float)G);
                bool ok = !single;   // a single sample is checked itself
                __syncwarp();
                for (int i = 0; i < D; ++i) {
                    float a, b;
                    point(it.seg, i, a, b);
                    ok = ok && fabsf(a) <= kSweepMaxQ && fabsf(b) <= kSweepMaxQ;
                    if ((i & (kSub - 1)) == u) {
                        qc[i] = fmaf(tm, b - a, a);
                        dq[i] = th * (b - a);
                    }
                }
                __syncwarp();
                bits &= path_sweep<kEsdf>(M, md, sc, ps.obs, qc, dq, margin, ok, self, ps.self, slot);
            }
            if (u == 0 && k0 + slot < n && bits) {   // in any order
                const int k = atomicAdd(&blk.n_list, 1);
                blk.list[k] = PathItem{it.seg, it.lo, it.hi, (int)bits};
                atomicAdd(&blk.n_samples, min(it.hi - it.lo + 1, 1 << 20));
            }
        }
        __syncthreads();
        const int nl = blk.n_list;
        const bool all = blk.n_samples <= 2 * kPathGroups;
        // samples of an interval that are checked now: all, or one and sample G + 1 (defer() takes no more than G)
        auto count = [&](const PathItem& x) { return all ? x.hi - x.lo + 1 : (x.lo <= G && x.hi > G ? 2 : 1); };
        int per = 0;
        for (int k = 0; k < nl; ++k) per = max(per, count(blk.list[k]));
        // ---- samples: task t is sample t / nl of interval t % nl, so that every
        //      interval is looked at before any is finished ----
        const int total = per * nl;
        for (int t0 = first; t0 < total; t0 += kPathGroups) {
            if (__any_sync(kGrpFull, *hit_flag != 0 || stop())) break;   // one decision for the warp
            const int t = min(t0 + (slot - first), total - 1);
            const PathItem x = blk.list[t % nl];
            const int s = t / nl, cnt = x.hi - x.lo + 1;
            const bool on = t0 + (slot - first) < total && s < count(x);
            if (!__any_sync(kGrpFull, on)) continue;   // uniform
            const int j = s == 1 && !all ? x.hi : x.lo + (ends ? s : (s + cnt / 2) % cnt);   // from the middle on
            const float tj = __fdiv_rn((float)j, (float)G);
            __syncwarp();
            for (int i = u; i < D; i += kSub) {
                float a, b;
                point(x.seg, i, a, b);
                qc[i] = j > G ? b : (ends && j == 0 ? a : __fmaf_rn(tj, __fadd_rn(b, -a), a));
            }
            __syncwarp();
            bool hit = false;
            if (__any_sync(kGrpFull, on && (x.what & 1))) {   // uniform
                bool h;
                float clr;
                group_verdict<kSub, false, kEsdf, false>(M, sc, sv, ps.obs, qc, margin, false, h, clr, st);
                hit = on && (x.what & 1) && h;
            }
            if (self && on && (x.what & 2) && !hit)   // uniform over the group
                hit = group_self_hit<kPathGroups>(M, md, qc, ps.self, slot, u, st);
            if (hit && u == 0) *hit_flag = 1;
            __syncwarp();
        }
        if (__syncthreads_or(*hit_flag != 0 || stop()) || all) break;   // one decision for the block
        const bool quarter = again > 0 && nl <= kPathQuarter;
        if (threadIdx.x < nl) {
            PathItem x = blk.list[threadIdx.x];
            x.hi = max(min(x.hi, G), x.lo);
            const int cnt = x.hi - x.lo + 1;
            if (!quarter && cnt > 1) defer(x);
            for (int k = 0; k < 4 && quarter; ++k) {   // an empty quarter, and a sample by itself, which is done: nothing
                const int lo = x.lo + (int)((long long)cnt * k / 4), hi = x.lo + (int)((long long)cnt * (k + 1) / 4) - 1;
                blk.item[4 * threadIdx.x + k] = PathItem{x.seg, lo, max(lo, hi), lo <= hi && cnt > 1 ? x.what : 0};
            }
        }
        if (!quarter) break;
        n = 4 * nl;
        __syncthreads();
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// The list: paths whose samples are left, and which
// ---------------------------------------------------------------------------
// A path's samples 1 .. G in up to 32 units of rest_unit(G) samples, a whole
// number of warps' worth; bit u of `scene` / `self`: unit u is to be checked.
struct RestItem {
    int row, G;   // the path's ends are rows `row` of from and to
    unsigned scene, self;
};
constexpr int kRestSelf = 32 / kSelfSub;   // samples a warp checks for self collision at a time

__device__ __forceinline__ int rest_unit(int G) { return 32 * ((G - 1) / 1024 + 1); }

// The units that samples lo .. hi lie in.
__device__ __forceinline__ unsigned rest_bits(int lo, int hi, int G) {
    const int unit = rest_unit(G);
    return (0xffffffffu >> (31 - (min(hi, G) - 1) / unit)) & (0xffffffffu << ((max(lo, 1) - 1) / unit));
}

// Marks an interval's units in blk.left (the start configuration, sample 0,
// goes with the last one: rest_run checks it behind sample G).
__device__ __forceinline__ void path_left(PathBlock& blk, const PathItem& x, int G) {
    const unsigned bits = rest_bits(x.lo, x.hi, G) | (x.lo == 0 ? rest_bits(G, G, G) : 0u);
    if (x.what & 1) atomicOr(&blk.left[0], bits);
    if (x.what & 2) atomicOr(&blk.left[1], bits);
}

// Blocks that work through a list: all that fit at once.
template <class K>
inline int rest_grid(K k, size_t smem, int& grid) {
    PS_TRY_CUDA(allow_smem((const void*)k, smem));
    int per_sm = 0;
    PS_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kPathThreads, smem));
    grid = sm_count() * std::max(per_sm, 1);
    return PS_OK;
}

// Checks what n paths have left, get(k) the k-th of them (unit: the longest
// rest_unit among them): every warp of the grid takes 32 samples for the scene
// or 8 for the self check at a time, consecutive ones on consecutive blocks.
// known(row): the path is known to collide; report(row): a sample of it does.
template <bool kEsdf, class Get, class Known, class Report>
__device__ __forceinline__ void rest_run(const ModelSmem& M, const ModelDev& md, const SceneSmem& sc,
                                         const ps_scene_view& sv, const PathSmem& ps, float margin, bool self,
                                         const float* __restrict__ from, const float* __restrict__ to, int n, int unit,
                                         Get&& get, Known&& known, Report&& report) {
    const int D = M.H->n_dof;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, u = lane & (kSelfSub - 1);
    const WarpScratch ws{ps.q + warp * 32 * D, ps.cand + warp * rest_cand(sv.n_obbs), ps.obs};
    LaneStats st;
    st.zero();
    const int per_scene = unit / 32, per_self = self ? unit / kRestSelf : 0;   // tasks a unit
    const long long scene = 32ll * n * per_scene, total = scene + 32ll * n * per_self;
    const long long warps = (long long)gridDim.x * kPathWarps, me = (long long)warp * gridDim.x + blockIdx.x;
    for (long long base = me; base < total; base += 32 * warps) {
        const long long v = base + lane * warps;   // the lanes look at 32 tasks of this warp
        RestItem x{};
        int j0 = 0;
        bool live = false;
        if (v < total) {
            // task w is part k of unit b of path w % n: the paths' first units
            // first, which most have, so that the warps share them evenly
            const long long w = v < scene ? v : v - scene, r = w / n;
            x = get((int)(w - r * n));
            const int un = rest_unit(x.G), b = (int)(r & 31), k = (int)(r >> 5) * (v < scene ? 32 : kRestSelf);
            j0 = b * un + k;
            // the start configuration (see process_chunk) follows the last sample
            const int last = x.G + (v >= scene && x.G % 16 != 0 ? 1 : 0);
            live = k < un && j0 < last && (((v < scene ? x.scene : x.self) >> b) & 1u);
        }
        for (unsigned todo = __ballot_sync(kFull, live); todo; todo &= todo - 1) {
            const int src = __ffs(todo) - 1;
            const int row = __shfl_sync(kFull, x.row, src), G = __shfl_sync(kFull, x.G, src),
                      j = __shfl_sync(kFull, j0, src);
            if (__any_sync(kFull, known(row))) continue;   // one decision for the warp
            bool hit;
            if (base + src * warps < scene) {   // uniform
                hit = process_chunk_fast<false, kEsdf>(M, sc, sv, margin, from, to, row, G, j, ws, st);
            } else {
                const int raw = j + 1 + lane / kSelfSub;   // past the end: the last one
                const float t = __fdiv_rn((float)(raw == G + 1 && G % 16 != 0 ? 0 : min(raw, G)), (float)G);
                float* qc = ws.q + (lane / kSelfSub) * D;
                for (int i = u; i < D; i += kSelfSub) {
                    const float a = __ldg(from + (size_t)row * D + i), b = __ldg(to + (size_t)row * D + i);
                    qc[i] = __fmaf_rn(t, __fadd_rn(b, -a), a);
                }
                __syncwarp();
                hit = __any_sync(kFull, group_self_hit<kPathGroups>(M, md, qc, ps.self, threadIdx.x / kSelfSub, u, st));
            }
            if (hit && lane == 0) report(row);
            __syncwarp();
        }
    }
}

// Stages the model and the scene. False: the staging gave up (uniform).
__device__ __forceinline__ bool path_stage(const ModelDev& md, const ps_scene_view& sv, unsigned char* smem,
                                           uint64_t* mbar, int* counters, float* bmax, bool self, bool rest, PathSmem& ps,
                                           SceneSmem& sc) {
    if (!stage_model(md, smem, mbar)) return false;
    if (self) warm_self_tables<true>(md, reinterpret_cast<const BlobHeader*>(smem)->n_joints);
    ps = path_carve(smem, md, sv, rest);
    stage_scene(sv, ps.obbs, ps.orig, ps.layers, counters, bmax, sc);
    box_spheres(sc, ps.obs);
    __syncthreads();
    box_limits(sc, ps.obs);
    __syncthreads();
    return true;
}

// Sample count of an edge (edge_eval.cuh:54-60 plus the L-inf rule).
__device__ __forceinline__ int edge_samples(const ps_edge_params& P, const int* given, int e, const float* a,
                                            const float* b, int D, float len) {
    if (given) return given[e];
    if (P.resolution > 0.0f) {
        int g = (int)ceilf(__fdiv_rn(len, P.resolution));
        return min(max(g, 2), 1024);
    }
    if (P.max_joint_step > 0.0f) {
        float m = 0.0f;
        for (int i = 0; i < D; ++i) m = fmaxf(m, fabsf(__fadd_rn(b[i], -a[i])));
        int g = (int)ceilf(__fdiv_rn(m, P.max_joint_step));
        const int cap = P.max_samples > 0 ? P.max_samples : 1024;
        return min(max(g, 1), cap);
    }
    return P.granularity;
}

__device__ __forceinline__ float edge_length(const float* a, const float* b, int D) {
    float len2 = 0.0f;   // edge_eval.cuh:104-106
    for (int i = 0; i < D; ++i) {
        float d = __fadd_rn(b[i], -a[i]);
        len2 = __fmaf_rn(d, d, len2);
    }
    return sqrtf(len2);
}

}  // namespace
}  // namespace ps
