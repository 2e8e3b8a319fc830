/*
 * orca_group.cuh -- the per-agent step (ORCA::GetVelocity and the
 * integration) with G lanes per agent, 32 / G agents per warp.
 *
 * The lanes of a group build the agent's obstacle and neighbour half-planes
 * in parallel, keep them in shared memory in the reference's order (ballot
 * compaction preserves the candidate order), and share the linear programs'
 * loops: finding the next half-plane that the solution violates, and the
 * bounds of that half-plane's line from the ones before it.  min / max are
 * exact, the per-element arithmetic is the per-thread code's, and "some line
 * is parallel and opposite" / "lo > hi" are order-free predicates, so the
 * results equal the per-thread LP's bit for bit.  The groups of a warp run
 * their loops together; a group that is done waits for the others.
 */
#ifndef ECMG_ORCA_GROUP_CUH
#define ECMG_ORCA_GROUP_CUH

#include "ecmg_internal.h"

namespace ecmg {

constexpr unsigned kFull = 0xffffffffu;

/* reductions over a group's lanes (every lane of the warp calls) */
template <int G>
__device__ __forceinline__ int group_min(int v)
{
#pragma unroll
    for (int o = G / 2; o; o >>= 1) v = min(v, __shfl_xor_sync(kFull, v, o));
    return v;
}
template <int G>
__device__ __forceinline__ unsigned group_ballot(bool p)
{
    const unsigned b = __ballot_sync(kFull, p);
    return G == 32 ? b : (b >> (threadIdx.x & 31 & ~(G - 1))) & ((1u << (G & 31)) - 1u);
}

__device__ __forceinline__ Con line_of(const float4* s, int i)
{
    const float4 f = s[i];
    Con c;
    c.p = mk(f.x, f.y);
    c.n = mk(f.z, f.w);
    return c;
}
__device__ __forceinline__ float4 line_f4(const Con& c) { return make_float4(c.p.x, c.p.y, c.n.x, c.n.y); }

/* bounds [lo, hi] on line h from the lines x < i (ORCA.cpp:461-497); a
   parallel line that excludes h gives lo > hi.  TRACE: *jlo / *jhi the first
   line that gave the bound (-1: none did) */
template <int G, bool TRACE, class Get>
__device__ __forceinline__ void group_bounds(const Get& get, bool on, const Con& h, int i, int sub, float* lo,
                                             float* hi, int* jlo, int* jhi)
{
    float llo = -INFINITY, lhi = INFINITY;
    int kl = 0x7fffffff, kh = 0x7fffffff;
    if (on) {
        const V2 rh = right(h.n);
        for (int x = sub; x < i; x += G) {
            Con g;
            if (!get(x, &g)) continue;
            const float den = det(rh, right(g.n));
            const float num = det(right(g.n), h.p - g.p);
            if (fabsf(den) <= kEps) {
                if (num < 0.0f) {
                    llo = INFINITY;
                    lhi = -INFINITY;
                }
                continue;
            }
            const float t = num / den;
            if (den >= 0.0f) {
                if (t < lhi) {
                    lhi = t;
                    if (TRACE) kh = x;
                }
            } else if (llo < t) {
                llo = t;
                if (TRACE) kl = x;
            }
        }
    }
#pragma unroll
    for (int o = G / 2; o; o >>= 1) {
        const float vh = __shfl_xor_sync(kFull, lhi, o), vl = __shfl_xor_sync(kFull, llo, o);
        if (TRACE) {
            const int oh = __shfl_xor_sync(kFull, kh, o), ol = __shfl_xor_sync(kFull, kl, o);
            if (vh < lhi || (vh == lhi && oh < kh)) kh = oh;
            if (llo < vl || (vl == llo && ol < kl)) kl = ol;
        }
        if (vh < lhi) lhi = vh;
        if (llo < vl) llo = vl;
    }
    if (lhi < *hi) {
        *hi = lhi;
        if (TRACE) *jhi = kh;
    }
    if (*lo < llo) {
        *lo = llo;
        if (TRACE) *jlo = kl;
    }
}

/* ORCA::RandomizedLP (ORCA.cpp:428-587) over the lines 0 .. n-1 that get()
   has; returns the failing index or n; every lane of a group has the result.
   Groups with `on` false take no part (n is returned, *out untouched). */
template <int G, bool TRACE, class Get>
__device__ __forceinline__ int lp2d_group(const Get& get, bool on, int n, V2 opt, float maxSpeed, bool useDirOpt,
                                          int sub, V2* out, LpTrace* tr)
{
    V2 v = *out;
    if (on) v = lp2d_start(opt, maxSpeed, useDirOpt);
    int i = -1, res = n;
    bool run = on;
    while (__any_sync(kFull, run)) {
        /* the next line whose half-plane does not contain v
           (Constraint::Contains; the lines between are skipped by the
           sequential loop) */
        int first = 0x7fffffff;
        if (run)
            for (int x = i + 1 + ((sub - i - 1) & (G - 1)); x < n; x += G) {
                Con c;
                if (!get(x, &c) || det(right(c.n), c.p - v) <= 0.0f) continue;
                first = x;
                break;
            }
        first = group_min<G>(first);
        run = run && first < n;
        Con h{};
        V2 dir{};
        float disc = 0.0f, dpd = 0.0f;
        if (run) {
            i = first;
            get(i, &h);
            dir = right(h.n);
            dpd = dot(dir, h.p);
            disc = dpd * dpd + maxSpeed * maxSpeed - dot(h.p, h.p);
            if (disc <= 0.0f) {
                res = i;
                run = false;
            }
        }
        /* a NaN discriminant: the line is passed over (ORCA.cpp:498-506) */
        const bool step = run && disc > 0.0f;
        const float sq = sqrtf(step ? disc : 0.0f);
        float lo = -dpd - sq, hi = -dpd + sq;
        int jlo = -1, jhi = -1;
        group_bounds<G, TRACE>(get, step, h, i, sub, &lo, &hi, &jlo, &jhi);
        if (step) {
            if (lo > hi) {
                res = i;
                run = false;
            } else if (useDirOpt) {
                if (dot(opt, dir) > 0) v = h.p + dir * hi;
                else v = h.p + dir * lo;
            } else {
                const float t = dot(dir, opt - h.p);
                if (t < lo) {
                    v = h.p + dir * lo;
                    if (TRACE) { tr->h = i; tr->src = jlo < 0 ? 1 : 2; tr->j = jlo; }
                } else if (t > hi) {
                    v = h.p + dir * hi;
                    if (TRACE) { tr->h = i; tr->src = jhi < 0 ? 1 : 2; tr->j = jhi; }
                } else {
                    v = h.p + dir * t;
                    if (TRACE) { tr->h = i; tr->src = 0; tr->j = -1; }
                }
            }
        }
    }
    *out = v;
    return res;
}

/* the agent's lines in order */
struct GroupLines {
    const float4* s;
    __device__ __forceinline__ bool operator()(int i, Con* c) const
    {
        *c = line_of(s, i);
        return true;
    }
};
/* the projected lines of RandomizedLP3D: the obstacle lines, then line i's
   bisectors with the neighbour lines j < i, at index j; where lines i and j
   have none (the reference skips them) the entry is marked by a NaN payload
   that no arithmetic produces */
struct GroupBisectors {
    const float4* s;
    const float4* bis;
    int nObst;
    __device__ __forceinline__ bool operator()(int i, Con* c) const
    {
        *c = line_of(i < nObst ? s + i : bis + (i - nObst), 0);
        return i < nObst || __float_as_uint(c->p.x) != kNoBisector;
    }
    static constexpr unsigned kNoBisector = 0x7fc0dea1u;
};

/* ORCA::RandomizedLP3D (ORCA.cpp:592-669) from line `failed` on.  The lines
   between two that v violates by more than the largest penetration so far are
   skipped, as in the sequential loop. */
template <int G>
__device__ __forceinline__ void lp3d_group(const float4* s, float4* bis, bool on, int m, int nObst, float maxSpeed,
                                           int failed, bool fp64, int sub, V2* vout)
{
    V2 v = *vout;
    float maxPen = 0.0f;
    int i = failed - 1;
    bool run = on;
    while (true) {
        int first = 0x7fffffff;
        if (run)
            for (int x = i + 1 + ((sub - i - 1) & (G - 1)); x < m; x += G) {
                const Con c = line_of(s, x);
                if (det(right(c.n), c.p - v) <= maxPen) continue;
                first = x;
                break;
            }
        first = group_min<G>(first);
        run = run && first < m;
        if (!__any_sync(kFull, run)) break;
        Con ci{};
        if (run) {
            i = first;
            ci = line_of(s, i);
            for (int j = nObst + sub; j < i; j += G) {
                const Con cj = line_of(s, j);
                const float dt = det(right(ci.n), right(cj.n));
                Con nc;
                nc.p = mk(__uint_as_float(GroupBisectors::kNoBisector), 0.0f);
                nc.n = mk(0.0f, 0.0f);
                bool keep = true;
                if (fabsf(dt) <= kEps) {
                    keep = !(dot(ci.n, cj.n) > 0);
                    if (keep) nc.p = (ci.p + cj.p) * 0.5f;
                } else if (!fp64) {
                    const float t = det(right(cj.n), ci.p - cj.p) / dt;
                    nc.p = ci.p + right(ci.n) * t;
                } else {
                    double ax = (double)cj.n.y, ay = -(double)cj.n.x; /* Right(cj.N) */
                    double bx = (double)ci.p.x - (double)cj.p.x, by = (double)ci.p.y - (double)cj.p.y;
                    double rx = (double)ci.n.y, ry = -(double)ci.n.x; /* Right(ci.N) */
                    double dd = rx * ay - ry * ax;
                    double t = (ax * by - ay * bx) / dd;
                    nc.p = mk((float)((double)ci.p.x + rx * t), (float)((double)ci.p.y + ry * t));
                }
                if (keep) nc.n = normalized(cj.n - ci.n);
                bis[j - nObst] = line_f4(nc);
            }
        }
        __syncwarp();
        V2 w = v;
        const int r = lp2d_group<G, false>(GroupBisectors{s, bis, nObst}, run, i, ci.n, maxSpeed, true, sub, &w, nullptr);
        if (run) {
            if (r >= i) v = w; /* else ORCA.cpp:658-664: the result before */
            maxPen = det(right(ci.n), ci.p - v);
        }
        __syncwarp(); /* bis is rewritten for the next line */
    }
    *vout = v;
}

/* verify_proposal (kernels.cu) for a group: the same conditions, the lanes
   over the lines */
template <int G>
__device__ __forceinline__ bool verify_group(const float4* s, bool on, int m, int nObst, int ncnt, V2 opt,
                                             float maxSpeed, int cls, int sub, V2* out)
{
    const float margin = 1e-4f;
    bool ok = on && cls < kClsOther;
    const bool pref = cls == kClsPref;
    int q = 0, qj = -1, kind = 0; /* kind 0 single, 1 circle, 2 pair */
    if (cls >= kClsCircle) {
        q = cls - kClsCircle;
        kind = 1;
    } else if (cls >= kClsPair) {
        const int p = cls - kClsPair;
        q = 1;
        while ((q + 1) * q / 2 <= p) q++; /* q*(q-1)/2 <= p < (q+1)*q/2 */
        qj = p - q * (q - 1) / 2;
        kind = 2;
    } else {
        q = cls - kClsSingle;
    }
    const int h = nObst + q, jsrc = kind == 2 ? nObst + qj : -1;
    if (!pref) ok = ok && q < ncnt && q < kMlpNbrs && h < m;
    Con H{};
    V2 dir{};
    float dpd = 0.0f, disc = 0.0f;
    if (ok && !pref) {
        H = line_of(s, h);
        dir = right(H.n);
        dpd = dot(dir, H.p);
        disc = dpd * dpd + maxSpeed * maxSpeed - dot(H.p, H.p);
        ok = disc > 0.0f;
    }
    const bool line = ok && !pref;
    const float sq = sqrtf(line ? disc : 0.0f);
    float lo = -dpd - sq, hi = -dpd + sq;
    int jlo = -1, jhi = -1;
    group_bounds<G, true>(GroupLines{s}, line, H, h, sub, &lo, &hi, &jlo, &jhi);
    V2 v = mk(0.0f, 0.0f);
    if (pref) {
        v = (len(opt) > maxSpeed) ? normalized(opt) * maxSpeed : opt;
    } else if (ok) {
        ok = !(lo > hi);
        const float t = dot(dir, opt - H.p);
        int src; /* -2 projection, -1 circle, else constraint index */
        if (t < lo) { v = H.p + dir * lo; src = jlo; }
        else if (t > hi) { v = H.p + dir * hi; src = jhi; }
        else { v = H.p + dir * t; src = -2; }
        ok = ok && src == (kind == 0 ? -2 : (kind == 1 ? -1 : jsrc));
        const V2 r = v - opt;
        if (kind != 1) { /* the speed circle must be slack as well */
            const float rs = maxSpeed - margin;
            ok = ok && rs > 0.0f && dot(v, v) < rs * rs;
        }
        if (kind == 0) {
            ok = ok && dot(r, H.n) > margin;
        } else if (kind == 2) {
            if (ok) {
                const Con g = line_of(s, jsrc);
                const float d2 = det(H.n, g.n);
                ok = det(r, g.n) / d2 > margin && det(H.n, r) / d2 > margin;
            }
        } else {
            const V2 nv = v * -1.0f;
            const float d2 = det(H.n, nv);
            ok = ok && fabsf(d2) > kEps && det(r, nv) / d2 > margin && det(H.n, r) / d2 > margin * maxSpeed;
        }
    }
    bool bad = false;
    if (ok)
        for (int i = sub; i < m; i += G) {
            const Con c = line_of(s, i);
            const float d = det(right(c.n), c.p - v);
            if (pref) bad |= d > 0.0f;
            else if (i > h) bad |= d > 0.0f;
            else if (i != h && i != jsrc) bad |= !(d < -margin);
        }
    ok = group_ballot<G>(bad) == 0u && ok;
    if (ok) *out = v;
    return ok;
}

struct GroupCounts {
    int lp3d = 0, proposed = 0, accepted = 0;
};

/* shared memory of one agent: its lines, then the bisectors; the pad puts
   the groups of a quarter warp on different banks for G = 4 */
template <int K>
constexpr int kGroupLines = K + kMaxObstCons;
template <int K>
constexpr int kGroupRow = kGroupLines<K> + K + 4;

/* ApplyObstacleAvoidanceForce + UpdateVelocitySystem + UpdatePositionSystem
   of grid-order agent t (`in` false: none), G lanes.  FULL keeps the learned
   proposal's check, the trace labels and the recording of the step. */
template <int K, int G, bool FULL>
__device__ __forceinline__ void orca_group(const TickArgs& a, int t, bool in, float4* s, GroupCounts& gc)
{
    const int sub = threadIdx.x & (G - 1);
    const int slot = in ? a.s_slot[t] : 0;
    const bool on = in && a.active[slot] == 1; /* else inactive, or waiting for its re-plan (k_fixup) */
    V2 pos{}, vel{}, pv{};
    float clr = 0.0f, speed = 0.0f;
    int ncnt = 0;
    int b = 0, e = 0;
    const int* items = nullptr;
    const SceneDev& sc = a.scenes[on && a.slot_scene ? a.slot_scene[slot] : 0];
    if (on) {
        pos = a.s_pos[t];
        const float4 rec = a.s_rec[t];
        vel = mk(rec.x, rec.y);
        clr = rec.z;
        speed = rec.w;
        pv = a.pref_vel[slot];
        ncnt = a.ncnt[t];
    }
    const float maxSpeed = a.max_speed > 0.0f ? a.max_speed : speed;
    const int* nbr = a.nbr + (size_t)t * a.k;
    const float range = a.tau_o * maxSpeed + clr;
    const float rsq = range * range;
    const ObstView& ob = sc.ob;
    if (on) {
        const float fx = (pos.x - ob.gx0) * ob.ginv, fy = (pos.y - ob.gy0) * ob.ginv;
        if (ob.g_start && range <= ob.reach && fx >= 0.0f && fy >= 0.0f && fx < (float)ob.gw && fy < (float)ob.gh) {
            const int g = (int)fy * ob.gw + (int)fx;
            b = ob.g_start[g];
            e = ob.g_start[g + 1];
            items = ob.g_items;
        } else {
            e = ob.n_verts; /* linear scan: the reference's own loop */
        }
    }
    int m = 0;
    for (; __any_sync(kFull, b < e); b += G) {
        const int q = b + sub;
        bool emit = false;
        Con c;
        if (q < e) {
            const int L = items ? items[q] : q;
            if (obstacle_in_range(ob, L, pos, rsq)) emit = obstacle_constraint(ob, L, pos, vel, clr, a.tau_o, &c);
        }
        const unsigned bal = group_ballot<G>(emit);
        if (emit) {
            const int at = m + __popc(bal & ((1u << sub) - 1u));
            if (at < kMaxObstCons) s[at] = line_f4(c);
            else atomicOr(&a.counters[C_ERROR], ECMG_DEV_ERR_CONSTRAINTS);
        }
        m += __popc(bal);
    }
    const int nObst = min(m, kMaxObstCons);
    for (int q = sub; q < ncnt; q += G) {
        const int j = nbr[q];
        V2 np, nv;
        float nc;
        if (j >= 0) {
            np = a.s_pos[j];
            const float4 rec = a.s_rec[j];
            nv = mk(rec.x, rec.y);
            nc = rec.z;
        } else {
            /* kd-tree mode: a cache entry left by an earlier agent that is
               not in this tick's grid; its slot is not written this tick */
            const int sl = -j - 1;
            np = a.pos[sl];
            nv = a.vel[sl];
            nc = a.clear[sl];
        }
        s[nObst + q] = line_f4(agent_constraint(pos, vel, clr, np, nv, nc, a.tau_a, a.dt, a.inv_tau_a));
    }
    m = nObst + ncnt;
    __syncwarp();

    V2 v = mk(0.0f, 0.0f);
    bool accepted = false;
    if (FULL && (a.cls || a.cls_slot)) {
        const int c = !on ? kClsOther : (a.cls_slot ? a.cls_slot[slot] : a.cls[t]);
        accepted = verify_group<G>(s, on, m, nObst, ncnt, pv, maxSpeed, c, sub, &v);
        if (sub == 0) {
            gc.proposed += c != kClsOther ? 1 : 0;
            gc.accepted += accepted ? 1 : 0;
        }
    }
    int failed = m;
    const bool solve = on && !accepted;
    if (FULL && a.label) {
        LpTrace tr;
        failed = lp2d_group<G, true>(GroupLines{s}, solve, m, pv, maxSpeed, false, sub, &v, &tr);
        if (solve && sub == 0) a.label[t] = (unsigned char)label_of(tr, failed, m, nObst);
    } else {
        failed = lp2d_group<G, false>(GroupLines{s}, solve, m, pv, maxSpeed, false, sub, &v, nullptr);
    }
    const bool need3d = solve && failed < m;
    if (__any_sync(kFull, need3d)) {
        lp3d_group<G>(s, s + kGroupLines<K>, need3d, m, nObst, maxSpeed, failed, FULL && a.lp3d_fp64, sub, &v);
        if (need3d && sub == 0) gc.lp3d++;
    }

    if (on) {
        /* force = vOrca - v (Simulator.cpp:676-677); UpdateVelocitySystem
           (Simulator.cpp:619-635); UpdatePositionSystem (Simulator.cpp:592-606) */
        if (sub == 0) {
            const float fx = v.x - vel.x, fy = v.y - vel.y;
            const V2 nv = mk(vel.x + fx * a.mass_recip * a.dt, vel.y + fy * a.mass_recip * a.dt);
            a.vel[slot] = nv;
            a.pos[slot] = mk(pos.x + (nv.x * a.dt), pos.y + (nv.y * a.dt));
        }
        if (FULL && a.rec_cnt) {
            for (int q = sub; q < a.k; q += G)
                a.rec_nbr[slot * a.k + q] = q < ncnt ? (nbr[q] >= 0 ? a.s_slot[nbr[q]] : -nbr[q] - 1) : -1;
            if (sub == 0) {
                a.rec_cnt[slot] = ncnt;
                a.rec_vorca[slot] = v;
                a.rec_fail[slot] = failed;
                a.rec_ncons[slot] = m;
                a.rec_nobst[slot] = nObst;
            }
        }
    }
    __syncwarp(); /* the lines are rewritten for the warp's next agents */
}

}  // namespace ecmg
#endif
