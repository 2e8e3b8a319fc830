/*
 * kernels.cu -- the per-tick kernels.
 *
 * One tick (Simulator::Update, ECMAgentSimulator/Simulator.cpp:314-323) is
 *   k_bin      bucket every active slot into the uniform agent grid
 *   k_scan     exclusive scan of the bucket counts
 *   k_scatter  tick-start snapshot of position/velocity/radius in grid order
 *   k_attract  attraction point (IRM) and preferred velocity (second stream)
 *   k_neighbors exact kNN on the grid (knn_rows.cuh)
 *   k_agents_group / k_agents  several lanes or one thread per agent
 *              (orca_group.cuh): obstacle + agent ORCA half-planes, 2D LP
 *              (+3D LP), velocity and position update
 * The snapshot makes the tick Jacobi-exact: neighbours are read from the
 * tick-start copy while each thread writes its own slot, which is what the
 * reference's system order guarantees (velocities change only in
 * UpdateVelocitySystem, after every agent's ORCA query).
 *
 * Built with -fmad=false: every float expression is the reference's sequence
 * of separately rounded operations.
 */
#include "ecmg_internal.h"
#include "knn_rows.cuh"
#include "launch_ahead.cuh"

#include <cuda_bf16.h>
#include <stdint.h>

#include <type_traits>

namespace ecmg {

/* the counters of a tick: zero but for the last slot (the other kernels of
   the tick start after the binning) */
__device__ __forceinline__ int start_counters(const BinArgs& a)
{
    const int last = a.n_fixed > 0 ? a.n_fixed - 1 : *a.last;
    if (blockIdx.x == 0 && threadIdx.x < kCounters) a.counters[threadIdx.x] = threadIdx.x == C_LAST ? last : 0;
    return last;
}

__global__ void k_bin(BinArgs a)
{
    const int last = start_counters(a);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= last; i += gridDim.x * blockDim.x) {
        if (!a.active[i]) {
            if (a.out_cnt) a.out_cnt[i] = 0;
            continue;
        }
        int b;
        if (a.scenes) {
            const SceneDev& sc = a.scenes[a.slot_scene ? a.slot_scene[i] : 0];
            b = sc.bucket_base + bucket_of(sc.grid, a.pos[i]);
        } else {
            b = bucket_of(a.grid, a.pos[i]);
        }
        a.key[i] = b;
        a.rank[i] = atomicAdd(&a.cell_count[b], 1);
    }
}

/* ---- exclusive scan of the bucket counts --------------------------------
   Three launches bin a tick: k_bin, k_scan (every block scans its 4,096
   counts in place; the last block to finish scans the block sums) and
   k_scatter (adds the block sums while it places the agents, and writes the
   final bucket starts).  The launches bound small crowds: with a scan of
   three launches and a clearing of the counts in front (now k_attract's) a
   tick of 1,000 agents took 95 us of device time, with this and the 64-byte
   edge records 72.  At a million 14.8, 8.1 and 36.1 us: k_scatter is bound by
   its scattered sectors (four slots in flight per thread: 37 -> 42). */
constexpr int kScanBlock = 1024, kScanPer = 4, kScanTile = kScanBlock * kScanPer;

__device__ __forceinline__ int block_exclusive_scan(int v, int* sh, int* total)
{
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[w] = x;
    __syncthreads();
    if (w == 0) {
        int s = lane < (blockDim.x >> 5) ? sh[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        sh[lane] = s;
    }
    __syncthreads();
    int incl = x + (w > 0 ? sh[w - 1] : 0);
    *total = sh[(blockDim.x >> 5) - 1];
    __syncthreads();
    return incl - v;
}

__global__ void __launch_bounds__(kScanBlock) k_scan(int* counts, int n, int* block_sums, int* counters)
{
    __shared__ int sh[32];
    __shared__ bool last;
    wait_for_previous();
    const int i0 = blockIdx.x * kScanTile + threadIdx.x * kScanPer;
    int v[kScanPer], sum = 0, tot;
#pragma unroll
    for (int q = 0; q < kScanPer; q++) {
        v[q] = i0 + q < n ? counts[i0 + q] : 0;
        sum += v[q];
    }
    int run = block_exclusive_scan(sum, sh, &tot);
#pragma unroll
    for (int q = 0; q < kScanPer; q++) {
        if (i0 + q < n) counts[i0 + q] = run;
        run += v[q];
    }
    if (threadIdx.x == 0) {
        block_sums[blockIdx.x] = tot;
        __threadfence();
        last = atomicAdd(&counters[C_SCANNED], 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    int carry = 0;
    const int nb = gridDim.x;
    for (int base = 0; base < nb; base += kScanBlock) {
        const int i = base + threadIdx.x;
        const int x = i < nb ? __ldcg(block_sums + i) : 0;
        const int ex = block_exclusive_scan(x, sh, &tot);
        if (i < nb) block_sums[i] = ex + carry;
        carry += tot;
    }
    if (threadIdx.x == 0) counters[C_NSORTED] = carry;
}

int scan_tmp_ints(int n) { return (n + 1023) / 1024 + 32; }

/* tick-start snapshot in grid order, and the final bucket starts */
__global__ void k_scatter(BinArgs a)
{
    wait_for_previous();
    const int last = a.counters[C_LAST];
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    for (int i = t0; i <= last; i += step) {
        if (!a.active[i]) continue;
        const int b = a.key[i];
        const int d = a.cell_count[b] + a.block_sums[b / kScanTile] + a.rank[i];
        a.s_slot[d] = i;
        a.s_pos[d] = a.pos[i];
        if (a.s_rec) a.s_rec[d] = make_float4(a.vel[i].x, a.vel[i].y, a.clear[i], a.speed[i]);
    }
    for (int c = t0; c < a.total_buckets; c += step) a.cell_start[c] = a.cell_count[c] + a.block_sums[c / kScanTile];
    if (t0 == 0) a.cell_start[a.total_buckets] = a.counters[C_NSORTED];
}

/* the whole binning of up to kSmallSlots slots by one block, the counts in
   shared memory: below that size the three launches' latency is all there is
   (1,000 agents: with three launches the tick's device time 72 us, with this
   65; the kernel 8.3 us under ncu).  The line is what a block's shared memory
   and registers hold. */
constexpr int kSmallSlots = 8192, kSmallCells = 11264, kSmallBlock = 1024;
__global__ void __launch_bounds__(kSmallBlock) k_bin_small(BinArgs a)
{
    constexpr int R = kSmallSlots / kSmallBlock, C = kSmallCells / kSmallBlock;
    __shared__ int count[kSmallCells];
    __shared__ int sh[32];
    const int last = start_counters(a);
    for (int c = threadIdx.x; c < kSmallCells; c += kSmallBlock) count[c] = 0;
    __syncthreads();
    int bucket[R], rank[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int i = r * kSmallBlock + threadIdx.x;
        bucket[r] = -1;
        rank[r] = 0;
        if (i > last) continue;
        if (!a.active[i]) {
            if (a.out_cnt) a.out_cnt[i] = 0;
            continue;
        }
        if (a.scenes) {
            const SceneDev& sc = a.scenes[a.slot_scene ? a.slot_scene[i] : 0];
            bucket[r] = sc.bucket_base + bucket_of(sc.grid, a.pos[i]);
        } else {
            bucket[r] = bucket_of(a.grid, a.pos[i]);
        }
    }
#pragma unroll
    for (int r = 0; r < R; r++)
        if (bucket[r] >= 0) rank[r] = atomicAdd(&count[bucket[r]], 1);
    __syncthreads();
    int v[C], sum = 0, tot;
#pragma unroll
    for (int q = 0; q < C; q++) {
        v[q] = count[threadIdx.x * C + q]; /* an odd stride: no bank conflicts */
        sum += v[q];
    }
    int run = block_exclusive_scan(sum, sh, &tot);
#pragma unroll
    for (int q = 0; q < C; q++) {
        count[threadIdx.x * C + q] = run;
        run += v[q];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; r++) {
        if (bucket[r] < 0) continue;
        const int i = r * kSmallBlock + threadIdx.x;
        const int d = count[bucket[r]] + rank[r];
        a.key[i] = bucket[r];
        a.rank[i] = rank[r];
        a.s_slot[d] = i;
        a.s_pos[d] = a.pos[i];
        if (a.s_rec) a.s_rec[d] = make_float4(a.vel[i].x, a.vel[i].y, a.clear[i], a.speed[i]);
    }
    for (int c = threadIdx.x; c < a.total_buckets; c += kSmallBlock) a.cell_start[c] = count[c];
    if (threadIdx.x == 0) {
        a.cell_start[a.total_buckets] = tot;
        a.counters[C_NSORTED] = tot;
    }
}

static bool bins_small(const BinArgs& b, int slots) { return slots <= kSmallSlots && b.total_buckets <= kSmallCells; }
int bin_kernels(int total_buckets, int slots)
{
    BinArgs b{};
    b.total_buckets = total_buckets;
    return bins_small(b, slots) ? 1 : 3;
}

/* blocks for work on every bucket, four buckets a thread to 8 blocks an SM:
   where the agents alone give the grid, a few of them in a large one leave the
   buckets to a few threads (300 agents in 25 million cells: query 18,450 us,
   with these 206; in 3 million cells of 0.3 m: tick 1,572 and 120) */
static int blocks_of_buckets(int buckets, int threads)
{
    const int per = 4 * threads;
    return std::min((buckets + per - 1) / per, 152 * 8);
}

/* counts (zero) -> bins, starts and snapshot */
static cudaError_t launch_bin(const BinArgs& b, int slots, int blocks, cudaStream_t s)
{
    if (bins_small(b, slots)) {
        k_bin_small<<<1, kSmallBlock, 0, s>>>(b);
        return cudaGetLastError();
    }
    k_bin<<<blocks, 256, 0, s>>>(b);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess)
        e = launch_ahead(k_scan, (b.total_buckets + kScanTile - 1) / kScanTile, kScanBlock, 0, s, b.cell_count,
                         b.total_buckets, b.block_sums, b.counters);
    /* k_scatter writes every bucket's start too: enough blocks for those of a
       few agents in a large grid */
    if (e == cudaSuccess)
        e = launch_ahead(k_scatter, std::max(blocks, blocks_of_buckets(b.total_buckets, 256)), 256, 0, s, b);
    return e;
}

/* ---------------------------------------------------------------------- */
struct LocalGet {
    const Con* c;
    __device__ Con operator()(int i) const { return c[i]; }
};

/* adds the number of lanes with pred set to *ctr with one atomic per warp */
__device__ __forceinline__ void warp_count(int* ctr, bool pred)
{
    unsigned m = __activemask();
    unsigned b = __ballot_sync(m, pred);
    if ((threadIdx.x & 31) == __ffs(m) - 1 && b) atomicAdd(ctr, __popc(b));
}

/* class of an LP result for the proposal's training labels (kCls*) */
__device__ __forceinline__ int label_of(const LpTrace& tr, int failed, int m, int nObst)
{
    if (failed < m) return kClsOther;
    if (tr.h < 0) return kClsPref;
    int q = tr.h - nObst;
    if (q < 0 || q >= kMlpNbrs) return kClsOther;
    if (tr.src == 0) return kClsSingle + q;
    if (tr.src == 1) return kClsCircle + q;
    int qj = tr.j - nObst;
    if (qj < 0) return kClsOther;
    return kClsPair + q * (q - 1) / 2 + qj;
}

}  // namespace ecmg
#include "orca_group.cuh"
namespace ecmg {

constexpr int kGroupWarps = 4; /* per block */

/* Exact check of a proposed active set.  Returns true only when the
   incremental LP (lp2d, ORCA.cpp:428-587) provably ends with its last update
   on the proposed half-plane h, fixed by the proposed bound; *out is then
   computed with the LP's own final-step formula, so it is the LP's result.
   Conditions: the bounds of h over every earlier half-plane and the speed
   circle reproduce the proposed source; every later half-plane contains the
   point (the LP's own test); the KKT multipliers of the proposed active set
   are positive and every other earlier half-plane is slack, both by a margin,
   so that the LP state before h violates h. */
template <class Get>
__device__ __noinline__ bool verify_proposal(const Get& get, int m, int nObst, int ncnt, V2 opt, float maxSpeed,
                                             int cls, V2* out)
{
    const float margin = 1e-4f;
    if (cls == kClsPref) {
        V2 v0 = (len(opt) > maxSpeed) ? normalized(opt) * maxSpeed : opt;
        for (int i = 0; i < m; i++) {
            Con c = get(i);
            if (det(right(c.n), c.p - v0) > 0.0f) return false;
        }
        *out = v0;
        return true;
    }
    int q, qj = -1, kind; /* kind 0 single, 1 circle, 2 pair */
    if (cls >= kClsSingle && cls < kClsPair) { q = cls - kClsSingle; kind = 0; }
    else if (cls >= kClsCircle && cls < kClsOther) { q = cls - kClsCircle; kind = 1; }
    else if (cls >= kClsPair && cls < kClsCircle) {
        int p = cls - kClsPair;
        q = 1;
        while ((q + 1) * q / 2 <= p) q++; /* q*(q-1)/2 <= p < (q+1)*q/2 */
        qj = p - q * (q - 1) / 2;
        kind = 2;
    } else return false;
    if (q >= ncnt || q >= kMlpNbrs) return false;
    const int h = nObst + q, jsrc = kind == 2 ? nObst + qj : -1;
    if (h >= m) return false;
    Con H = get(h);
    V2 dir = right(H.n);
    float dpd = dot(dir, H.p);
    float disc = dpd * dpd + maxSpeed * maxSpeed - dot(H.p, H.p);
    if (!(disc > 0.0f)) return false;
    float sq = sqrtf(disc);
    float lo = -dpd - sq, hi = -dpd + sq;
    int lo_src = -1, hi_src = -1;
    for (int j = 0; j < h; j++) {
        Con G = get(j);
        float den = det(right(H.n), right(G.n));
        float num = det(right(G.n), H.p - G.p);
        if (fabsf(den) <= kEps) {
            if (num < 0.0f) return false;
            continue;
        }
        const float t = num / den;
        if (den >= 0.0f) {
            if (t < hi) hi_src = j;
            hi = (t < hi) ? t : hi;
        } else {
            if (lo < t) lo_src = j;
            lo = (lo < t) ? t : lo;
        }
    }
    if (lo > hi) return false;
    float t = dot(dir, opt - H.p);
    V2 v;
    int src; /* -2 projection, -1 circle, else constraint index */
    if (t < lo) { v = H.p + dir * lo; src = lo_src; }
    else if (t > hi) { v = H.p + dir * hi; src = hi_src; }
    else { v = H.p + dir * t; src = -2; }
    if (kind == 0 && src != -2) return false;
    if (kind == 1 && src != -1) return false;
    if (kind == 2 && src != jsrc) return false;
    for (int i = h + 1; i < m; i++) {
        Con c = get(i);
        if (det(right(c.n), c.p - v) > 0.0f) return false;
    }
    /* KKT of min |v - opt|^2 s.t. dot(N_i, v - P_i) >= 0, |v| <= maxSpeed */
    V2 r = v - opt;
    if (kind != 1) { /* the speed circle must be slack as well */
        float rs = maxSpeed - margin;
        if (!(rs > 0.0f && dot(v, v) < rs * rs)) return false;
    }
    if (kind == 0) {
        if (!(dot(r, H.n) > margin)) return false;
    } else if (kind == 2) {
        Con G = get(jsrc);
        float d2 = det(H.n, G.n);
        float la = det(r, G.n) / d2, lb = det(H.n, r) / d2;
        if (!(la > margin && lb > margin)) return false;
    } else {
        V2 nv = v * -1.0f;
        float d2 = det(H.n, nv);
        if (!(fabsf(d2) > kEps)) return false;
        float la = det(r, nv) / d2, lb = det(H.n, r) / d2;
        if (!(la > margin && lb > margin * maxSpeed)) return false;
    }
    for (int i = 0; i < h; i++) {
        if (i == jsrc) continue;
        Con c = get(i);
        if (!(det(right(c.n), c.p - v) < -margin)) return false;
    }
    *out = v;
    return true;
}

/* out-of-line copies keep the per-agent kernel small enough for the
   instruction cache: each is called from a loop or a rare branch */
__device__ __noinline__ Con agent_constraint_ni(V2 position, V2 velocity, float clr, V2 np, V2 nv, float nclr,
                                                float tau, float dt, float inv_tau)
{
    return agent_constraint(position, velocity, clr, np, nv, nclr, tau, dt, inv_tau);
}

template <int MC, bool FULL>
__device__ __noinline__ void lp3d_local(const Con* cons, int m, int nObst, float maxSpeed, int failed, V2* v,
                                        bool fp64)
{
    Con proj[MC - kMaxObstCons]; /* bisectors: at most the neighbour constraints */
    LocalGet get{cons};
    lp3d(get, m, nObst, maxSpeed, failed, v, proj, FULL && fp64);
}

/* attraction point and preferred velocity of grid-order agent t; `lead`: this
   thread writes (all threads of an agent take the same way); locate and
   attract_point: the point location and the IRM, by one thread or by several */
template <class Locate, class AttractPoint>
__device__ __forceinline__ void attract_agent(const TickArgs& a, int t, bool lead, Locate locate,
                                              AttractPoint attract_point)
{
    const int slot = a.s_slot[t];
    if (a.active[slot] & kActivePending) return; /* done by k_fixup once its new path is in */
    const V2 pos = a.s_pos[t];
    const float speed = a.s_rec[t].w;
    const SceneDev& sc = a.scenes[a.slot_scene ? a.slot_scene[slot] : 0];
    /* the point location of the retraction, issued before the path loads
       (independent chains of dependent loads); unused when the agent arrives */
    const int cell = locate(sc.ecm, pos);

    /* UpdateAttractionPointSystem (Simulator.cpp:538-590) */
    const int off = a.path_off[slot], np = a.path_len[slot];
    const V2* path = a.path_xy + off;
    const V2 goal = path[np - 1];
    float gdx = pos.x - goal.x, gdy = pos.y - goal.y;
    float dist = gdx * gdx + gdy * gdy;
    V2 attr;
    if (dist < a.arr_sq) {
        attr = goal;
        if (lead) a.attr[slot] = attr;
        if (dist < a.del_sq) { /* DestroyAgent: skipped by every later system */
            if (!lead) return;
            a.active[slot] = 0;
            int q = atomicAdd(&a.counters[C_DESTROYED], 1);
            if (q < a.list_cap) a.destroyed_list[q] = slot;
            else atomicOr(&a.counters[C_ERROR], ECMG_DEV_ERR_LIST);
            if (a.rec_cnt) a.rec_cnt[slot] = -1;
            return;
        }
    } else {
        V2 ap = mk(0.0f, 0.0f); /* Point attractionPoint; (0,0) */
        bool no_retract = false;
        int red = -1;
        if (attract_point(sc.ecm, pos, path, np, &ap, &no_retract, &red, cell)) {
            attr = ap;
            if (lead) a.attr[slot] = attr;
        } else {
            attr = a.attr[slot]; /* unchanged; the host re-plans before the next tick */
            if (!lead) return;
            if (a.replan_dev_fail && (no_retract || (red >= 0 && a.fail_edge[slot] == red))) {
                /* the built-in planner starts by retracting this same position
                   with the same point location; it fails there, or its search
                   already failed from this ECM edge for this goal and clearance
                   (a property of the edge only).  Either way the re-plan fails:
                   the agent keeps its path and attraction point without a host
                   round trip. */
                atomicAdd(&a.counters[C_REPLAN_DEV], 1);
            } else {
                int q = atomicAdd(&a.counters[C_REPLAN], 1);
                if (q < a.list_cap) { a.replan_list[q] = slot; a.replan_pos[q] = pos; }
                else atomicOr(&a.counters[C_ERROR], ECMG_DEV_ERR_LIST);
            }
        }
    }

    /* ApplySteeringForce (Simulator.cpp:638-657) */
    V2 pv = normalize(attr - pos) * speed;
    if (lead) a.pref_vel[slot] = pv;
}

__device__ void attract_tick(const TickArgs& a, int t)
{
    attract_agent(
        a, t, true, [](const EcmView& e, V2 p) { return point_location_inl(e, p); },
        [](const EcmView& e, V2 p, const V2* path, int np, V2* out, bool* nr, int* ed, int cell) {
            return irm(e, p, path, np, out, nr, ed, cell);
        });
}

/* ApplyObstacleAvoidanceForce + UpdateVelocitySystem + UpdatePositionSystem
   of grid-order agent t (agents destroyed this tick are skipped).  FULL
   keeps the learned proposal's check, the trace labels, the recording of the
   step, the FP64 bisectors and the kd-tree mode's entries outside the grid;
   the plain tick's kernel is compiled without them (a fifth of its stalls are
   for instructions; the same arithmetic). */
template <int K, bool FULL = true>
__device__ void orca_tick(const TickArgs& a, int t)
{
    const int slot = a.s_slot[t];
    if (a.active[slot] != 1) return; /* inactive, or waiting for its re-plan (k_fixup) */
    const V2 pos = a.s_pos[t];
    const float4 rec = a.s_rec[t];
    const V2 vel = mk(rec.x, rec.y);
    const float clr = rec.z, speed = rec.w;
    const SceneDev& sc = a.scenes[a.slot_scene ? a.slot_scene[slot] : 0];
    const V2 pv = a.pref_vel[slot];

    /* ORCA::GetVelocity (ORCA.cpp:14-57) with maxSpeed = preferred speed
       (Simulator.cpp:671) unless a global maximum is configured */
    const float maxSpeed = a.max_speed > 0.0f ? a.max_speed : speed;
    const int ncnt = a.ncnt[t];
    const int* nbr = a.nbr + (size_t)t * a.k;
    constexpr int MC = K + kMaxObstCons; /* constraint capacity */
    Con cons[MC];
    LocalGet get{cons};
    /* the plain tick takes each constraint into RandomizedLP as soon as it is
       built (the LP's steps in the same order as over the finished list) */
    V2 v = lp2d_start(pv, maxSpeed, false);
    int failed2 = -1;
    int m = 0;
    bool overflow = false;
    const float range = a.tau_o * maxSpeed + clr;
    const float rsq = range * range;
    {
        const ObstView& o = sc.ob;
        int b = 0, e = 0;
        const int* items = nullptr;
        float fx = (pos.x - o.gx0) * o.ginv, fy = (pos.y - o.gy0) * o.ginv;
        if (o.g_start && range <= o.reach && fx >= 0.0f && fy >= 0.0f && fx < (float)o.gw && fy < (float)o.gh) {
            int g = (int)fy * o.gw + (int)fx;
            b = o.g_start[g];
            e = o.g_start[g + 1];
            items = o.g_items;
        } else {
            e = o.n_verts; /* linear scan: the reference's own loop */
        }
        for (int q = b; q < e; q++) {
            int L = items ? items[q] : q;
            if (!obstacle_in_range(o, L, pos, rsq)) continue;
            Con c;
            if (obstacle_constraint_inl(o, L, pos, vel, clr, a.tau_o, &c)) {
                if (m < MC - K) {
                    cons[m] = c;
                    if (!FULL && failed2 < 0 && !lp2d_step(get, m, c, pv, maxSpeed, false, &v)) failed2 = m;
                    m++;
                } else {
                    overflow = true;
                }
            }
        }
    }
    const int nObst = m;
    for (int q = 0; q < ncnt; q++) {
        const int j = nbr[q];
        if (!FULL || j >= 0) {
            /* inline in the plain kernel (no other callers compete for the
               instruction cache there), out of line in the full one */
            const float4 r = a.s_rec[j];
            cons[m] = agent_constraint(pos, vel, clr, a.s_pos[j], mk(r.x, r.y), r.z, a.tau_a, a.dt, a.inv_tau_a);
        } else {
            /* kd-tree mode: a cache entry left by an earlier agent that is
               not in this tick's grid; its slot is not written this tick */
            const int sl = -j - 1;
            cons[m] = agent_constraint_ni(pos, vel, clr, a.pos[sl], a.vel[sl], a.clear[sl], a.tau_a, a.dt,
                                          a.inv_tau_a);
        }
        if (!FULL && failed2 < 0 && !lp2d_step(get, m, cons[m], pv, maxSpeed, false, &v)) failed2 = m;
        m++;
    }
    if (overflow) atomicOr(&a.counters[C_ERROR], ECMG_DEV_ERR_CONSTRAINTS);

    int failed = -1;
    if (FULL && (a.cls || a.cls_slot)) { /* learned proposal: accepted only when the exact check passes */
        const int c = a.cls_slot ? a.cls_slot[slot] : a.cls[t];
        bool ok = c != kClsOther && verify_proposal(get, m, nObst, ncnt, pv, maxSpeed, c, &v);
        if (ok) failed = m;
        warp_count(&a.counters[C_PROPOSED], c != kClsOther);
        warp_count(&a.counters[C_ACCEPTED], ok);
    }
    bool need3d = false;
    if (failed < 0) {
        if (FULL && a.label) {
            LpTrace tr;
            failed = lp2d<LocalGet, true>(get, m, pv, maxSpeed, false, &v, &tr);
            a.label[t] = (unsigned char)label_of(tr, failed, m, nObst);
        } else if (FULL) {
            failed = lp2d(get, m, pv, maxSpeed, false, &v);
        } else {
            failed = failed2 < 0 ? m : failed2;
        }
        if (failed < m) {
            lp3d_local<MC, FULL>(cons, m, nObst, maxSpeed, failed, &v, a.lp3d_fp64 != 0);
            need3d = true;
        }
    }
    warp_count(&a.counters[C_LP3D], need3d);

    /* force = vOrca - v (Simulator.cpp:676-677); UpdateVelocitySystem
       (Simulator.cpp:619-635); UpdatePositionSystem (Simulator.cpp:592-606) */
    float fx = v.x - vel.x, fy = v.y - vel.y;
    V2 nv = mk(vel.x + fx * a.mass_recip * a.dt, vel.y + fy * a.mass_recip * a.dt);
    V2 npos = mk(pos.x + (nv.x * a.dt), pos.y + (nv.y * a.dt));
    a.vel[slot] = nv;
    a.pos[slot] = npos;

    if (FULL && a.rec_cnt) {
        a.rec_cnt[slot] = ncnt;
        for (int q = 0; q < a.k; q++)
            a.rec_nbr[slot * a.k + q] = q < ncnt ? (nbr[q] >= 0 ? a.s_slot[nbr[q]] : -nbr[q] - 1) : -1;
        a.rec_vorca[slot] = v;
        a.rec_fail[slot] = failed;
        a.rec_ncons[slot] = m;
        a.rec_nobst[slot] = nObst;
    }
}

/* neighbour lists of every grid-order agent of the tick (knn_rows.cuh).
   Persistent: a warp takes 32 consecutive grid-order agents per work grab
   (neighbouring agents: their candidates share L1), so that warps whose
   agents have more candidates do not leave the SMs' last wave ragged.  Bound
   by instruction issue: 158 warp instructions per agent at 30.2 of 32 threads
   (250,000 of the crossing); a million 287 us beside k_attract (416 with one
   insertion per candidate and cells in distance order), 25,000 23 (86-105,
   where a cell of more than 32 agents sent its lanes to the 64-bit search) */
constexpr int kNbrWarps = 4; /* per block */
/* The variant for crowded cells (CROWDS) costs the ordinary search registers
   wherever it stands in the kernel: a tick of 100 agents 55.7 -> 56.7 us, of
   1,000 60.3 -> 60.9, a query of 100 points 16.5 -> 17.4, of 3,000 26.6 -> 27.4.
   Crowds that are small leave a lane's 64-bit search little to do: ticks to
   8,192 slots and queries to 2,048 points do without. */
constexpr int kCrowdSlots = 8192, kCrowdPoints = 2048;
template <int K, bool CROWDS>
__global__ void __launch_bounds__(32 * kNbrWarps, K <= 16 ? 8 : 4) k_neighbors(TickArgs a)
{
    __shared__ KnnSm<K> sm[kNbrWarps];
    const int n = a.counters[C_NSORTED];
    const int lane = threadIdx.x & 31;
    while (true) {
        int base = 0;
        if (lane == 0) base = atomicAdd(&a.counters[C_NBR_WORK], 32);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= n) break;
        const int t = min(base + lane, n - 1);
        const bool in = base + lane < n;
        const SceneDev& sc = a.scenes[a.slot_scene ? a.slot_scene[a.s_slot[t]] : 0];
        const int c = knn_list<K, false, CROWDS>(sm[threadIdx.x >> 5], in, a.k, a.s_pos[t], a.rnb2, a.s_pos, a.s_slot,
                                                 a.cell_start + sc.bucket_base, sc.grid, a.nbr + (size_t)t * a.k);
        if (in) a.ncnt[t] = c;
    }
}

/* ---- the attraction stage with kAttractLanes lanes per agent --------------
   attract_tick's steps, the cells of the point location and the segments of
   the path shared out: the first cell (list order) that holds the agent, and
   the last segment that gives a point, are the sequential loops' results.
   Bound by that chain of dependent loads; 8 lanes because paths have about a
   dozen points and grid cells a handful of ECM cells (1,000 agents: 20.5 ->
   12.3 us, their tick 71 -> 65). */
constexpr int kAttractLanes = 8;

__device__ __forceinline__ int locate_group(const EcmView& e, V2 p, int sub, unsigned mask)
{
    int best = -1;
    V2 q[4];
    const int s = e.n_special > 0 ? special_index(e, p.y) : -1;
    if (s >= 0) {
        for (int i = e.sp_start[s], en = e.sp_start[s + 1]; i < en; i++) {
            const int c = e.sp_items[i];
            cell_quad(e, c, q);
            if (contains_quad(p, q)) {
                best = c;
                break;
            }
        }
    }
    const float fx = (p.x - e.gx0) * e.ginv, fy = (p.y - e.gy0) * e.ginv;
    if (!(fx >= 0.0f && fy >= 0.0f && fx < (float)e.gw && fy < (float)e.gh)) return best;
    const int g = (int)fy * e.gw + (int)fx;
    const int en = e.g_start[g + 1];
    for (int i0 = e.g_start[g]; i0 < en; i0 += kAttractLanes) {
        const int i = i0 + sub;
        int c = -1;
        bool hit = false;
        if (i < en) {
            c = e.g_items[i];
            if (best < 0 || c < best) {
                cell_quad(e, c, q);
                hit = contains_quad(p, q);
            }
        }
        const unsigned h = __ballot_sync(mask, hit) & mask;
        if (h) return __shfl_sync(mask, c, __ffs(h) - 1);
    }
    return best;
}

/* irm() of ecmg_geom.cuh */
__device__ __forceinline__ bool irm_group(const EcmView& e, V2 pos, const V2* path, int n, V2* out, bool* no_retract,
                                          int* edge, int cell, int sub, unsigned mask)
{
    V2 r;
    int ed;
    if (!retract(e, pos, &r, &ed, cell)) {
        *no_retract = true;
        return false;
    }
    *edge = ed;
    const V2 co = closest_on_segment(r, e.edge[ed].l0, e.edge[ed].r1);
    const float clr = len(r - co);
    const float rcs = clr * clr;
    const V2 goal = path[n - 1];
    if (len2(goal - r) < rcs) {
        *out = goal;
        return true;
    }
    bool success = false;
    int at = -1; /* the lane's last segment that gave a point */
    V2 point = mk(0.0f, 0.0f);
    for (int i = sub; i < n - 1; i += kAttractLanes) {
        const V2 p1 = path[i] - r;
        const V2 p2 = path[i + 1] - r;
        V2 a, b;
        float t1, t2;
        if (!irm_segment(p1, p2, r, rcs, &a, &b, &t1, &t2)) continue;
        success = true;
        float maxT = -1.0f;
        if (t1 >= 0.0f && t1 <= 1.0f) {
            point = a;
            maxT = t1;
            at = i;
        }
        if (t2 >= 0.0f && t2 <= 1.0f && t2 > maxT) {
            point = b;
            at = i;
        }
    }
    int last = at;
#pragma unroll
    for (int o = kAttractLanes / 2; o; o >>= 1) last = max(last, __shfl_xor_sync(mask, last, o));
    const unsigned owner = __ballot_sync(mask, at >= 0 && at == last) & mask;
    if (owner) {
        const int w = __ffs(owner) - 1;
        out->x = __shfl_sync(mask, point.x, w);
        out->y = __shfl_sync(mask, point.y, w);
    }
    return __any_sync(mask, success);
}

__global__ void __launch_bounds__(128) k_attract_group(TickArgs a)
{
    const int n = a.counters[C_NSORTED];
    const int lane = threadIdx.x & 31, sub = lane & (kAttractLanes - 1);
    const unsigned mask = ((1u << kAttractLanes) - 1u) << (lane & ~(kAttractLanes - 1));
    const int per = blockDim.x / kAttractLanes;
    for (int t = blockIdx.x * per + threadIdx.x / kAttractLanes; t < n; t += gridDim.x * per)
        attract_agent(
            a, t, sub == 0, [&](const EcmView& e, V2 p) { return locate_group(e, p, sub, mask); },
            [&](const EcmView& e, V2 p, const V2* path, int np, V2* out, bool* nr, int* ed, int cell) {
                return irm_group(e, p, path, np, out, nr, ed, cell, sub, mask);
            });
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < a.total_buckets; c += gridDim.x * blockDim.x)
        a.cell_count[c] = 0;
}

/* UpdateAttractionPointSystem + ApplySteeringForce for every agent.  Bound by
   its dependent loads; 8 resident blocks at 64 registers (24 bytes of spills)
   against 6 at 80: 158 and 191 us beside the search at a million agents, no
   difference at 25,000; 10 blocks spill 92 bytes and take 247 */
__global__ void __launch_bounds__(128, 8) k_attract(TickArgs a)
{
    const int n = a.counters[C_NSORTED];
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) attract_tick(a, t);
    /* the bucket counts are cleared for the next tick's binning */
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < a.total_buckets; c += gridDim.x * blockDim.x)
        a.cell_count[c] = 0;
}

/* agents whose re-plan is still being computed on the host when the tick
   starts: the tick's attraction and ORCA kernels skip them */
__global__ void k_mark_pending(TickArgs a, const int* list, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        a.active[list[i]] |= kActivePending;
}

/* the skipped step of those agents, after the tick's kernels and the upload
   of their new paths: UpdateAttractionPointSystem with the new path, then
   ApplyObstacleAvoidanceForce and the integration on the tick's snapshot and
   neighbour lists (still in place until the next tick's binning) -- the
   same functions on the same inputs as the tick's own kernels.  One warp per
   agent: a few agents, whose serial step would be what the tick waits for */
template <int K, bool FULL>
__global__ void __launch_bounds__(32) k_fixup(TickArgs a, const int* list)
{
    __shared__ __align__(16) float4 sm[kGroupRow<K>];
    const int slot = list[blockIdx.x], lane = threadIdx.x;
    if (!(a.active[slot] & kActivePending)) return;
    __syncwarp();
    const int t = a.cell_start[a.slot_bucket[slot]] + a.slot_rank[slot];
    if (lane == 0) {
        a.active[slot] = 1;
        attract_tick(a, t);
    }
    __syncwarp();
    GroupCounts gc;
    orca_group<K, 32, FULL>(a, t, true, sm, gc);
    if (lane == 0) {
        if (gc.lp3d) atomicAdd(&a.counters[C_LP3D], gc.lp3d);
        if (FULL && gc.proposed) atomicAdd(&a.counters[C_PROPOSED], gc.proposed);
        if (FULL && gc.accepted) atomicAdd(&a.counters[C_ACCEPTED], gc.accepted);
    }
}

/* proposal features of every grid-order agent (zeros for agents destroyed
   this tick): 16 neighbours x (relative position / neighbour distance,
   relative velocity / 2, radius sum), preferred velocity / LP radius */
__global__ void __launch_bounds__(128) k_features(TickArgs a)
{
    const int n = a.counters[C_NSORTED];
    __nv_bfloat16* F = (__nv_bfloat16*)a.feat;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        float f[kMlpIn];
#pragma unroll
        for (int i = 0; i < kMlpIn; i++) f[i] = 0.0f;
        const int slot = a.s_slot[t];
        if (a.active[slot]) {
            const float4 rec = a.s_rec[t];
            const V2 pos = a.s_pos[t], vel = mk(rec.x, rec.y);
            const float clr = rec.z, speed = rec.w;
            const float maxSpeed = a.max_speed > 0.0f ? a.max_speed : speed;
            const int ncnt = a.ncnt[t];
            const int* nbr = a.nbr + (size_t)t * a.k;
            const float inv_r = 1.0f / a.rnb;
#pragma unroll
            for (int q = 0; q < kMlpNbrs; q++) {
                if (q < ncnt) {
                    int j = nbr[q];
                    const float4 rj = a.s_rec[j];
                    V2 pj = a.s_pos[j], vj = mk(rj.x, rj.y);
                    f[5 * q + 0] = (pj.x - pos.x) * inv_r;
                    f[5 * q + 1] = (pj.y - pos.y) * inv_r;
                    f[5 * q + 2] = (vel.x - vj.x) * 0.5f;
                    f[5 * q + 3] = (vel.y - vj.y) * 0.5f;
                    f[5 * q + 4] = rj.z + clr;
                }
            }
            V2 pv = a.pref_vel[slot];
            float im = maxSpeed > 0.0f ? 1.0f / maxSpeed : 0.0f;
            f[5 * kMlpNbrs] = pv.x * im;
            f[5 * kMlpNbrs + 1] = pv.y * im;
        }
        uint4* row = reinterpret_cast<uint4*>(F + (size_t)t * kMlpIn);
#pragma unroll
        for (int c = 0; c < kMlpIn / 8; c++) {
            __nv_bfloat162 h0 = __floats2bfloat162_rn(f[8 * c + 0], f[8 * c + 1]);
            __nv_bfloat162 h1 = __floats2bfloat162_rn(f[8 * c + 2], f[8 * c + 3]);
            __nv_bfloat162 h2 = __floats2bfloat162_rn(f[8 * c + 4], f[8 * c + 5]);
            __nv_bfloat162 h3 = __floats2bfloat162_rn(f[8 * c + 6], f[8 * c + 7]);
            uint4 u;
            u.x = *reinterpret_cast<unsigned*>(&h0);
            u.y = *reinterpret_cast<unsigned*>(&h1);
            u.z = *reinterpret_cast<unsigned*>(&h2);
            u.w = *reinterpret_cast<unsigned*>(&h3);
            row[c] = u;
        }
    }
}

/* persistent kernel: a warp takes `tile` consecutive grid-order agents per
   work grab (one atomic per grab) and runs them 32 at a time */
template <int K, bool FULL>
__global__ void __launch_bounds__(256, (K <= 16) ? 4 : 1) k_agents(TickArgs a)
{
    const int n = a.counters[C_NSORTED];
    const int lane = threadIdx.x & 31;
    while (true) {
        int base = 0;
        if (lane == 0) base = atomicAdd(&a.counters[C_WORK], a.tile);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= n) break;
        for (int o = 0; o < a.tile; o += 32) {
            int t = base + o + lane;
            if (t < n) orca_tick<K, FULL>(a, t);
        }
    }
}

/* G lanes per agent (orca_group.cuh): a warp steps 32 / G consecutive
   grid-order agents.  Bound by an agent's chain of half-planes and LP steps;
   the figures by G and agent count are at lanes_of in ctx.cu */
template <int K, int G, bool FULL>
__global__ void __launch_bounds__(32 * kGroupWarps, K <= 16 ? 7 : 4) k_agents_group(TickArgs a)
{
    constexpr int A = 32 / G; /* agents per warp */
    __shared__ __align__(16) float4 sm[kGroupWarps][A][kGroupRow<K>];
    const int n = a.counters[C_NSORTED];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    GroupCounts gc;
    for (int t0 = (blockIdx.x * kGroupWarps + w) * A; t0 < n; t0 += gridDim.x * kGroupWarps * A) {
        const int t = t0 + lane / G;
        orca_group<K, G, FULL>(a, min(t, n - 1), t < n, sm[w][lane / G], gc);
    }
    const int lp3d = __reduce_add_sync(kFull, gc.lp3d);
    if (lane == 0 && lp3d) atomicAdd(&a.counters[C_LP3D], lp3d);
    if (FULL && (a.cls || a.cls_slot)) {
        const int pr = __reduce_add_sync(kFull, gc.proposed), ac = __reduce_add_sync(kFull, gc.accepted);
        if (lane == 0 && pr) atomicAdd(&a.counters[C_PROPOSED], pr);
        if (lane == 0 && ac) atomicAdd(&a.counters[C_ACCEPTED], ac);
    }
}

/* the stand-alone query: lists of slots by slot */
template <int K, bool CROWDS>
__global__ void __launch_bounds__(32 * kNbrWarps, K <= 16 ? 8 : 4)
    k_knn(const V2* s_pos, const int* s_slot, const int* cell_start, AgentGrid g, int k, float r2, const int* counters,
          int* out_ids, int* out_cnt)
{
    __shared__ KnnSm<K> sm[kNbrWarps];
    wait_for_previous();
    const int n = counters[C_NSORTED];
    const int lane = threadIdx.x & 31;
    for (int base = (blockIdx.x * kNbrWarps + (threadIdx.x >> 5)) * 32; base < n; base += gridDim.x * kNbrWarps * 32) {
        const int t = min(base + lane, n - 1);
        const bool in = base + lane < n;
        const int slot = s_slot[t];
        int* o = out_ids + (size_t)slot * k;
        const int c = knn_list<K, true, CROWDS>(sm[threadIdx.x >> 5], in, k, s_pos[t], r2, s_pos, s_slot, cell_start, g, o);
        if (in) out_cnt[slot] = c;
    }
}

/* ---------------------------------------------------------------------- */
static int grid_for(int n, int block, int sms, int per_sm)
{
    int g = (n + block - 1) / block;
    int cap = sms * per_sm;
    return g < 1 ? 1 : (g > cap ? cap : g);
}

/* a launch with a given split of an SM's memory between L1 and shared memory
   (per cent of shared memory).  Two kernels are resident on an SM together
   only under one split: with the defaults -- the attraction kernel uses no
   shared memory -- the search beside it waited for it to end on every SM that
   it had reached (25,000 agents: 45 us from their common start, now 23). */
template <class Kern>
static cudaError_t launch_split(Kern kern, int blocks, int threads, int split, cudaStream_t s, const TickArgs& t)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    at.val.sharedMemCarveout = split;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, t);
}

cudaError_t launch_tick(const BinArgs& b, const TickArgs& t, int max_slots, int block, int sms,
                        cudaStream_t s, cudaStream_t s2, cudaEvent_t ev_fork, cudaEvent_t ev_join,
                        const cudaEvent_t* ev, ProposeFn propose, void* propose_user,
                        HookFn after_attract, void* after_attract_user, const KdArgs* kd)
{
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(s, &cap);
    const unsigned evflags = cap == cudaStreamCaptureStatusActive ? cudaEventRecordExternal : 0u;
    int gb = grid_for(max_slots, 256, sms, 8);
    cudaError_t e = launch_bin(b, max_slots, gb, s);
    if (e != cudaSuccess) return e;
    /* external event nodes when captured, so that the kernel can be timed */
    if (ev) cudaEventRecordWithFlags(ev[0], s, evflags);
    if (block != 64 && block != 128 && block != 256) block = 128;
    int gk = grid_for(max_slots, 128, sms, 16);
    int per_sm = 1;
    /* the attraction kernel (second stream) and the neighbour search are
       independent: they run side by side and join before the features /
       per-agent kernels */
    e = cudaEventRecord(ev_fork, s);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s2, ev_fork, 0);
    if (e != cudaSuccess) return e;
    /* one split for both: enough shared memory for the search's blocks that an
       SM gets, the rest L1 for both (tick at 100,000 agents 218 us at 50 %, 220
       at 75, 221 at 30; at a million 802, 791 and 831) */
    const int split = max_slots <= sms * 2048 ? 50 : 75;
    int ao = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ao, k_attract, 128, 0);
    /* blocks for the agents and for the bucket counts that these kernels clear */
    const int gc = blocks_of_buckets(t.total_buckets, 128);
    const int ga = std::max(gk, gc);
    if (t.attract_lanes)
        e = launch_split(k_attract_group, std::max(grid_for(max_slots, 128 / kAttractLanes, sms, 32), gc), 128, split, s2, t);
    else e = launch_split(k_attract, ao > 0 ? std::min(ga, sms * ao) : ga, 128, split, s2, t); /* one wave, grid-stride */
    if (e != cudaSuccess) return e;
    if (ev) cudaEventRecordWithFlags(ev[1], s2, evflags);
    /* the per-agent kernel waits for the attraction kernel, not for the
       copies of its lists behind it (joined at the end) */
    e = cudaEventRecord(ev_join, s2);
    if (e != cudaSuccess) return e;
    if (after_attract) {
        e = after_attract(after_attract_user, s2, evflags);
        if (e != cudaSuccess) return e;
    }
    if (kd) {
        /* the reference's kd-tree: build and per-member query beside the
           attraction kernel, the cache composition after it */
        e = kd_build_and_query(*kd, s, sms);
        if (e != cudaSuccess) return e;
    } else {
        /* one resident wave of the persistent search at most */
        auto go = [&](auto kern) {
            int pn = 1;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&pn, kern, 32 * kNbrWarps, 0);
            e = launch_split(kern, grid_for(max_slots, 32 * kNbrWarps, sms, std::max(1, std::min(pn, t.knn_blocks))),
                             32 * kNbrWarps, split, s, t);
        };
        const bool crowds = max_slots > kCrowdSlots;
        if (t.k <= 8) crowds ? go(k_neighbors<8, true>) : go(k_neighbors<8, false>);
        else if (t.k <= 16) crowds ? go(k_neighbors<16, true>) : go(k_neighbors<16, false>);
        else crowds ? go(k_neighbors<32, true>) : go(k_neighbors<32, false>);
        if (e != cudaSuccess) return e;
    }
    if (ev && !kd) cudaEventRecordWithFlags(ev[2], s, evflags);
    e = cudaStreamWaitEvent(s, ev_join, 0);
    if (e != cudaSuccess) return e;
    if (kd) {
        e = kd_finish(*kd, s, sms);
        if (e != cudaSuccess) return e;
        if (ev) cudaEventRecordWithFlags(ev[2], s, evflags);
    }
    if (t.feat) {
        k_features<<<gk, 128, 0, s>>>(t);
        if (propose) {
            cudaError_t e2 = propose(propose_user, s);
            if (e2 != cudaSuccess) return e2;
        }
    }
    if (ev && t.feat) cudaEventRecordWithFlags(ev[3], s, evflags);
    if (t.lanes > 1) {
        const bool full = t.cls || t.cls_slot || t.label || t.rec_cnt || t.lp3d_fp64;
        auto go = [&](auto kern) {
            /* one agent set per warp, so that the block scheduler evens out
               their unequal work; a slot range far above the agents in it
               takes the capped grid more than once */
            kern<<<grid_for(max_slots, kGroupWarps * 32 / t.lanes, sms, 64), 32 * kGroupWarps, 0, s>>>(t);
        };
        auto by_k = [&](auto lanes) {
            constexpr int G = decltype(lanes)::value;
            if (t.k <= 8) full ? go(k_agents_group<8, G, true>) : go(k_agents_group<8, G, false>);
            else if (t.k <= 16) full ? go(k_agents_group<16, G, true>) : go(k_agents_group<16, G, false>);
            else full ? go(k_agents_group<32, G, true>) : go(k_agents_group<32, G, false>);
        };
        if (t.lanes == 4) by_k(std::integral_constant<int, 4>());
        else if (t.lanes == 8) by_k(std::integral_constant<int, 8>());
        else if (t.lanes == 16) by_k(std::integral_constant<int, 16>());
        else by_k(std::integral_constant<int, 32>());
    } else {
        /* persistent grid: the resident blocks per SM, divided by occ_div
           (fewer resident warps leave each more L1 for its local arrays) */
        const int div = t.occ_div > 1 ? t.occ_div : 1;
        const bool full = t.cls || t.cls_slot || t.label || t.rec_cnt || t.lp3d_fp64 || kd;
        auto go = [&](auto kern) {
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, block, 0);
            kern<<<sms * (per_sm / div > 0 ? per_sm / div : 1), block, 0, s>>>(t);
        };
        if (t.k <= 8) full ? go(k_agents<8, true>) : go(k_agents<8, false>);
        else if (t.k <= 16) full ? go(k_agents<16, true>) : go(k_agents<16, false>);
        else full ? go(k_agents<32, true>) : go(k_agents<32, false>);
    }
    if (ev) cudaEventRecordWithFlags(ev[4], s, evflags);
    e = cudaEventRecord(ev_fork, s2);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s, ev_fork, 0);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

cudaError_t launch_mark_pending(const TickArgs& t, const int* list, int n, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    k_mark_pending<<<(n + 127) / 128, 128, 0, s>>>(t, list, n);
    return cudaGetLastError();
}

__global__ void k_mirror(const float4* __restrict__ pos, const float4* __restrict__ vel, float4* h_pos,
                         float4* h_vel, int n2, const V2* __restrict__ pos_tail, const V2* __restrict__ vel_tail,
                         V2* h_pos_tail, V2* h_vel_tail)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n2; i += gridDim.x * blockDim.x) {
        const float4 p = pos[i], v = vel[i];
        h_pos[i] = p;
        h_vel[i] = v;
    }
    if (pos_tail && blockIdx.x == 0 && threadIdx.x == 0) {
        *h_pos_tail = *pos_tail;
        *h_vel_tail = *vel_tail;
    }
}

cudaError_t launch_mirror(const V2* pos, const V2* vel, V2* h_pos, V2* h_vel, int n, int sms, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    const int n2 = n / 2; /* pairs of slots as 16-byte words (the arrays are 256-byte aligned) */
    const bool odd = n & 1;
    const int g = std::max(1, std::min((n2 + 255) / 256, sms * 4));
    k_mirror<<<g, 256, 0, s>>>((const float4*)pos, (const float4*)vel, (float4*)h_pos, (float4*)h_vel, n2,
                               odd ? pos + n - 1 : nullptr, odd ? vel + n - 1 : nullptr, h_pos + n - 1, h_vel + n - 1);
    return cudaGetLastError();
}

cudaError_t launch_fixup(const TickArgs& t, const int* list, int n, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    const bool full = t.cls || t.cls_slot || t.label || t.rec_cnt || t.lp3d_fp64;
    if (t.k <= 8) full ? k_fixup<8, true><<<n, 32, 0, s>>>(t, list) : k_fixup<8, false><<<n, 32, 0, s>>>(t, list);
    else if (t.k <= 16) full ? k_fixup<16, true><<<n, 32, 0, s>>>(t, list) : k_fixup<16, false><<<n, 32, 0, s>>>(t, list);
    else full ? k_fixup<32, true><<<n, 32, 0, s>>>(t, list) : k_fixup<32, false><<<n, 32, 0, s>>>(t, list);
    return cudaGetLastError();
}

cudaError_t launch_knn(const V2* pos, const unsigned char* active, int n, int k, float r, AgentGrid g,
                       int* key, int* rank, int* cell_count, int* cell_start, int* s_slot, V2* s_pos,
                       int* scan_tmp, int* out_ids, int* out_cnt, cudaStream_t s)
{
    /* the counters live behind the bucket counts: [nb+1 .. nb+1+kCounters) */
    int nb = g.ncells + 1;
    int* counters = cell_count + nb + 1;
    /* the slot range is passed by value: the query queues no host-to-device copy */
    BinArgs b{};
    b.n_fixed = n;
    b.pos = pos;
    b.active = active;
    b.key = key;
    b.rank = rank;
    b.cell_count = cell_count;
    b.s_slot = s_slot;
    b.s_pos = s_pos;
    b.cell_start = cell_start;
    b.counters = counters;
    b.grid = g;
    b.total_buckets = g.ncells;
    b.block_sums = scan_tmp;
    b.out_cnt = out_cnt; /* zero for the inactive */
    cudaError_t e = cudaSuccess;
    if (!bins_small(b, n)) e = cudaMemsetAsync(cell_count, 0, sizeof(int) * (size_t)nb, s);
    if (e == cudaSuccess) e = launch_bin(b, n, (n + 255) / 256, s);
    if (e != cudaSuccess) return e;
    const int ga = (n + 32 * kNbrWarps - 1) / (32 * kNbrWarps);
    const float r2 = r * r;
    auto query = [&](auto kern) {
        return launch_ahead(kern, ga, 32 * kNbrWarps, 0, s, s_pos, s_slot, cell_start, g, k, r2, counters, out_ids, out_cnt);
    };
    if (n > kCrowdPoints) return k <= 8 ? query(k_knn<8, true>) : (k <= 16 ? query(k_knn<16, true>) : query(k_knn<32, true>));
    return k <= 8 ? query(k_knn<8, false>) : (k <= 16 ? query(k_knn<16, false>) : query(k_knn<32, false>));
}

}  // namespace ecmg
