/*
 * kdtree.cu -- the reference's kd-tree neighbour query on the device
 * (neighbour mode ECMG_NEIGHBORS_KDTREE), results identical to
 * KDTree::Construct / KDTree::KNearestAgents_R (ECMAgentSimulator/
 * KDTree.cpp:22-202) with ORCA's neighbour cache (ORCA.h:87,100) carried from
 * agent to agent and from tick to tick.
 *
 * Build.  ConstructRecursive sorts each subtree's agents on x (even depth) or
 * y (odd depth) and takes the element at mid = lo + (hi - 1 - lo) / 2.  Equal
 * coordinates keep the order of the level above (a stable sort; libstdc++'s
 * std::sort agrees on segments of up to 16 agents, where it is an insertion
 * sort).  That order is, for depth 0, (x, agent index); for the depths after
 * it (x, y, index) and (y, x, index).  So the build sorts the members once
 * into three lists, X0 = (x, index), X = (x, y, index), Y = (y, x, index), by
 * stable LSD radix passes, and then walks the levels: the list of the level's
 * axis is already sorted inside every segment, its element at mid is the node,
 * and the other list is partitioned stably into (left, node, right) with one
 * scan of left / right flags.  Segments are position ranges shared by both
 * lists.  O(N) work per level.
 *
 * Query.  One thread per member replays KNearestAgents_R with an explicit
 * stack.  The reference does not clear the cache between agents: slots that a
 * query does not overwrite keep the previous agent's entries, and entries
 * move between slots.  The thread therefore starts from the symbolic cache
 * (-1, -2, ..., -k) = "previous agent's slot q" and ends with a map: each
 * slot either an agent or a previous slot.  Maps compose associatively; the
 * composition over the querying agents in index order (members still active
 * after the attraction stage) folds 64 maps at a time, level by level, and the
 * lists that refer to an earlier one look it up -- the last agent's list is
 * the cache the next tick starts from.
 */
#include "ecmg_internal.h"
#include "launch_ahead.cuh"

#include <cfloat>

namespace ecmg {

namespace {

constexpr int kRsThreads = 256, kRsItems = 8, kRsTile = kRsThreads * kRsItems;
constexpr int kScanThreads = 256, kScanItems = 8, kScanTile = kScanThreads * kScanItems;
constexpr int kFold = 64;

__device__ __forceinline__ unsigned order_key(float f)
{
    unsigned u = __float_as_uint(f);
    if (u == 0x80000000u) u = 0u; /* -0 == +0 for operator< */
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

/* ---- exclusive scan (in place), T = int or unsigned long long ---------- */
template <typename T>
__device__ T block_excl_scan(T v, T* total)
{
    __shared__ T warp_sum[kScanThreads / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    T x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sum[w] = x;
    __syncthreads();
    if (w == 0) {
        T s = lane < kScanThreads / 32 ? warp_sum[lane] : (T)0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            T y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        if (lane < kScanThreads / 32) warp_sum[lane] = s;
    }
    __syncthreads();
    const T before = (w > 0 ? warp_sum[w - 1] : (T)0) + x - v;
    if (total) *total = warp_sum[kScanThreads / 32 - 1];
    __syncthreads();
    return before;
}

template <typename T>
__global__ void __launch_bounds__(kScanThreads) k_scan_reduce(const T* in, int n, T* sums)
{
    wait_for_previous();
    const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    T s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++)
        if (base + i < n) s += in[base + i];
    T tot;
    block_excl_scan<T>(s, &tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

/* one block of 1024 threads: exclusive scan of nb <= 8192 block sums */
template <typename T>
__global__ void __launch_bounds__(1024) k_scan_top(T* sums, int nb)
{
    wait_for_previous();
    __shared__ T ws[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    T v[8];
    T s = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int j = threadIdx.x * 8 + i;
        v[i] = j < nb ? sums[j] : (T)0;
        s += v[i];
    }
    T x = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    if (w == 0) {
        T t = ws[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            T y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        ws[lane] = t;
    }
    __syncthreads();
    T run = (w > 0 ? ws[w - 1] : (T)0) + x - s;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int j = threadIdx.x * 8 + i;
        if (j < nb) sums[j] = run;
        run += v[i];
    }
}

template <typename T>
__global__ void __launch_bounds__(kScanThreads) k_scan_down(T* data, int n, const T* sums)
{
    wait_for_previous();
    const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    T v[kScanItems];
    T s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        v[i] = base + i < n ? data[base + i] : (T)0;
        s += v[i];
    }
    T run = block_excl_scan<T>(s, nullptr) + sums[blockIdx.x];
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        if (base + i < n) data[base + i] = run;
        run += v[i];
    }
}

template <typename T>
cudaError_t scan_excl(T* data, int n, T* tmp, cudaStream_t s)
{
    const int nb = (n + kScanTile - 1) / kScanTile;
    if (nb < 1) return cudaSuccess;
    if (nb > 8192) return cudaErrorInvalidValue;
    launch_ahead(k_scan_reduce<T>, nb, kScanThreads, 0, s, data, n, tmp);
    launch_ahead(k_scan_top<T>, 1, 1024, 0, s, tmp, nb);
    launch_ahead(k_scan_down<T>, nb, kScanThreads, 0, s, data, n, tmp);
    return cudaGetLastError();
}

/* ---- stable LSD radix sort of (key, value) pairs, 8-bit digits ----------
   Tiles of 2,048 keys: a quarter of a million agents fill the GPU (with 4,096
   they were 62 blocks). */
__global__ void __launch_bounds__(kRsThreads) k_rs_hist(const unsigned* keys, const int* n_ptr,
                                                        int shift, int* hist)
{
    wait_for_previous();
    __shared__ int h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const int n = *n_ptr;
    const int base = blockIdx.x * kRsTile;
#pragma unroll
    for (int i = 0; i < kRsItems; i++) {
        const int idx = base + i * kRsThreads + threadIdx.x;
        if (idx < n) atomicAdd(&h[(keys[idx] >> shift) & 255u], 1);
    }
    __syncthreads();
    hist[blockIdx.x * 256 + threadIdx.x] = h[threadIdx.x];
}

/* hist [nblk][256] -> the keys of each digit in the tiles before each tile, in
   place, and the digits' totals: a warp per digit.  (One block over all
   digits took 9.6 us a pass at 123 tiles, as long as the scatter.) */
__global__ void __launch_bounds__(256) k_rs_scan(int* hist, int nblk, int* total)
{
    wait_for_previous();
    const int lane = threadIdx.x & 31, d = blockIdx.x * 8 + (threadIdx.x >> 5);
    int carry = 0;
    for (int b0 = 0; b0 < nblk; b0 += 128) {
        int v[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int b = b0 + q * 32 + lane;
            v[q] = b < nblk ? hist[b * 256 + d] : 0;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            int x = v[q];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            const int b = b0 + q * 32 + lane;
            if (b < nblk) hist[b * 256 + d] = carry + x - v[q];
            carry += __shfl_sync(0xffffffffu, x, 31);
        }
    }
    if (lane == 0) total[d] = carry;
}

/* elements of a tile are placed in tile order, round by round (256 per
   round, in thread order): rank among equal digits = warps before + lanes
   before, so the pass is stable */
__global__ void __launch_bounds__(kRsThreads) k_rs_scatter(const unsigned* kin, const int* vin,
                                                           unsigned* kout, int* vout,
                                                           const int* n_ptr, int shift,
                                                           const int* offs,
                                                           const int* total)
{
    wait_for_previous();
    __shared__ int base[256];
    __shared__ int wc[kRsThreads / 32][256];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int n = *n_ptr;
    const int t0 = blockIdx.x * kRsTile;
    if (t0 >= n) return;
    /* the keys of smaller digits, then those of this digit in earlier tiles */
    base[threadIdx.x] = block_excl_scan<int>(total[threadIdx.x], nullptr) + offs[blockIdx.x * 256 + threadIdx.x];
    unsigned keys[kRsItems];
    int vals[kRsItems];
#pragma unroll
    for (int r = 0; r < kRsItems; r++) {
        const int idx = t0 + r * kRsThreads + threadIdx.x;
        keys[r] = idx < n ? kin[idx] : 0u;
        vals[r] = idx < n ? vin[idx] : 0;
    }
#pragma unroll
    for (int r = 0; r < kRsItems; r++) {
#pragma unroll
        for (int q = 0; q < kRsThreads / 32; q++) wc[q][threadIdx.x] = 0;
        __syncthreads();
        const bool valid = t0 + r * kRsThreads + (int)threadIdx.x < n;
        const int d = valid ? (int)((keys[r] >> shift) & 255u) : 256 + lane;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const int rank = __popc(peers & ((1u << lane) - 1u));
        if (valid && rank == 0) wc[w][d] = __popc(peers);
        __syncthreads();
        {
            int run = base[threadIdx.x];
#pragma unroll
            for (int q = 0; q < kRsThreads / 32; q++) {
                const int c = wc[q][threadIdx.x];
                wc[q][threadIdx.x] = run;
                run += c;
            }
            base[threadIdx.x] = run;
        }
        __syncthreads();
        if (valid) {
            const int pos = wc[w][d] + rank;
            kout[pos] = keys[r];
            vout[pos] = vals[r];
        }
        __syncthreads();
    }
}

/* sorts keys[0, n) with their values; n is read on the device; the result
   ends in (keys, vals) after the four passes */
cudaError_t radix_sort(unsigned* keys, int* vals, unsigned* ktmp, int* vtmp, const int* n_ptr, int cap, int* hist,
                       cudaStream_t s)
{
    const int nblk = (cap + kRsTile - 1) / kRsTile;
    unsigned* ka = keys;
    int* va = vals;
    unsigned* kb = ktmp;
    int* vb = vtmp;
    for (int shift = 0; shift < 32; shift += 8) {
        launch_ahead(k_rs_hist, nblk, kRsThreads, 0, s, ka, n_ptr, shift, hist);
        launch_ahead(k_rs_scan, 32, 256, 0, s, hist, nblk, hist + nblk * 256);
        launch_ahead(k_rs_scatter, nblk, kRsThreads, 0, s, ka, va, kb, vb, n_ptr, shift, hist, hist + nblk * 256);
        unsigned* tk = ka; ka = kb; kb = tk;
        int* tv = va; va = vb; vb = tv;
    }
    return cudaGetLastError();
}

/* ---- members, keys and lists ------------------------------------------- */
__global__ void k_kd_mark(KdArgs a)
{
    wait_for_previous();
    const int n = a.counters[C_NSORTED];
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int slot = a.s_slot[t];
        a.mark[slot] = 1;
        a.gidx[slot] = t;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.n_dev[0] = n;
        /* KDTree.cpp:47: ceil(log2(size + 1) - 1) = bit length of size - 1 */
        a.n_dev[1] = n > 0 ? 31 - __clz(n) : -1;
    }
}

__global__ void k_kd_flag(KdArgs a, int* flags)
{
    wait_for_previous();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.max_slots; i += gridDim.x * blockDim.x)
        flags[i] = a.mark[i];
}

__global__ void k_kd_compact(KdArgs a, const int* flags, int* ids)
{
    wait_for_previous();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.max_slots; i += gridDim.x * blockDim.x)
        if (a.mark[i]) ids[flags[i]] = i;
}

__global__ void k_kd_keys(KdArgs a, const int* ids, int axis, unsigned* keys, int* vals)
{
    wait_for_previous();
    const int n = a.n_dev[0];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int id = ids[i];
        const V2 p = a.pos[id];
        keys[i] = order_key(axis ? p.y : p.x);
        vals[i] = id;
    }
}

__global__ void k_kd_seg_init(KdArgs a)
{
    wait_for_previous();
    const int n = a.n_dev[0];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.cap; i += gridDim.x * blockDim.x) {
        a.seg_lo[i] = 0;
        a.seg_hi[i] = i < n ? n : 0;
        a.seg_node[i] = 0;
    }
}

/* ---- one level of ConstructRecursive over the whole lists ---------------- */
__global__ void k_kd_side(KdArgs a, const int* A)
{
    wait_for_previous();
    const int n = a.n_dev[0];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int lo = a.seg_lo[i], hi = a.seg_hi[i];
        if (lo >= hi) continue;
        const int mid = lo + (hi - 1 - lo) / 2;
        const int id = A[i];
        a.side[id] = i < mid ? 0 : (i == mid ? 1 : 2);
        if (i == mid) a.tree[a.seg_node[i]] = id;
    }
}

/* left | right << 32 of the positions first, first + step, ... of list B: the
   loads of all of them in flight together */
__device__ __forceinline__ void kd_flags(const KdArgs& a, const int* B, int first, int step, int n,
                                         unsigned long long (&f)[kScanItems])
{
    int id[kScanItems];
#pragma unroll
    for (int q = 0; q < kScanItems; q++) {
        const int i = first + q * step;
        id[q] = -1;
        if (i < n) {
            const int lo = a.seg_lo[i], hi = a.seg_hi[i], b = B[i];
            id[q] = lo < hi ? b : -1;
        }
    }
#pragma unroll
    for (int q = 0; q < kScanItems; q++) {
        const int s = id[q] >= 0 ? a.side[id[q]] : 1;
        f[q] = (s == 0 ? 1ull : 0ull) | (s == 2 ? (1ull << 32) : 0ull);
    }
}

__global__ void __launch_bounds__(kScanThreads) k_kd_count(KdArgs a, const int* B)
{
    wait_for_previous();
    const int n = a.n_dev[0];
    const int base = blockIdx.x * kScanTile + threadIdx.x;
    unsigned long long f[kScanItems], s = 0;
    kd_flags(a, B, base, kScanThreads, n, f);
#pragma unroll
    for (int i = 0; i < kScanItems; i++) s += f[i];
    unsigned long long tot;
    block_excl_scan<unsigned long long>(s, &tot);
    if (threadIdx.x == 0) a.scan_tmp64[blockIdx.x] = tot;
}

/* exclusive left / right counts of every position (the tiles' sums scanned) */
__global__ void __launch_bounds__(kScanThreads) k_kd_prefix(KdArgs a, const int* B)
{
    wait_for_previous();
    const int n = a.n_dev[0];
    const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    unsigned long long v[kScanItems], s = 0;
    kd_flags(a, B, base, 1, n, v);
#pragma unroll
    for (int i = 0; i < kScanItems; i++) s += v[i];
    unsigned long long run = block_excl_scan<unsigned long long>(s, nullptr) + a.scan_tmp64[blockIdx.x];
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        if (base + i < n) a.flags[base + i] = run;
        run += v[i];
    }
}

/* stable partition of B's segments into (left, node, right); update_seg
   also moves every position to its child segment (after the last use of
   the level's segments) */
__global__ void k_kd_partition(KdArgs a, const int* B, int* Bout, int update_seg)
{
    wait_for_previous();
    const int n = a.n_dev[0];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int lo = a.seg_lo[i], hi = a.seg_hi[i];
        if (lo >= hi) {
            Bout[i] = B[i];
            continue;
        }
        const int mid = lo + (hi - 1 - lo) / 2;
        const unsigned long long f = a.flags[i], f0 = a.flags[lo];
        const int id = B[i];
        const int s = a.side[id];
        int pos;
        if (s == 0) pos = lo + (int)((unsigned)f - (unsigned)f0);
        else if (s == 1) pos = mid;
        else pos = mid + 1 + (int)((unsigned)(f >> 32) - (unsigned)(f0 >> 32));
        Bout[pos] = id;
        if (!update_seg) continue;
        const int node = a.seg_node[i];
        if (i < mid) {
            a.seg_hi[i] = mid;
            a.seg_node[i] = 2 * node + 1;
        } else if (i > mid) {
            a.seg_lo[i] = mid + 1;
            a.seg_node[i] = 2 * node + 2;
        } else {
            a.seg_lo[i] = hi;
        }
    }
}

cudaError_t kd_partition(const KdArgs& a, const int* B, int* Bout, int update_seg, int gc, cudaStream_t s)
{
    const int nb = (a.cap + kScanTile - 1) / kScanTile;
    if (nb > 8192) return cudaErrorInvalidValue;
    launch_ahead(k_kd_count, nb, kScanThreads, 0, s, a, B);
    launch_ahead(k_scan_top<unsigned long long>, 1, 1024, 0, s, a.scan_tmp64, nb);
    launch_ahead(k_kd_prefix, nb, kScanThreads, 0, s, a, B);
    launch_ahead(k_kd_partition, gc, 256, 0, s, a, B, Bout, update_seg);
    return cudaGetLastError();
}

/* ---- all remaining levels of one segment of up to kKdSmall members, by one
   block in shared memory.  A level over the whole lists is six launches bound
   by their latency (29 us each level at 250,000 agents); a segment of 4,096
   has as many levels left as the ones above it have, and they cost it a few
   block scans each.  Members are numbered by their place in the segment's X
   list. */
constexpr int kKdSmall = 4096, kSmallThreads = 1024, kSmallPer = kKdSmall / kSmallThreads;
struct KdSmallSm {
    int id[kKdSmall];             /* slot of each member */
    unsigned count[kKdSmall + 1]; /* left | right << 16 before each position */
    unsigned short list[3][kKdSmall]; /* X, Y and the list being written */
    unsigned short lo[kKdSmall], hi[kKdSmall], node[kKdSmall]; /* of each position; node: place in its level */
    unsigned char side[kKdSmall];
    unsigned warp[32];
};

__global__ void __launch_bounds__(kSmallThreads) k_kd_small(KdArgs a, const int* X, const int* Y, int top, int* place)
{
    wait_for_previous();
    extern __shared__ __align__(16) unsigned char raw[];
    KdSmallSm& m = *reinterpret_cast<KdSmallSm*>(raw);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    /* the segment: the block's path of left / right turns from the root */
    int lo0 = 0, hi0 = a.n_dev[0];
    for (int b = top - 1; b >= 0 && lo0 < hi0; b--) {
        const int mid = lo0 + (hi0 - 1 - lo0) / 2;
        if ((blockIdx.x >> b) & 1) lo0 = mid + 1;
        else hi0 = mid;
    }
    const int n = hi0 - lo0;
    if (n <= 0) return;
    for (int i = tid; i < n; i += kSmallThreads) {
        const int id = X[lo0 + i];
        m.id[i] = id;
        m.list[0][i] = (unsigned short)i;
        m.lo[i] = 0;
        m.hi[i] = (unsigned short)n;
        m.node[i] = 0;
        place[id] = i;
    }
    __syncthreads();
    for (int i = tid; i < n; i += kSmallThreads) m.list[1][i] = (unsigned short)place[Y[lo0 + i]];
    __syncthreads();
    int lx = 0, ly = 1, spare = 2;
    for (int lv = top; lv < a.levels; lv++) {
        const bool on_y = (lv & 1) != 0;
        const unsigned short* A = m.list[on_y ? ly : lx];
        const unsigned short* B = m.list[on_y ? lx : ly];
        unsigned short* out = m.list[spare];
        const int depth = lv - top;
        bool any = false;
        for (int i = tid; i < n; i += kSmallThreads) {
            const int lo = m.lo[i], hi = m.hi[i];
            if (lo >= hi) continue;
            any = true;
            const int mid = lo + (hi - 1 - lo) / 2;
            const int q = A[i];
            m.side[q] = i < mid ? 0 : (i == mid ? 1 : 2);
            /* heap index: node `place` of depth lv under the segment's root */
            if (i == mid) a.tree[((((1 << top) + (int)blockIdx.x) << depth) - 1) + m.node[i]] = m.id[q];
        }
        if (!__syncthreads_or(any)) return;
        /* exclusive left / right counts over the segment's positions */
        unsigned v[kSmallPer], sum = 0;
#pragma unroll
        for (int r = 0; r < kSmallPer; r++) {
            const int i = tid * kSmallPer + r;
            v[r] = 0;
            if (i < n && m.lo[i] < m.hi[i]) {
                const int sd = m.side[B[i]];
                v[r] = (sd == 0 ? 1u : 0u) | (sd == 2 ? 0x10000u : 0u);
            }
            sum += v[r];
        }
        unsigned x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) m.warp[w] = x;
        __syncthreads();
        if (w == 0) {
            unsigned y = m.warp[lane];
            const unsigned own = y;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned z = __shfl_up_sync(0xffffffffu, y, o);
                if (lane >= o) y += z;
            }
            m.warp[lane] = y - own;
        }
        __syncthreads();
        unsigned run = m.warp[w] + x - sum;
#pragma unroll
        for (int r = 0; r < kSmallPer; r++) {
            m.count[tid * kSmallPer + r] = run;
            run += v[r];
        }
        __syncthreads();
        for (int i = tid; i < n; i += kSmallThreads) {
            const int lo = m.lo[i], hi = m.hi[i];
            const int q = B[i];
            int pos = i;
            if (lo < hi) {
                const int mid = lo + (hi - 1 - lo) / 2;
                const unsigned f = m.count[i], f0 = m.count[lo];
                const int sd = m.side[q];
                if (sd == 0) pos = lo + (int)((f & 0xffffu) - (f0 & 0xffffu));
                else if (sd == 1) pos = mid;
                else pos = mid + 1 + (int)((f >> 16) - (f0 >> 16));
                if (i < mid) {
                    m.hi[i] = (unsigned short)mid;
                    m.node[i] = (unsigned short)(2 * m.node[i]);
                } else if (i > mid) {
                    m.lo[i] = (unsigned short)(mid + 1);
                    m.node[i] = (unsigned short)(2 * m.node[i] + 1);
                } else {
                    m.lo[i] = (unsigned short)hi;
                }
            }
            out[pos] = (unsigned short)q;
        }
        __syncthreads();
        const int freed = on_y ? lx : ly;
        if (on_y) lx = spare;
        else ly = spare;
        spare = freed;
    }
}

/* position and grid index of each node's agent (-1: none) in tree order: one
   load per visit in the query */
__global__ void k_kd_tree_pos(KdArgs a)
{
    wait_for_previous();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.tree_cap; i += gridDim.x * blockDim.x) {
        const int id = a.tree[i];
        const V2 p = id >= 0 ? a.pos[id] : mk(0.0f, 0.0f);
        a.tree_pos[i] = make_float4(p.x, p.y, __int_as_float(id >= 0 ? a.gidx[id] : -1), 0.0f);
    }
}

/* ---- KNearestAgents_R (KDTree.cpp:98-202) with a symbolic cache ----------
   A lane walks down the near children and keeps, by depth, each far child's
   split distance and a lower bound of its region's distance (the far child is
   the sibling of the path's node at that depth); one visit per lane and round, the lanes together (left
   to itself a lane that goes on down never meets the others again: 5 of 32
   lanes active).  The lists are columns in shared memory: their positions are
   written by index.  Bound by issue and divergence: about 115 rounds a warp
   for about 50 visits an agent, an update in nearly every round. */
constexpr int kQueryWarps = 4;
template <int K>
__global__ void __launch_bounds__(32 * kQueryWarps, K <= 16 ? 8 : 4) k_kd_query(KdArgs a, const int* members)
{
    wait_for_previous();
    __shared__ float s_nd[kQueryWarps][K][33];
    __shared__ int s_ni[kQueryWarps][K][33];
    extern __shared__ float2 s_far[]; /* [warp][depth][lane]: distance to the split line, bounds (two upper halves) */
    const int n = a.n_dev[0];
    const int max_depth = a.n_dev[1];
    const int k = a.k;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    float (*nd)[33] = s_nd[wp];
    int (*ni)[33] = s_ni[wp];
    float2* far = s_far + wp * a.levels * 32 + lane;
    for (int i0 = blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < n; i0 += gridDim.x * blockDim.x) {
        const int i = i0 + lane;
        const V2 target = a.pos[members[min(i, n - 1)]];
        for (int q = 0; q < k; q++) {
            ni[q][lane] = -(q + 1); /* the previous agent's slot q */
            nd[q][lane] = FLT_MAX;  /* Utility::MAX_FLOAT */
        }
        float first = FLT_MAX, last = FLT_MAX; /* nd[0], nd[k - 1] */
        int kfound = 0;
        unsigned todo = 0u; /* depths of the far children to come back to */
        int node = 0;
        /* the least |x - target.x|, |y - target.y| of the node's region known
           from the split lines above it */
        float bx = 0.0f, by = 0.0f;
        bool run = i < n;
        while (__any_sync(0xffffffffu, run)) {
            const int depth = 31 - __clz(node + 1);
            float4 rec = make_float4(0.0f, 0.0f, __int_as_float(-1), 0.0f);
            if (run && depth <= max_depth) rec = a.tree_pos[node];
            const int cur = __float_as_int(rec.z);
            /* Once k are found, visiting a node changes nothing unless
               d < nd[0]; every node of this subtree has d >= bx^2 + by^2
               (rounding is monotonic), so when that bound reaches nd[0] the
               whole subtree is visited by the reference without effect and
               is skipped here. */
            const bool visit = cur != -1 && !(kfound == k && bx * bx + by * by >= first);
            const float dx = rec.x - target.x, dy = rec.y - target.y;
            const float d = dx * dx + dy * dy;
            /* fill slot kfound, or replace slot 0; then the largest entry (the
               first one, if above d) moves to slot 0 and d takes its place */
            bool full = false;
            int li = 0; /* where d is going */
            if (visit) {
                if (kfound < k && d > 1e-4f) {
                    li = kfound++;
                    nd[li][lane] = d;
                    ni[li][lane] = cur;
                    if (li == 0) first = d;
                    if (li == k - 1) last = d;
                    full = kfound == k;
                } else {
                    kfound = k;
                    full = d < first && d > 1e-4f;
                }
            }
            if (full) {
                float lg = d;
                /* a replaced slot 0 is out of the search, a filled slot k - 1
                   is not above d */
                const int q0 = li == 0 ? 1 : 0;
                if (K <= 16) {
#pragma unroll
                    for (int q = 0; q < K; q++) {
                        const float x = q >= q0 && q < k ? nd[q][lane] : 0.0f;
                        if (x > lg) {
                            lg = x;
                            li = q;
                        }
                    }
                } else {
                    for (int q = q0; q < k; q++) {
                        const float x = nd[q][lane];
                        if (x > lg) {
                            lg = x;
                            li = q;
                        }
                    }
                }
                const int ln = lg > d ? ni[li][lane] : cur;
                nd[0][lane] = lg;
                ni[0][lane] = ln;
                first = lg;
                nd[li][lane] = d;
                ni[li][lane] = cur;
                if (li == 0) first = d;
                if (li == k - 1) last = d;
            }
            __syncwarp();
            if (visit) {
                const bool x_axis = (depth & 1) == 0;
                const float db = x_axis ? target.x - rec.x : target.y - rec.y;
                if (depth < max_depth) { /* a child on each side at most */
                    /* the far side: at least |db| away along the axis; the
                       bounds rounded down to 16 bits */
                    const float fx = x_axis ? fmaxf(bx, fabsf(db)) : bx, fy = x_axis ? by : fmaxf(by, fabsf(db));
                    far[(depth + 1) * 32] = make_float2(
                        db, __uint_as_float((__float_as_uint(fx) & 0xffff0000u) | (__float_as_uint(fy) >> 16)));
                    todo |= 2u << depth;
                }
                node = db < 0.0f ? 2 * node + 1 : 2 * node + 2; /* the near side: no new bound */
            } else if (run) {
                /* back to the last far child that is still within reach */
                run = false;
                while (todo && !run) {
                    const int at = 31 - __clz(todo);
                    todo ^= 1u << at;
                    const float2 e = far[at * 32];
                    if (e.x * e.x < last) {
                        run = true;
                        node = (((node + 1) >> (depth - at)) ^ 1) - 1;
                        bx = __uint_as_float(__float_as_uint(e.y) & 0xffff0000u);
                        by = __uint_as_float(__float_as_uint(e.y) << 16);
                    }
                }
            }
            __syncwarp();
        }
        /* rows of the warp's 32 agents, coalesced; a row with a reference to
           the list before it is open */
        bool open = false;
        for (int q = 0; q < k; q++) open |= ni[q][lane] < 0;
        if (i < n) {
            a.ncnt[i] = kfound;
            a.open[i] = open ? 1 : 0;
        }
        int* out = a.nbr + (size_t)i0 * k;
        const int cnt = min(32, n - i0) * k;
        for (int e = lane; e < cnt; e += 32) out[e] = ni[e % k][e / k];
        __syncwarp();
    }
}

/* ---- composition of the maps in slot order ------------------------------ */
__device__ __forceinline__ bool querying(const KdArgs& a, int s)
{
    return a.mark[s] && a.active[s];
}

/* rows of level 0 (slots) in use, and of the levels above it: a row of level
   l + 1 is the composition of kFold rows of level l */
__device__ __forceinline__ int fold_rows(const KdArgs& a, int level)
{
    int n = a.counters[C_LAST] + 1;
    for (int l = 0; l < level; l++) n = (n + kFold - 1) / kFold;
    return n;
}

/* the rows of a level (level 0: the slots' maps, kept in grid order): in groups
   of kFold, each row becomes the composition of its group up to it, the
   group's the row of the next level.  A warp per group, lane q = cache slot q;
   the sequential chain runs on shared memory and is only kFold long (one warp
   per 1,024 rows and one over the blocks took 504 us at 250,000 agents). */
constexpr int kFoldWarps = 4;
__global__ void __launch_bounds__(32 * kFoldWarps) k_kd_fold(KdArgs a, int level, int* rows, int* out)
{
    wait_for_previous();
    __shared__ int sm[kFoldWarps][32 * kMaxK];
    const int q = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int k = a.k, n = fold_rows(a, level);
    int* row = sm[w];
    for (int g = blockIdx.x * kFoldWarps + w; g * kFold < n; g += gridDim.x * kFoldWarps) {
        const int s1 = min((g + 1) * kFold, n);
        int cur = -(q + 1);
        for (int c0 = g * kFold; c0 < s1; c0 += 32) {
            const int cn = min(32, s1 - c0);
            bool mine = q < cn, mine_open = true;
            int at = c0 + q; /* the lane's row */
            if (level == 0) {
                mine = mine && querying(a, c0 + q);
                at = mine ? a.gidx[c0 + q] : 0;
                mine_open = mine && a.open[at];
            }
            const unsigned use = __ballot_sync(0xffffffffu, mine);
            unsigned refers = __ballot_sync(0xffffffffu, mine && mine_open), negative = 0u;
            /* 32 rows of k entries, 32 entries at a time */
            int j = q / k, x = q - j * k;
            const int dj = 32 / k, dx = 32 - dj * k;
#pragma unroll 8
            for (int i = 0; i < k; i++) {
                const int t = __shfl_sync(0xffffffffu, at, j);
                if ((use >> j) & 1u) {
                    const int v = rows[(size_t)t * k + x];
                    row[i * 32 + q] = v;
                    if (v < 0) negative |= 1u << j;
                }
                j += dj;
                x += dx;
                if (x >= k) {
                    x -= k;
                    j++;
                }
            }
            refers &= __reduce_or_sync(0xffffffffu, negative);
            __syncwarp();
            /* the open rows in order, each after the row in use before it */
            for (unsigned left = refers; left; left &= left - 1u) {
                const int r = __ffs(left) - 1;
                const unsigned before = use & ((1u << r) - 1u);
                if (before && q < k) cur = row[(31 - __clz(before)) * k + q];
                int v = q < k ? row[r * k + q] : 0;
                const int got = __shfl_sync(0xffffffffu, cur, v < 0 ? -v - 1 : q);
                if (v < 0) v = got;
                if (q < k) row[r * k + q] = v;
                __syncwarp();
            }
            if (use && q < k) cur = row[(31 - __clz(use)) * k + q];
            __syncwarp();
            j = q / k;
            x = q - j * k;
#pragma unroll 4
            for (int i = 0; i < k; i++) {
                const int t = __shfl_sync(0xffffffffu, at, j);
                if ((refers >> j) & 1u) rows[(size_t)t * k + x] = row[i * 32 + q];
                j += dj;
                x += dx;
                if (x >= k) {
                    x -= k;
                    j++;
                }
            }
            __syncwarp();
        }
        if (q < k) out[(size_t)g * k + q] = cur;
    }
}

/* entry -v - 1 of the list that slot group b starts from: the rows before b in
   its group of the next level, then of the level above that, ..., then the
   cache the tick started with (a slot: its grid index, or -(slot + 1) for one
   that is not in this tick's grid) */
__device__ __forceinline__ int fold_resolve(const KdArgs& a, int v, int b)
{
    const int* rows = a.agg;
    int n = (a.max_slots + kFold - 1) / kFold;
    while (v < 0) {
        if (b == 0) {
            const int c = a.cache[-v - 1];
            return a.mark[c] ? a.gidx[c] : -(c + 1);
        }
        if (b % kFold) v = rows[(size_t)(b - 1) * a.k + (-v - 1)];
        rows += (size_t)n * a.k;
        n = (n + kFold - 1) / kFold;
        b /= kFold;
    }
    return v;
}

/* the cache the next tick starts from: the composition of all rows (`total`)
   on this tick's.  One warp: every lane comes to the barrier between the
   reads, which go to other lanes' entries, and the writes. */
__global__ void __launch_bounds__(32) k_kd_cache(KdArgs a, const int* total)
{
    wait_for_previous();
    const int q = threadIdx.x;
    const bool mine = q < a.k && a.counters[C_LAST] >= 0;
    int c = 0;
    if (mine) {
        const int v = total[q];
        c = v < 0 ? a.cache[-v - 1] : a.s_slot[v];
    }
    __syncwarp();
    if (mine) a.cache[q] = c;
}

/* the open rows' references, looked up: the per-agent kernel's inputs (grid
   order; a neighbour in this tick's grid by its grid index, any other slot as
   -(slot + 1)) */
__global__ void k_kd_emit(KdArgs a)
{
    wait_for_previous();
    const int k = a.k, n = a.counters[C_NSORTED];
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        if (!a.open[t]) continue;
        const int slot = a.s_slot[t];
        if (!a.active[slot]) continue;
        int* row = a.nbr + (size_t)t * k;
        for (int q = 0; q < k; q++) {
            const int v = row[q];
            if (v < 0) row[q] = fold_resolve(a, v, slot / kFold);
        }
    }
}

int grid_n(int n, int threads, int sms)
{
    const long long need = ((long long)n + threads - 1) / threads;
    const long long cap = (long long)sms * 16;
    return (int)std::max(1LL, std::min(need, cap));
}

}  // namespace

/* rows of the composition's levels above the slots, together */
int kd_compose_rows(int max_slots)
{
    int n = max_slots, total = 0;
    do {
        n = (n + kFold - 1) / kFold;
        total += n;
    } while (n > 1);
    return total;
}
/* levels over the whole lists: at least the first (its own order), then until a
   segment fits a block */
static int kd_top(int cap)
{
    int top = 1;
    while ((cap >> top) > kKdSmall) top++;
    return top;
}
/* launches of the build, the query and the composition */
int kd_kernels(int max_slots)
{
    int fold = 0;
    for (int n = max_slots; fold == 0 || n > 1; fold++) n = (n + kFold - 1) / kFold;
    return 6 + 3 * 13 + 1 + 5 * kd_top(max_slots) + 4 + 1 + 2 + fold + 2;
}
int kd_hist_ints(int cap) { return 256 * ((cap + kRsTile - 1) / kRsTile + 1); } /* tiles, totals */
int kd_scan_tmp(int n) { return (n + kScanTile - 1) / kScanTile + 1; }

/* the build and the per-member maps, on s (beside the attraction kernel) */
cudaError_t kd_build_and_query(const KdArgs& a, cudaStream_t s, int sms)
{
    cudaError_t e = cudaMemsetAsync(a.mark, 0, (size_t)a.max_slots, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(a.tree, 0xff, sizeof(int) * (size_t)a.tree_cap, s);
    if (e != cudaSuccess) return e;
    const int gs = grid_n(a.max_slots, 256, sms), gc = grid_n(a.cap, 256, sms);
    k_kd_mark<<<gc, 256, 0, s>>>(a);
    /* members in slot order */
    launch_ahead(k_kd_flag, gs, 256, 0, s, a, a.iscan);
    e = scan_excl<int>(a.iscan, a.max_slots, a.scan_tmp32, s);
    if (e != cudaSuccess) return e;
    launch_ahead(k_kd_compact, gs, 256, 0, s, a, a.iscan, a.ids0);
    /* X0 = (x, index); Y = (y, x, index) sorted from X0; X = (x, y, index)
       sorted from Y (equal x keep Y's order, and equal x and y the index's) */
    launch_ahead(k_kd_keys, gc, 256, 0, s, a, a.ids0, 0, a.keys, a.X0);
    e = radix_sort(a.keys, a.X0, a.ktmp, a.vtmp, a.n_dev, a.cap, a.hist, s);
    if (e != cudaSuccess) return e;
    launch_ahead(k_kd_keys, gc, 256, 0, s, a, a.X0, 1, a.keys, a.Y[0]);
    e = radix_sort(a.keys, a.Y[0], a.ktmp, a.vtmp, a.n_dev, a.cap, a.hist, s);
    if (e != cudaSuccess) return e;
    launch_ahead(k_kd_keys, gc, 256, 0, s, a, a.Y[0], 0, a.keys, a.X[0]);
    e = radix_sort(a.keys, a.X[0], a.ktmp, a.vtmp, a.n_dev, a.cap, a.hist, s);
    if (e != cudaSuccess) return e;
    launch_ahead(k_kd_seg_init, gc, 256, 0, s, a);
    /* level 0 splits on X0 and partitions X and Y; then Y / X alternate; from
       level `top` on a segment is one block's */
    int xi = 0, yi = 0;
    const int top = kd_top(a.cap);
    for (int lv = 0; lv < top; lv++) {
        const bool on_y = (lv & 1) != 0;
        launch_ahead(k_kd_side, gc, 256, 0, s, a, lv == 0 ? a.X0 : (on_y ? a.Y[yi] : a.X[xi]));
        if (lv == 0 || on_y) {
            e = kd_partition(a, a.X[xi], a.X[xi ^ 1], lv == 0 ? 0 : 1, gc, s);
            xi ^= 1;
        }
        if (e == cudaSuccess && !on_y) {
            e = kd_partition(a, a.Y[yi], a.Y[yi ^ 1], 1, gc, s);
            yi ^= 1;
        }
        if (e != cudaSuccess) return e;
    }
    e = cudaFuncSetAttribute(k_kd_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(KdSmallSm));
    if (e != cudaSuccess) return e;
    launch_ahead(k_kd_small, 1 << top, kSmallThreads, sizeof(KdSmallSm), s, a, a.X[xi], a.Y[yi], top, a.iscan);
    /* queries in grid order: the agents of a warp are neighbours, so their
       traversals share nodes in cache */
    launch_ahead(k_kd_tree_pos, grid_n(a.tree_cap, 256, sms), 256, 0, s, a);
    const int gq = grid_n(a.cap, 128, sms);
    /* at most 25 levels (2^24 slots): 25.6 KB beside the lists' 33.8 KB at
       K = 32, above the default limit of 48 KB only there */
    const size_t far = sizeof(float2) * 32 * kQueryWarps * (size_t)a.levels;
    if (a.k <= 8) launch_ahead(k_kd_query<8>, gq, 32 * kQueryWarps, far, s, a, a.s_slot);
    else if (a.k <= 16) launch_ahead(k_kd_query<16>, gq, 32 * kQueryWarps, far, s, a, a.s_slot);
    else {
        e = cudaFuncSetAttribute(k_kd_query<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, 32 * 1024);
        if (e != cudaSuccess) return e;
        launch_ahead(k_kd_query<32>, gq, 32 * kQueryWarps, far, s, a, a.s_slot);
    }
    return cudaGetLastError();
}

/* after the attraction kernel: composition in slot order, then the inputs
   of the per-agent kernel */
cudaError_t kd_finish(const KdArgs& a, cudaStream_t s, int sms)
{
    int* rows = a.nbr;
    int* out = a.agg;
    int n = a.max_slots, level = 0;
    do {
        const int m = (n + kFold - 1) / kFold;
        const int gf = grid_n(m, kFoldWarps, sms);
        if (level == 0) k_kd_fold<<<gf, 32 * kFoldWarps, 0, s>>>(a, level, rows, out); /* after the join */
        else launch_ahead(k_kd_fold, gf, 32 * kFoldWarps, 0, s, a, level, rows, out);
        rows = out;
        out += (size_t)m * a.k;
        n = m;
        level++;
    } while (n > 1);
    launch_ahead(k_kd_emit, grid_n(a.cap, 256, sms), 256, 0, s, a);
    launch_ahead(k_kd_cache, 1, 32, 0, s, a, rows);
    return cudaGetLastError();
}

}  // namespace ecmg
