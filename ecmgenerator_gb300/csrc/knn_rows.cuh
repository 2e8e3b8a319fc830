/*
 * knn_rows.cuh -- the exact kNN on the uniform agent grid: the k smallest
 * (d2, slot) with EPS < d2 < r^2 (KNearestAgents, KDTree.cpp:85-202, as an
 * exact query), one lane per agent, a warp at a time.
 *
 * The grid holds every agent: one outside the grid rectangle belongs to the
 * nearest border cell, so the border cells stand for half-infinite strips
 * and no agent needs a list of its own.
 */
#ifndef ECMG_KNN_ROWS_CUH
#define ECMG_KNN_ROWS_CUH

#include "ecmg_internal.h"

namespace ecmg {

/* cell index of a scaled coordinate, clamped to [0, n) (NaN: 0) */
__device__ __forceinline__ int cell_clamp(float f, int n)
{
    f = fminf(fmaxf(f, 0.0f), (float)n);
    return min((int)f, n - 1);
}

__device__ __forceinline__ int bucket_of(const AgentGrid& g, V2 p)
{
    return cell_clamp((p.y - g.y0) * g.inv, g.gh) * g.gw + cell_clamp((p.x - g.x0) * g.inv, g.gw);
}

/* ------------------------------------------------------------------------
 * The search.  A lane scans the grid rows that its search disc meets, the
 * nearest row first, from the disc's left to its right end: a row's cells are
 * consecutive in grid order, so a row is one range of candidates.  The disc
 * starts at the radius at which the local density (the 3 x 3 cells around the
 * agent) promises about 1.8 (k + 2) agents, shrinks to the k-th distance once
 * k are found, and grows (candidates below the old radius excluded) when it
 * held fewer than k.
 *
 * Accepted candidates go to the lane's column of a shared-memory buffer; when
 * a lane's buffer is full the whole warp sorts its buffers and merges them
 * into the lanes' lists with min / max networks, so that the warp does not run
 * a K-entry insertion for nearly every candidate because one of its lanes
 * wants one.  Keys are d2 with its 6 low mantissa bits replaced by the entry
 * of the lane's index column that holds the candidate's grid index: one float
 * min / max pair per comparator, and the lists come out sorted by d2 except
 * for keys within 2^-17 of each other ("near ties"), which are re-sorted by
 * the exact (d2, slot).  A near tie that may reach past the list (`rej` is the
 * smallest key dropped) is settled among the entries of the index column: a
 * crowd on a lattice has one nearly everywhere (100,000 points, k = 16: 88 us;
 * 508 when such lanes went to the 64-bit search).
 * ---------------------------------------------------------------------- */
constexpr unsigned kKnnCode = 63u; /* low key bits: entry of the index column */
/* list capacity K: the k nearest in key[K-k .. K-1]; entries below hold 0.
   Buffer entries: 8 merge into 16 at the cost per candidate of 16, with less
   of the buffers empty (a flush takes the whole warp); for K = 32 the merge
   weighs more.  Index column: every candidate accepted (24 on average at
   k = 16); with 46 entries eight blocks of the stand-alone query fit an SM's
   shared memory (the tick's, beside the attraction kernel, gets half or three
   quarters of it: four or six).  A lane that needs more (9 % of the warps have
   one in the 1M crossing) searches again, twice at most (renumbering the
   column instead cost every warp 15 % of its instructions, run or not; sent to
   the 64-bit search these lanes took the kernel from 318 to 369 us). */
template <int K>
constexpr int kKnnBuf = K <= 16 ? 8 : 16;
template <int K>
constexpr int kKnnIdx = K <= 8 ? 32 : (K <= 16 ? 46 : 64);

/* agents of the 3 x 3 cells around an agent from which its warp takes the
   search for crowded cells (CROWD).  There most of a row lies outside the disc
   that is wanted, whose first estimate is unreliable, and a column that is full
   would begin the search again and again: rows are tested eight at a time, and
   a full column is renumbered.  20,000 points in one cell of 4 m take 2,470 to
   3,400 us so, 17,900 with the ordinary search; 20,000 outside the grid 1,890
   and 13,000.  Evenly spread crowds set the line (100,000 points, ordinary /
   crowded; k = 16: 337 in the 3 x 3 89 / 102 us, 864 141 / 150, 1,944 279 / 233,
   3,456 437 / 330; k = 3: 740 66 / 117). */
constexpr int kKnnDense = 1024;

template <int K>
struct KnnSm { /* of one warp */
    float key[kKnnBuf<K>][32];
    int idx[kKnnIdx<K>][32];
    static_assert(kKnnIdx<K> <= (int)kKnnCode + 1, "index entries must fit the code");
    static_assert(kKnnIdx<K> - kKnnBuf<K> >= K, "a column without room for a buffer has filled the list");
};

__device__ __forceinline__ float knn_hi(float key) { return __uint_as_float(__float_as_uint(key) & ~kKnnCode); }

/* Batcher's odd-even merge sort of N = 2^m floats, ascending */
template <int N>
__device__ __forceinline__ void sort_net(float (&v)[N])
{
#pragma unroll
    for (int p = 1; p < N; p <<= 1)
#pragma unroll
        for (int q = p; q >= 1; q >>= 1)
#pragma unroll
            for (int j = q % p; j + q < N; j += 2 * q)
#pragma unroll
                for (int i = 0; i < q; i++)
                    if (i + j + q < N && (i + j) / (2 * p) == (i + j + q) / (2 * p)) {
                        const float a = v[i + j], b = v[i + j + q];
                        v[i + j] = fminf(a, b);
                        v[i + j + q] = fmaxf(a, b);
                    }
}

/* sorts a bitonic sequence of N = 2^m floats, ascending */
template <int N>
__device__ __forceinline__ void bitonic_net(float (&v)[N])
{
#pragma unroll
    for (int s = N / 2; s >= 1; s >>= 1)
#pragma unroll
        for (int i = 0; i < N; i++)
            if ((i & s) == 0) {
                const float a = v[i], b = v[i + s];
                v[i] = fminf(a, b);
                v[i + s] = fmaxf(a, b);
            }
}

/* the buffer's cnt entries into the list; *rej takes the smallest key dropped */
template <int K>
__device__ __forceinline__ void knn_flush(const KnnSm<K>& sm, int lane, int cnt, float (&key)[K], float* rej)
{
    constexpr int B = kKnnBuf<K>;
    float b[B];
#pragma unroll
    for (int i = 0; i < B; i++) b[i] = i < cnt ? sm.key[i][lane] : INFINITY;
    sort_net<B>(b);
    float d[B]; /* the dropped ones; their minimum as a tree, not a chain */
#pragma unroll
    for (int i = 0; i < B; i++) {
        const float o = key[K - B + i], n = b[B - 1 - i];
        d[i] = fmaxf(o, n);
        key[K - B + i] = fminf(o, n);
    }
#pragma unroll
    for (int w = B / 2; w >= 1; w >>= 1)
#pragma unroll
        for (int i = 0; i < w; i++) d[i] = fminf(d[i], d[i + w]);
    *rej = fminf(*rej, d[0]);
    bitonic_net<K>(key);
}

/* the column's entries that the (full) list refers to become its first K */
template <int K>
__device__ __forceinline__ void knn_renumber(int* column, float (&key)[K])
{
    int id[K];
#pragma unroll
    for (int q = 0; q < K; q++) id[q] = column[(__float_as_uint(key[q]) & kKnnCode) * 32];
#pragma unroll
    for (int q = 0; q < K; q++) {
        column[q * 32] = id[q];
        if (key[q] > 0.0f) key[q] = __uint_as_float((__float_as_uint(key[q]) & ~kKnnCode) | (unsigned)q);
    }
}

/* dx*dx + dy*dy of KDTree.cpp:107-108 (np: the negated centre; adding it is
   the subtraction), two components per instruction */
__device__ __forceinline__ float dist2(V2 q, float2 np)
{
    const float2 d = __fadd2_rn(make_float2(q.x, q.y), np);
    const float2 e = __fmul2_rn(d, d);
    return e.x + e.y;
}

/* The k nearest of the agents at p (one per lane; `valid` false: none) into
   the lanes' lists.  All 32 lanes must call.  Returns 1 when key[K-k .. K-1]
   (INFINITY beyond the count) is the answer in order, 2 when it holds near
   ties that must be re-sorted by the exact key, 3 when a near tie may reach
   past the list (whoever it may mean was accepted and is among the first
   *column entries of the lane's index column), 0 when the index column was too
   short for the search or (CHECK) the warp is one for the other variant (CROWD:
   for such a tie, the list itself is right but for it).  cs: the scene's cell
   starts. */
template <int K, bool CROWD, bool CHECK>
__device__ __forceinline__ int knn_rows(KnnSm<K>& sm, bool valid, int k, V2 p, float r2, const V2* s_pos,
                                        const int* cs, const AgentGrid& g, float (&key)[K], int* column)
{
    constexpr int B = kKnnBuf<K>;
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < K; q++) key[q] = q < K - k ? 0.0f : INFINITY;
    float rej = INFINITY;
    int ord = 0, ord0 = 0; /* next entry of the index column; that of the buffer's first candidate */
    bool over = false;     /* the index column is full (CROWD: has been renumbered) */
    int tries = 0;         /* searches begun again for that */
    valid = valid && p.x - p.x == 0.0f && p.y - p.y == 0.0f; /* no distance to a non-finite position is finite */
    const float fy = (p.y - g.y0) * g.inv;
    const int cx = cell_clamp((p.x - g.x0) * g.inv, g.gw), cy = cell_clamp(fy, g.gh);
    /* distance to the nearer end of the own row (0 outside the grid) and the
       side it lies on */
    const float ry = p.y - (g.y0 + (float)cy * g.cell);
    const int sy = ry + ry < g.cell ? -1 : 1;
    const float edge = fmaxf(fminf(ry, g.cell - ry), 0.0f) - g.slack;
    const float2 np = make_float2(-p.x, -p.y);
    float lim = 0.0f, lo = kEps, disc = 0.0f, more_area = 3.0f;
    int n9 = 0; /* agents of the 3 x 3 cells around p */
    if (valid) {
        const int xa = max(cx - 1, 0), xb = min(cx + 1, g.gw - 1), ya = max(cy - 1, 0), yb = min(cy + 1, g.gh - 1);
        for (int y = ya; y <= yb; y++) n9 += cs[y * g.gw + xb + 1] - cs[y * g.gw + xa];
        const float area = (float)((xb - xa + 1) * (yb - ya + 1)) * g.cell * g.cell;
        /* pi disc n9 / area = 1.8 (k + 2) */
        disc = fminf(r2, 0.573f * (float)(k + 2) * area / (float)max(n9, 1));
        /* a border cell is endless: the agents outside the grid are in it */
        if (CROWD && (cx == 0 || cx == g.gw - 1 || cy == 0 || cy == g.gh - 1)) disc = r2;
        lim = disc;
    }
    if (CHECK && __any_sync(kAll, n9 > kKnnDense)) { /* not a search for this variant */
        over = valid;
        tries = 2;
        lim = 0.0f;
        disc = r2;
    }
    while (true) {
        const int far_row = max(cy, g.gh - 1 - cy);
        for (int s = 0;; s++) {
            const int m = (s + 1) >> 1;
            const int y = cy + ((s & 1) ? sy * m : -sy * m);
            /* every row from here on is at least this far */
            const float at_least = (float)(m - 1) * g.cell + edge;
            const bool more = s == 0 ? lim > 0.0f : (m <= far_row && !(at_least > 0.0f && at_least * at_least >= lim));
            if (!__any_sync(kAll, more)) break;
            int j = 0, left = 0;
            if (more && y >= 0 && y < g.gh) {
                float dy = 0.0f;
                if (y > cy) dy = g.y0 + (float)y * g.cell - p.y;
                else if (y < cy) dy = p.y - (g.y0 + (float)(y + 1) * g.cell);
                dy = fmaxf(dy - g.slack, 0.0f);
                const float w2 = lim - dy * dy;
                if (w2 > 0.0f) {
                    const float w = sqrtf(w2) * 1.000001f + g.slack;
                    const int xa = cell_clamp((p.x - w - g.x0) * g.inv, g.gw);
                    const int xb = cell_clamp((p.x + w - g.x0) * g.inv, g.gw);
                    j = cs[y * g.gw + xa];
                    left = cs[y * g.gw + xb + 1] - j;
                }
            }
            const int longest = __reduce_max_sync(kAll, left);
            const int end = j + left;
            /* candidates beyond the k-th key (its code bits taken as ones)
               cannot enter any more; equal leading bits still count as near
               ties */
            auto shrink = [&] {
                if (key[K - 1] < INFINITY)
                    lim = fminf(lim, __uint_as_float((__float_as_uint(key[K - 1]) | kKnnCode) + 1u));
            };
            auto push = [&](float d2, int at) {
                sm.key[ord - ord0][lane] = __uint_as_float((__float_as_uint(d2) & ~kKnnCode) | (unsigned)ord);
                sm.idx[ord][lane] = at;
                ord++;
            };
            if (CROWD) {
                /* a long row: eight at a time while no lane wants one, else
                   four, with room for them made before */
                auto at = [&](int q) { return dist2(s_pos[max(min(j + q, end - 1), 0)], np); };
                for (int todo = longest; todo > 0;) {
                    if (todo >= 8) {
                        float d[8];
                        bool want = false;
#pragma unroll
                        for (int q = 0; q < 8; q++) d[q] = at(q);
#pragma unroll
                        for (int q = 0; q < 8; q++) want |= j + q < end && d[q] > lo && d[q] < lim;
                        if (!__any_sync(kAll, want)) {
                            j += 8;
                            todo -= 8;
                            continue;
                        }
                    }
                    const bool full = ord + 4 > kKnnIdx<K>; /* more than K accepted */
                    if (__any_sync(kAll, full || ord - ord0 > B - 4)) {
                        knn_flush<K>(sm, lane, ord - ord0, key, &rej);
                        if (full) {
                            knn_renumber<K>(&sm.idx[0][lane], key);
                            ord = K;
                            over = true;
                        }
                        ord0 = ord;
                        shrink();
                    }
                    float d[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) d[q] = at(q);
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        if (j + q < end && d[q] > lo && d[q] < lim) push(d[q], j + q);
                    j += 4;
                    todo -= 4;
                }
            } else {
                /* the next candidate's position is loaded while this one is used */
                V2 q = mk(0.0f, 0.0f);
                if (left > 0) q = s_pos[j];
                for (int it = longest; it > 0; it--) {
                    const float d2 = dist2(q, np);
                    const bool in = j < end && d2 > lo && d2 < lim;
                    if (j + 1 < end) q = s_pos[j + 1];
                    if (in) push(d2, j);
                    j++;
                    if (__any_sync(kAll, ord == ord0 + B)) {
                        knn_flush<K>(sm, lane, ord - ord0, key, &rej);
                        ord0 = ord;
                        shrink();
                        if (ord > kKnnIdx<K> - B) { /* no room for another buffer */
                            over = true;
                            lim = 0.0f;
                        }
                    }
                }
            }
        }
        if (__any_sync(kAll, ord != ord0)) {
            knn_flush<K>(sm, lane, ord - ord0, key, &rej);
            ord0 = ord;
        }
        /* fewer than k inside the disc: a larger one, without what the last
           one held (d2 >= disc is d2 > the float before it) */
        const bool grow = valid && !(key[K - 1] < INFINITY) && disc < r2;
        /* a full index column: once more from the start, with the k-th
           distance known by now (a disc of little more than k agents) */
        const bool again = !CROWD && over && tries < 2;
        if (!__any_sync(kAll, grow || again)) break;
        lim = 0.0f;
        if (grow) {
            lo = fmaxf(kEps, __uint_as_float(__float_as_uint(disc) - 1u));
            if (CROWD) { /* by the density that the disc has shown, or all */
                disc = ord > 0 ? fminf(r2, fmaxf(3.0f, 1.8f * (float)(k + 2) / (float)ord) * disc) : r2;
            } else {
                disc = fminf(r2, more_area * disc);
                more_area *= more_area;
            }
            lim = disc;
        }
        if (again) {
            disc = fminf(r2, __uint_as_float((__float_as_uint(key[K - 1]) | kKnnCode) + 1u));
            lim = disc;
            lo = kEps;
            rej = INFINITY;
            ord = ord0 = 0;
            over = false;
            tries++;
#pragma unroll
            for (int q = 0; q < K; q++) key[q] = q < K - k ? 0.0f : INFINITY;
        }
    }
    bool tie = false;
#pragma unroll
    for (int q = 0; q + 1 < K; q++)
        if (q >= K - k && key[q + 1] < INFINITY && knn_hi(key[q]) == knn_hi(key[q + 1])) tie = true;
    *column = ord;
    const bool past = key[K - 1] < INFINITY && knn_hi(rej) == knn_hi(key[K - 1]);
    if (over && (past || !CROWD)) return 0;
    return past ? 3 : (tie ? 2 : 1);
}

/* near ties in the list (rare; out of line): the n indices in o[0 .. n)
   re-sorted by the exact (d2, slot) key.  The keys are gathered first, side by
   side: a lone lane here is what the last warp waits for. */
template <int K>
__device__ __noinline__ void knn_resort(int n, V2 p, const V2* s_pos, const int* s_slot, int* o)
{
    unsigned long long key[K];
    int id[K];
#pragma unroll
    for (int q = 0; q < K; q++) {
        const int j = q < n ? o[q] : o[0];
        const V2 c = s_pos[j];
        const float dx = c.x - p.x, dy = c.y - p.y;
        key[q] = ((unsigned long long)__float_as_uint(dx * dx + dy * dy) << 32) | (unsigned)s_slot[j];
        id[q] = j;
    }
    for (int q = 1; q < n; q++) {
        const unsigned long long kk = key[q];
        const int j = id[q];
        int r = q;
        for (; r > 0 && key[r - 1] > kk; r--) {
            key[r] = key[r - 1];
            id[r] = id[r - 1];
        }
        key[r] = kk;
        id[r] = j;
    }
    for (int q = 0; q < n; q++) o[q] = id[q];
}

/* a near tie across the k-th place (a lattice crowd has one nearly everywhere;
   out of line): o[0 .. k) in key order; its entries with the leading bits `hi`
   of the k-th key are replaced by those of the n column entries with these
   bits that come first by the exact (d2, slot).  `before`: entries in front of
   them */
template <int K>
__device__ __noinline__ void knn_tied(const int* column, int n, int k, int before, unsigned hi, V2 p, const V2* s_pos,
                                      const int* s_slot, int* o)
{
    unsigned long long key[K];
    int id[K];
    const int room = k - before;
    int have = 0;
    const float2 np = make_float2(-p.x, -p.y);
    for (int i0 = 0; i0 < n; i0 += 4) {
        unsigned d2[4];
        int j[4];
#pragma unroll
        for (int u = 0; u < 4; u++) j[u] = column[min(i0 + u, n - 1) * 32];
#pragma unroll
        for (int u = 0; u < 4; u++) d2[u] = __float_as_uint(dist2(s_pos[j[u]], np));
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (i0 + u >= n || (d2[u] & ~kKnnCode) != hi) continue;
            const unsigned long long kk = ((unsigned long long)d2[u] << 32) | (unsigned)s_slot[j[u]];
            if (have == room && kk >= key[room - 1]) continue;
            int q = have < room ? have++ : room - 1;
            for (; q > 0 && key[q - 1] > kk; q--) {
                key[q] = key[q - 1];
                id[q] = id[q - 1];
            }
            key[q] = kk;
            id[q] = j[u];
        }
    }
    for (int q = 0; q < have; q++) o[before + q] = id[q];
}

/* the search by 64-bit (d2, slot) keys (rare: a near tie across the k-th place
   after the column was renumbered, or a column full for the third time where
   there is no variant for crowded cells; out of line): the rows of the disc of
   squared radius `lim`, which holds at least k agents or is r^2; o[q] gets
   the grid indices, the return value is the count */
template <int K>
__device__ __noinline__ int knn_exact(int k, V2 p, float lim, float r2, const V2* s_pos, const int* s_slot,
                                      const int* cs, AgentGrid g, int* o)
{
    unsigned long long key[K];
    int id[K];
    for (int q = 0; q < k; q++) key[q] = ~0ull;
    int n = 0;
    const float w = sqrtf(lim) * 1.000001f + g.slack;
    const int xa = cell_clamp((p.x - w - g.x0) * g.inv, g.gw), xb = cell_clamp((p.x + w - g.x0) * g.inv, g.gw);
    const int ya = cell_clamp((p.y - w - g.y0) * g.inv, g.gh), yb = cell_clamp((p.y + w - g.y0) * g.inv, g.gh);
    const float2 np = make_float2(-p.x, -p.y);
    for (int y = ya; y <= yb; y++) {
        const int e = cs[y * g.gw + xb + 1];
        for (int j = cs[y * g.gw + xa], next = j; j < e; j++) {
            if (j == next) { /* eight at a time while none can enter: a lone lane waits for every load */
                float d[8];
                bool want = false;
#pragma unroll
                for (int q = 0; q < 8; q++) d[q] = dist2(s_pos[min(j + q, e - 1)], np);
#pragma unroll
                for (int q = 0; q < 8; q++) want |= !(d[q] > lim);
                next += 8;
                if (!want) {
                    j += 7;
                    continue;
                }
            }
            const V2 c = s_pos[j];
            const float dx = c.x - p.x, dy = c.y - p.y;
            const float d2 = dx * dx + dy * dy;
            if (!(d2 > kEps) || !(d2 < r2) || d2 > lim) continue;
            const unsigned long long kk = ((unsigned long long)__float_as_uint(d2) << 32) | (unsigned)s_slot[j];
            if (n == k && kk >= key[k - 1]) continue;
            int q = n < k ? n++ : k - 1;
            for (; q > 0 && key[q - 1] > kk; q--) {
                key[q] = key[q - 1];
                id[q] = id[q - 1];
            }
            key[q] = kk;
            id[q] = j;
            if (n == k) lim = __uint_as_float((unsigned)(key[k - 1] >> 32));
        }
    }
    for (int q = 0; q < n; q++) o[q] = id[q];
    return n;
}

/* o[0 .. k) of one lane from its list and column (knn_rows' answer st); returns
   the count */
template <int K, bool SLOTS>
__device__ __forceinline__ int knn_write(const KnnSm<K>& sm, int st, int k, V2 p, float r2, const float (&key)[K],
                                         int column, const V2* s_pos, const int* s_slot, const int* cs,
                                         const AgentGrid& g, int* o)
{
    const int lane = threadIdx.x & 31;
    int n = 0, before = 0; /* before: keys below the k-th's leading bits */
    int id[K];
#pragma unroll
    for (int q = 0; q < K; q++) {
        const bool in = q >= K - k && key[q] < INFINITY;
        id[q] = in ? sm.idx[__float_as_uint(key[q]) & kKnnCode][lane] : -1;
        n += in ? 1 : 0;
        before += in && knn_hi(key[q]) < knn_hi(key[K - 1]) ? 1 : 0;
    }
    if (SLOTS && st == 1) {
#pragma unroll
        for (int q = 0; q < K; q++)
            if (id[q] >= 0) id[q] = s_slot[id[q]];
    }
    if (k == K && (reinterpret_cast<size_t>(o) & 15) == 0) {
#pragma unroll
        for (int q = 0; q < K; q += 4)
            *reinterpret_cast<int4*>(o + q) = make_int4(id[q], id[q + 1], id[q + 2], id[q + 3]);
    } else {
#pragma unroll
        for (int q = 0; q < K; q++)
            if (q >= K - k) o[q - (K - k)] = id[q];
    }
    if (st == 3)
        knn_tied<K>(&sm.idx[0][lane], column, k, before, __float_as_uint(key[K - 1]) & ~kKnnCode, p, s_pos, s_slot, o);
    if (st >= 2) knn_resort<K>(n, p, s_pos, s_slot, o);
    else if (st == 0)
        n = knn_exact<K>(k, p, fminf(r2, __uint_as_float(__float_as_uint(key[K - 1]) | kKnnCode)), r2, s_pos, s_slot,
                         cs, g, o);
    if (SLOTS && st != 1)
        for (int q = 0; q < n; q++) o[q] = s_slot[o[q]];
    return n;
}

/* knn_list where the cells hold far more agents than a search wants (out of
   line, so that the ordinary search keeps its registers and instructions) */
template <int K, bool SLOTS>
__device__ __noinline__ int knn_list_crowd(KnnSm<K>* sm, bool valid, int k, V2 p, float r2, const V2* s_pos,
                                           const int* s_slot, const int* cs, AgentGrid g, int* o)
{
    float key[K];
    int column;
    const int st = knn_rows<K, true, false>(*sm, valid, k, p, r2, s_pos, cs, g, key, &column);
    return valid ? knn_write<K, SLOTS>(*sm, st, k, p, r2, key, column, s_pos, s_slot, cs, g, o) : 0;
}

/* the neighbour list of the agent at p: grid indices (SLOTS: slots) in
   o[0 .. k), -1 beyond the count, which is returned.  CROWDS: with the variant
   for crowded cells.  All 32 lanes must call; lanes with valid false write
   nothing. */
template <int K, bool SLOTS, bool CROWDS>
__device__ __forceinline__ int knn_list(KnnSm<K>& sm, bool valid, int k, V2 p, float r2, const V2* s_pos,
                                        const int* s_slot, const int* cs, const AgentGrid& g, int* o)
{
    float key[K];
    int column;
    const int st = knn_rows<K, false, CROWDS>(sm, valid, k, p, r2, s_pos, cs, g, key, &column);
    const bool left = CROWDS && valid && st == 0;
    int n = 0;
    if (valid && !left) n = knn_write<K, SLOTS>(sm, st, k, p, r2, key, column, s_pos, s_slot, cs, g, o);
    if (CROWDS && __any_sync(0xffffffffu, left)) {
        const int c = knn_list_crowd<K, SLOTS>(&sm, left, k, p, r2, s_pos, s_slot, cs, g, o);
        if (left) n = c;
    }
    return n;
}

}  // namespace ecmg
#endif
