// In-cell ordering of a tile of consecutive slots, shared by the gathers that
// complete a cell sort: the tile's source indices perm[a0, a0 + np) -- in cell
// order, in any order inside a cell -- are put in ascending order inside each
// cell (the reference's stable single-thread order, src/particle_system.f90:322-338)
// in shared memory, where the gather reads them.  Every index is placed at its
// rank among its cell's indices, one thread per index, so a crowded cell costs
// no more than its share, and the order needs neither its own pass over perm
// nor that pass's uncoalesced per-cell walks (31 us per sort at
// 64^3, 101-122 us at 128^3 FP32).  A 64^3 FP64 call-by-call run went from 17.6
// to 16.7 ms, the 32^3 dimer engine from 10.1 to 9.3 ms.
#pragma once
#include <cmath>

#include "rmpcd_common.cuh"

namespace rmpcd {

constexpr int kOrderThreads = 256;
constexpr int kOrderSlots = 128;  // 1,280 particles at density 10: five per thread
constexpr int kOrderCap = 1792;   // 14 standard deviations above that
// runs with a cell of more particles than this are ordered by merging: the ranks
// would take as many reads per index
constexpr int kOrderSmall = 64;

// Slots per tile at a mean occupancy: what kOrderCap holds with four standard
// deviations to spare, at most kOrderSlots.  us per sort at 48^3 FP64 with 128 slots
// whatever the density, with these, and with the ordering as a pass of its own:
// density 15: 102, 86, 106; 30: 202, 139, 213; 100: 1024, 418, 8140; at 16^3 100: 565, 39,
// 325.  (Density 10: 62.7, 62.8, 77.4.)
inline int order_slots(double mean)
{
    int per = kOrderSlots;
    while (per > 1 && per * mean + 4 * sqrt(per * mean) > kOrderCap) per--;
    return per;
}

struct OrderTile {
    int idx[kOrderCap], raw[kOrderCap];
    int cstart[kOrderSlots], ccount[kOrderSlots];
    unsigned char cell[kOrderCap];
};

// The n values a[0, n), with distinct keys, into ascending order of their keys
// by the whole block; b is scratch of the same extent.  Pieces of 32 by rank, then
// runs merged two by two, a thread taking up to 32 places of the result at a time:
// where they begin in the two runs takes one search, the rest is a walk along
// both.  (A search per element made a sort of the system with 276,000 particles in one
// cell take 18.4 ms; now 6.4, of which this is a part.)
template <typename Key>
__device__ inline void block_merge_sort(int *a, int *b, int n, Key key)
{
    constexpr int P = 32;
    const int T = blockDim.x;
    for (int i = threadIdx.x; i < n; i += T) {
        const int q = i / P * P, m = min(P, n - q), v = a[i];
        const auto kv = key(v);
        int r = 0;
        for (int k = 0; k < m; k++) r += key(a[q + k]) < kv;
        b[q + r] = v;
    }
    __syncthreads();
    int per = 1;
    while (per < P && per * T < n) per <<= 1;
    int *src = b, *dst = a;
    for (long long w = P; w < n; w <<= 1) {
        for (long long o = (long long)per * threadIdx.x; o < n; o += (long long)per * T) {
            const long long p = o / (2 * w) * (2 * w);
            const int na = (int)min(w, n - p), nb = (int)max(0LL, min(w, n - p - w)), d = (int)(o - p);
            const int *A = src + p, *B = A + na;
            // of the pair's first d places, those that come from A
            int lo = max(0, d - nb), hi = min(d, na);
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (key(A[mid]) < key(B[d - 1 - mid])) lo = mid + 1;
                else hi = mid;
            }
            int i = lo, j = d - lo;
            const int e = min(per, na + nb - d);
            int va = i < na ? A[i] : 0, vb = j < nb ? B[j] : 0;
            decltype(key(0)) ka = 0, kb = 0;
            if (i < na) ka = key(va);
            if (j < nb) kb = key(vb);
            for (int k = 0; k < e; k++) {
                if (j >= nb || (i < na && ka < kb)) {
                    dst[o + k] = va;
                    if (++i < na) ka = key(va = A[i]);
                } else {
                    dst[o + k] = vb;
                    if (++j < nb) kb = key(vb = B[j]);
                }
            }
        }
        __syncthreads();
        int *t = src;
        src = dst;
        dst = t;
    }
    if (src != a)
        for (int i = threadIdx.x; i < n; i += T) a[i] = src[i];
    __syncthreads();
}
__device__ inline void block_merge_sort(int *a, int *b, int n)
{
    block_merge_sort(a, b, n, [](int v) { return v; });
}

// The m indices raw[0, m) of consecutive cells (cell[j]: the cell of place j; b0:
// the first one's cstart) in order, to out[0, m): each at its rank among its
// cell's, which every one of the cell's reads.  raw may be written after a barrier.
__device__ __forceinline__ void order_by_rank(const OrderTile &sh, int b0, int m, int *out)
{
    for (int j = threadIdx.x; j < m; j += kOrderThreads) {
        const int c = sh.cell[j], b = sh.cstart[c] - b0, n = sh.ccount[c];
        const int v = sh.raw[j];
        int r = 0;
#pragma unroll 4
        for (int k = b; k < b + n; k++) r += sh.raw[k] < v;
        out[b + r] = v;
    }
}

// The same where a cell has more than kOrderSmall: pieces of 32 by
// rank, then every cell's runs merged two by two, each index by its rank in the
// partner run.  Leaves the result in idx or raw.  A function of its own, so that
// the gathers keep their registers for the tiles that there are.
static __device__ __noinline__ int *order_by_merge(OrderTile &sh, int b0, int m)
{
    constexpr int P = 32;
    int *src = sh.raw, *dst = sh.idx;
    for (int w = P / 2;; w <<= 1) {
        bool more = false;
        for (int j = threadIdx.x; j < m; j += kOrderThreads) {
            const int c = sh.cell[j], b = sh.cstart[c] - b0, n = sh.ccount[c], i = j - b, v = src[j];
            more = more || n > 2 * w;
            int to;
            if (w < P) {  // the first pass: the place among the 32
                const int q = i / P * P, e = min(P, n - q);
                to = q;
                for (int k = 0; k < e; k++) to += src[b + q + k] < v;
            } else {
                const int run = i / w, r0 = run * w, p0 = (run & 1) ? r0 - w : r0 + w;
                int lo = 0, hi = min(w, max(0, n - p0));
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (src[b + p0 + mid] < v) lo = mid + 1;
                    else hi = mid;
                }
                to = ((run & 1) ? p0 : r0) + (i - r0) + lo;
            }
            dst[b + to] = v;
        }
        more = __syncthreads_or(more);
        int *t = src;
        src = dst;
        dst = t;
        if (!more) return src;
    }
}

// The cells of a tile of more than kOrderCap particles, in place (tmp: scratch of the
// same extent), run by run: the next cells that fit, or one that does not by itself.
// A function of its own, as above.
static __device__ __noinline__ void order_dense(OrderTile &sh, int cells, int *perm, int *tmp)
{
    const int t = threadIdx.x;
    __syncthreads();
    for (int c0 = 0, k; c0 < cells; c0 += k) {
        const int a = sh.cstart[c0];
        // (its barrier also ends the run before)
        k = __syncthreads_count(t >= c0 && t < cells && sh.cstart[t] + sh.ccount[t] - a <= kOrderCap);
        if (k == 0) {
            block_merge_sort(perm + a, tmp + a, sh.ccount[c0]);
            k = 1;
            continue;
        }
        const int last = c0 + k - 1, m = sh.cstart[last] + sh.ccount[last] - a;
        const int n = t >= c0 && t <= last ? sh.ccount[t] : 0;
        for (int i = 0; i < n; i++) sh.cell[sh.cstart[t] - a + i] = (unsigned char)t;
        for (int j = t; j < m; j += kOrderThreads) sh.raw[j] = perm[a + j];
        if (__syncthreads_or(n > kOrderSmall)) {
            const int *v = order_by_merge(sh, a, m);
            for (int j = t; j < m; j += kOrderThreads) perm[a + j] = v[j];
        } else {
            order_by_rank(sh, a, m, perm + a);
        }
    }
    __syncthreads();
}

// Orders slots [s0, s1), s1 - s0 <= kOrderSlots, by a block of kOrderThreads;
// returns the tile's np ordered source indices, whose places start at a0.  A
// tile of more than kOrderCap particles is ordered in perm itself (tmp: scratch of the extent
// of perm, used at the tile's own places only; a gather passes its target's ids, which
// it writes afterwards).  Ends with a barrier; the caller puts one between its last
// use of the result and the next tile.
__device__ inline const int *order_tile(OrderTile &sh, int s0, int s1, const int *__restrict__ count,
                                        const int *__restrict__ start, int *perm, int *tmp, int &a0, int &np)
{
    const int t = threadIdx.x;
    a0 = start[s0];
    np = start[s1 - 1] + count[s1 - 1] - a0;
    int n = 0, a = 0;
    if (t < kOrderSlots && s0 + t < s1) {
        n = count[s0 + t];
        a = start[s0 + t];
    }
    if (t < kOrderSlots) {
        sh.cstart[t] = a - a0;
        sh.ccount[t] = n;
    }
    if (np <= kOrderCap) {
        for (int k = 0; k < n; k++) sh.cell[a - a0 + k] = (unsigned char)t;
        for (int j = t; j < np; j += kOrderThreads) sh.raw[j] = perm[a0 + j];
        // by rank whatever the cells' sizes (asking whether to merge them costs every
        // tile a few spilled registers: 64^3 sort 112.9 us for 111.8)
        __syncthreads();
        order_by_rank(sh, 0, np, sh.idx);
        __syncthreads();
        return sh.idx;
    }
    order_dense(sh, s1 - s0, perm + a0, tmp + a0);
    return perm + a0;
}

}  // namespace rmpcd
