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
#include "rmpcd_common.cuh"
#include "sortnet.cuh"

namespace rmpcd {

constexpr int kOrderThreads = 256;
constexpr int kOrderSlots = 128;  // 1,280 particles at density 10: five per thread
constexpr int kOrderCap = 1792;   // 14 standard deviations above that
// a cell of an over-full tile with more particles than this is sorted by the
// whole block
constexpr int kOrderSmall = 64;

struct OrderTile {
    int idx[kOrderCap], raw[kOrderCap];
    int cstart[kOrderSlots], ccount[kOrderSlots];
    unsigned char cell[kOrderCap];
};

// entries of a[0, n), ascending by key, whose key is below v
template <typename Key, typename V>
__device__ inline int lower_bound_by(const int *a, int n, V v, Key key)
{
    int lo = 0, hi = n;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (key(a[mid]) < v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// the n values a[0, n), with distinct keys, into ascending order of their keys
// by the whole block: bottom-up merge sort, every element placed by its rank in
// the partner run; b is scratch of the same extent
template <typename Key>
__device__ inline void block_merge_sort(int *a, int *b, int n, Key key)
{
    int *src = a, *dst = b;
    for (int w = 1; w < n; w <<= 1) {
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            int run = i / w;
            int r0 = run * w;
            int v = src[i];
            int pos;
            if ((run & 1) == 0) {
                int p0 = r0 + w;
                int pn = min(w, max(0, n - p0));
                pos = r0 + (i - r0) + lower_bound_by(src + p0, pn, key(v), key);
            } else {
                int p0 = r0 - w;
                pos = p0 + (i - r0) + lower_bound_by(src + p0, w, key(v), key);
            }
            dst[pos] = v;
        }
        __syncthreads();
        int *t = src;
        src = dst;
        dst = t;
    }
    if (src != a)
        for (int i = threadIdx.x; i < n; i += blockDim.x) a[i] = src[i];
    __syncthreads();
}
__device__ inline void block_merge_sort(int *a, int *b, int n)
{
    block_merge_sort(a, b, n, [](int v) { return v; });
}

// The cells of a tile of more than kOrderCap particles, in place (tmp: scratch
// of the same extent); n: this thread's cell.  A function of its own, so that
// the gathers keep their registers for the tiles that there are.
static __device__ __noinline__ void order_dense(const OrderTile &sh, int cells, int n, int *perm, int *tmp)
{
    __syncthreads();
    if (n > 1 && n <= kOrderSmall) sort_segment(perm + sh.cstart[threadIdx.x], n);
    __syncthreads();
    for (int c = 0; c < cells; c++)
        if (sh.ccount[c] > kOrderSmall) block_merge_sort(perm + sh.cstart[c], tmp + sh.cstart[c], sh.ccount[c]);
    __syncthreads();
}

// Orders slots [s0, s1), s1 - s0 <= kOrderSlots, by a block of kOrderThreads;
// returns the tile's np ordered source indices, whose places start at a0.  A
// tile of more than kOrderCap particles is ordered in perm itself (tmp: scratch
// of the extent of perm, used at the tile's own places only; a gather passes
// its target's ids, which it writes afterwards).  Ends with a barrier; the caller puts one between
// its last use of the result and the next tile.
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
        __syncthreads();
        for (int j = t; j < np; j += kOrderThreads) {
            const int c = sh.cell[j], b = sh.cstart[c], m = sh.ccount[c];
            const int v = sh.raw[j];
            int r = 0;
#pragma unroll 4
            for (int k = b; k < b + m; k++) r += sh.raw[k] < v;
            sh.idx[b + r] = v;
        }
        __syncthreads();
        return sh.idx;
    }
    order_dense(sh, s1 - s0, n, perm + a0, tmp + a0);
    return perm + a0;
}

}  // namespace rmpcd
