// The bulk schedule on buckets: one kernel per interval.
//
// Every cell owns a bucket of `cap` records in each of two buffers.  The
// interval kernel reads its tile's buckets -- each a contiguous run of
// records, so the reads are coalesced and wait for nothing but the counts --
// collides, streams and keys the particles in shared memory, takes a place in
// the next cell's bucket from the counting atomic, and writes the record
// there: a scattered write that nothing waits for takes the place of the
// scattered gather, and neither slot scan nor placement pass is left.
//   FP32 record, 32 B (one DRAM sector): [vx vy vz species][px py pz idx]
//   FP64 record, 64 B: [vx vy][vz (species,idx)][px py][pz order]
// In FP64 the order of a cell's particles matters: `order` is (slot, rank) of
// the particle in the grid it comes from, its place in the reference's
// single-thread order, and the next interval ranks each cell's particles by
// it.  A bucket's overflow goes to a linked list in a pool of N records.
// HBM traffic per particle: record read + write (64 B FP32, 128 B FP64); per
// cell 16 B (count read, next count, cleared count and list head).
//
// Buckets are numbered like the Hilbert slots, or, in a box whose slots are
// more than its cells, by the rank of the slot among those of the box's cells
// (BucketMap), so that memory and tiles go to cells only.  The slots outside
// the box follow; they have no bucket and keep their particles (positions
// outside the box, NaN) in lists.
//
// Work inside a tile: one bulk copy per cell brings its records into shared
// memory (no instruction and no load/store wavefront per particle) while the
// last warps draw the cells' rotations; the FP32 cell sums (exact, so in any
// order), the rotation and the streaming are spread over all threads; the FP64
// sums, one after the other in the reference's order, take a lane per cell and
// component.  A record is read once by the thread that streams it, which
// writes it to its bucket from registers.
#pragma once

namespace rmpcd {

template <typename R>
struct Bucket;
template <>
struct Bucket<float> {
    static constexpr int kBytes = 32;
    static constexpr int kChunks = 2;  // 16-byte chunks of a record
};
template <>
struct Bucket<double> {
    static constexpr int kBytes = 64;
    static constexpr int kChunks = 4;
};

// the bucket arrays of one grid
struct BucketGrid {
    unsigned char *rec;   // n_rec * cap records
    unsigned char *pool;  // overflow records
    int *link;            // pool: next node of the bucket's list, -1 at its end
    int *count;           // particles per bucket
    int *head;            // first pool node per bucket, -1 without overflow
    int *n_pool;          // nodes in use, and (n_pool[3]) places of ids in use
    int cap, n_rec;       // records per bucket, buckets with records
    __host__ __device__ int cap_of(int b) const { return b < n_rec ? cap : 0; }
};

// the numbering of the buckets (null: the slots')
struct BucketMap {
    const int *of_slot, *slot_of;
};

template <typename R>
struct BucketArgs {
    BucketGrid in, out;
    int *count_clear, *head_clear, *n_pool_clear;  // those of the grid after next
    int S;
    BucketMap map;
    int *ix, *iy, *iz;
    Grid g_next;  // lut: the bucket of every cell
    double e0, e1, e2;
    R dt;
    double sin_a, cos_a;
    uint64_t seed, step;
    const double *axes;
    unsigned *err;  // device error word
    int *ids, *ids_tmp;  // N places each for over-full tiles
};

// threads per cell in the sums of a tile
template <typename S>
constexpr int lanes_per_cell()
{
    int g = 1;
    while (2 * g * S::kSlots <= S::kThreads && 2 * g <= 16) g *= 2;
    return g;
}

template <typename R, typename S>
struct BucketTile {
    static constexpr int Q = Bucket<R>::kChunks;
    int4 rec[S::kCap][Q];
    // omega and the mean velocity of every cell, row by row: m0 m1 m2 lv
    alignas(16) R mat[S::kSlots][12];
    unsigned long long bar;
    int cstart[S::kSlots], ccount[S::kSlots];
    int wsum[S::kThreads / 32];
    unsigned char cell[S::kCap];    // tile-local cell of every particle
    unsigned char spin[S::kSlots];  // the cell is rotated (two particles or more)
    // FP64: slot of every cell, rank of every particle in its cell, and the
    // particles by rank, cell by cell
    static constexpr int M = sizeof(R) == 8 ? S::kCap : 1;
    int slot[sizeof(R) == 8 ? S::kSlots : 1];
    unsigned short rank[M], ord[M];
};

// All chunks of record j of the tile, j consecutive over the lanes.  The lanes
// start at different chunks, so that eight 16-byte reads 32 (64) bytes apart
// meet all banks once instead of two (four) times.
template <typename S>
__device__ __forceinline__ void read_record(const BucketTile<float, S> &sh, int j, int4 c[2])
{
    const int r = (threadIdx.x >> 2) & 1;
    const int4 a = sh.rec[j][r], b = sh.rec[j][r ^ 1];
    c[0] = r ? b : a;
    c[1] = r ? a : b;
}
template <typename S>
__device__ __forceinline__ void read_record(const BucketTile<double, S> &sh, int j, int4 c[4])
{
    const int r = (threadIdx.x >> 1) & 3;
    int4 x[4], y[4];
#pragma unroll
    for (int i = 0; i < 4; i++) x[i] = sh.rec[j][(i + r) & 3];
    // c[k] = x[(k - r) & 3]
#pragma unroll
    for (int k = 0; k < 4; k++) y[k] = r & 1 ? x[(k + 3) & 3] : x[k];
#pragma unroll
    for (int k = 0; k < 4; k++) c[k] = r & 2 ? y[(k + 2) & 3] : y[k];
}

__device__ inline void store_record(unsigned char *p, const int4 &a, const int4 &b)
{
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z),
                 "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                 : "memory");
}

__device__ inline double2 as_double2(const int4 &a)
{
    return make_double2(__hiloint2double(a.y, a.x), __hiloint2double(a.w, a.z));
}
__device__ inline int4 as_int4(double a, double b)
{
    return make_int4(__double2loint(a), __double2hiint(a), __double2loint(b), __double2hiint(b));
}

// exclusive scan over the block's T threads
template <int T>
__device__ inline int tile_scan(int n, int *wsum, int &total)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int inc = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) wsum[w] = inc;
    __syncthreads();
    int before = 0;
    total = 0;
#pragma unroll
    for (int k = 0; k < T / 32; k++) {
        before += k < w ? wsum[k] : 0;
        total += wsum[k];
    }
    return before + inc - n;
}

// the cell sums and means of the tile (src/mpcd.f90:127-160): FP32 by exact
// fixed-point sums, a group of lanes per cell; FP64 in the order ord, a lane
// per cell and component
template <typename S>
__device__ __forceinline__ void bucket_means(BucketTile<float, S> &sh)
{
    constexpr int G = lanes_per_cell<S>();
    const int c = threadIdx.x / G, g = threadIdx.x % G;
    const int n = c < S::kSlots ? sh.ccount[c] : 0, a = c < S::kSlots ? sh.cstart[c] : 0;
    int n_eff = 0;
    long long sx = 0, sy = 0, sz = 0;
    for (int k = a + g; k < a + n; k += G) {
        const int4 v = sh.rec[k][0];
        if (v.w > 0) {
            sx += to_fixed(__int_as_float(v.x));
            sy += to_fixed(__int_as_float(v.y));
            sz += to_fixed(__int_as_float(v.z));
            n_eff++;
        }
    }
#pragma unroll
    for (int o = 1; o < G; o <<= 1) {
        sx += __shfl_xor_sync(0xffffffffu, sx, o);
        sy += __shfl_xor_sync(0xffffffffu, sy, o);
        sz += __shfl_xor_sync(0xffffffffu, sz, o);
        n_eff += __shfl_xor_sync(0xffffffffu, n_eff, o);
    }
    if (c < S::kSlots && g < 3) {
        if (g == 0) sh.spin[c] = n_eff > 1;
        if (n_eff > 1) {
            if constexpr (G >= 3) {  // a lane per component divides
                sh.mat[c][4 * g + 3] = fixed_mean(g == 0 ? sx : (g == 1 ? sy : sz), n_eff);
            } else if (g == 0) {
                sh.mat[c][3] = fixed_mean(sx, n_eff);
                sh.mat[c][7] = fixed_mean(sy, n_eff);
                sh.mat[c][11] = fixed_mean(sz, n_eff);
            }
        }
    }
}
template <typename S>
__device__ __forceinline__ void bucket_means(BucketTile<double, S> &sh)
{
    constexpr int G = lanes_per_cell<S>();
    static_assert(G >= 4, "a lane per component");
    const int c = threadIdx.x / G, g = threadIdx.x % G;
    if (c >= S::kSlots || g > 2) return;
    const int n = sh.ccount[c], a = sh.cstart[c];
    const int q = g >> 1, w = 8 * (g & 1);  // component g: double g & 1 of chunk g / 2
    int n_eff = 0;
    double s = 0;
#pragma unroll 4
    for (int k = a; k < a + n; k++) {
        const int j = sh.ord[k];
        if (sh.rec[j][1].z > 0) {
            s = s + *(const double *)((const unsigned char *)&sh.rec[j][q] + w);
            n_eff++;
        }
    }
    if (g == 0) sh.spin[c] = n_eff > 1;
    if (n_eff > 1) sh.mat[c][4 * g + 3] = s / n_eff;
}

template <typename R, typename S>
__device__ __forceinline__ void bucket_rotate(const BucketTile<R, S> &sh, int c, R &x, R &y, R &z)
{
    if (!sh.spin[c]) return;
    alignas(16) R w[12];
    constexpr int V = 12 * sizeof(R) / 16;
#pragma unroll
    for (int i = 0; i < V; i++) ((int4 *)w)[i] = ((const int4 *)sh.mat[c])[i];
    CellRot<R> o;
    R lv[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
#pragma unroll
        for (int k = 0; k < 3; k++) o.m[i][k] = w[4 * i + k];
        lv[i] = w[4 * i + 3];
    }
    cell_rotate(x, y, z, lv, o);
}

// stream_values with the bucket of the new position
template <typename R>
__device__ __forceinline__ int bucket_stream_values(const BucketArgs<R> &A, R &x, R &y, R &z, R vx, R vy, R vz, int idx)
{
    stream_position<R>(A, x, y, z, vx, vy, vz, idx);
    int p[3];
    cell_coords(A.g_next, (double)x, (double)y, (double)z, p);
    if (in_grid(A.g_next, p)) return cell_entry(A.g_next, p);
    const int s = hilbert::compact_index(p, A.g_next.M);
    return A.map.of_slot ? A.map.of_slot[s] : s;
}

// rotate, stream and key particle j of the tile; c: its new record
template <typename S>
__device__ __forceinline__ int bucket_move(const BucketTile<float, S> &sh, const BucketArgs<float> &A, int j, int4 c[2])
{
    read_record(sh, j, c);
    float vx = __int_as_float(c[0].x), vy = __int_as_float(c[0].y), vz = __int_as_float(c[0].z);
    bucket_rotate<float, S>(sh, sh.cell[j], vx, vy, vz);
    float x = __int_as_float(c[1].x), y = __int_as_float(c[1].y), z = __int_as_float(c[1].z);
    const int key = bucket_stream_values<float>(A, x, y, z, vx, vy, vz, c[1].w);
    c[0] = make_int4(__float_as_int(vx), __float_as_int(vy), __float_as_int(vz), c[0].w);
    c[1] = make_int4(__float_as_int(x), __float_as_int(y), __float_as_int(z), c[1].w);
    return key;
}
template <typename S>
__device__ __forceinline__ int bucket_move(const BucketTile<double, S> &sh, const BucketArgs<double> &A, int j, int4 c[4])
{
    const int cell = sh.cell[j];
    read_record(sh, j, c);
    const double2 v = as_double2(c[0]), p = as_double2(c[2]);
    double vx = v.x, vy = v.y, vz = __hiloint2double(c[1].y, c[1].x);
    bucket_rotate<double, S>(sh, cell, vx, vy, vz);
    double x = p.x, y = p.y, z = __hiloint2double(c[3].y, c[3].x);
    const int key = bucket_stream_values<double>(A, x, y, z, vx, vy, vz, c[1].w);
    c[0] = as_int4(vx, vy);
    c[1] = make_int4(__double2loint(vz), __double2hiint(vz), c[1].z, c[1].w);
    c[2] = as_int4(x, y);
    // order: rank in the low word, slot above it
    c[3] = make_int4(__double2loint(z), __double2hiint(z), sh.rank[j], sh.slot[cell]);
    return key;
}

// A node of the pool.  kMany (over-full tiles): one atomic for the threads of the
// warp that are here, since every overflow of the grid counts on this one address
// (resting 48^3 fluid in one octant, FP32: 721 us per interval with an atomic each, 386
// so); in the other tiles, where one cell in
// 20,000 overflows, the shuffle's convergence costs 0.7 %.
template <bool kMany>
__device__ __forceinline__ int pool_node(const BucketGrid &g)
{
    if constexpr (!kMany) return atomicAdd(g.n_pool, 1);
    const unsigned here = __activemask();
    const int lead = __ffs(here) - 1;
    int base = 0;
    if ((int)(threadIdx.x & 31) == lead) base = atomicAdd(g.n_pool, __popc(here));
    return __shfl_sync(here, base, lead) + __popc(here & lanemask_lt());
}

// where record number `place` of bucket key goes: its bucket, or a new node of
// its list
template <typename R, bool kMany>
__device__ __forceinline__ unsigned char *bucket_place(const BucketGrid &g, int key, int place)
{
    if (place < g.cap_of(key)) return g.rec + ((size_t)key * g.cap + place) * Bucket<R>::kBytes;
    const int node = pool_node<kMany>(g);
    g.link[node] = atomicExch(g.head + key, node);
    return g.pool + (size_t)node * Bucket<R>::kBytes;
}

// FP64: rank and order of the tile's particles by their order words
template <typename S>
__device__ __forceinline__ void bucket_rank(BucketTile<double, S> &sh, int np)
{
    for (int j = threadIdx.x; j < np; j += S::kThreads) {
        const int c = sh.cell[j], a = sh.cstart[c], n = sh.ccount[c];
        const int lo = sh.rec[j][3].z, hi = sh.rec[j][3].w;
        int r = 0;
#pragma unroll 4
        for (int k = a; k < a + n; k++) {
            const int2 o = *(const int2 *)&sh.rec[k][3].z;
            r += o.y < hi || (o.y == hi && o.x < lo);
        }
        sh.rank[j] = (unsigned short)r;
        sh.ord[a + r] = (unsigned short)j;
    }
}

// Rotates, streams, keys and counts the np particles in shared memory; a record
// goes out when its place is back (one particle at a time: more warps per SM
// hide the round trip better than two particles per thread).
template <typename R, typename S, bool kMany>
__device__ __forceinline__ void bucket_move_all(const BucketTile<R, S> &sh, const BucketArgs<R> &A, int np)
{
    constexpr int Q = Bucket<R>::kChunks;
    const int t = threadIdx.x, lane = t & 31;
    const unsigned below = lanemask_lt();
    for (int jb = 0; jb < np; jb += S::kThreads) {
        const int j = jb + t;
        int4 rec[Q];
        int key = -1, base = 0;
        if (j < np) key = bucket_move<S>(sh, A, j, rec);
        const unsigned peers = __match_any_sync(0xffffffffu, key);
        const int lead = __ffs(peers) - 1;
        if (j < np && lane == lead) base = atomicAdd(A.out.count + key, __popc(peers));
        const int place = __shfl_sync(0xffffffffu, base, lead) + __popc(peers & below);
        if (j < np) {
            unsigned char *p = bucket_place<R, kMany>(A.out, key, place);
            store_record(p, rec[0], rec[1]);
            if constexpr (Q == 4) store_record(p + 32, rec[2], rec[3]);
        }
    }
}

// The particles of an over-full tile (more than fit in shared memory) as
// indices, cell by cell: ids[k] of a cell is its record k, or -1 - node for a
// record in the list.  Each of the tile's first SL threads lists one cell.
__device__ inline void bucket_list(const BucketGrid &g, int b, int n, int *ids)
{
    const int cap = n > 0 ? g.cap_of(b) : 0;
    for (int k = 0; k < min(n, cap); k++) ids[k] = k;
    int node = n > cap ? g.head[b] : -1;
    for (int k = cap; k < n; k++) {
        ids[k] = -1 - node;
        node = g.link[node];
    }
}
template <typename R>
__device__ inline const unsigned char *bucket_record(const BucketGrid &g, int b, int id)
{
    return id >= 0 ? g.rec + ((size_t)b * g.cap + id) * Bucket<R>::kBytes : g.pool + (size_t)(-1 - id) * Bucket<R>::kBytes;
}
// what a cell's particles are ordered by: FP32 idx, FP64 the order word
template <typename R>
__device__ inline unsigned long long bucket_order(const unsigned char *p)
{
    if constexpr (sizeof(R) == 4) return (unsigned long long)((const int *)p)[7];
    else return ((const unsigned long long *)p)[7];
}

// FP64: a run of cells of an over-full tile whose m particles ids[0, m) fit in shared
// memory; n: the particles of this thread's cell in the run, a: its first one.  In
// turn, cell by cell as below, a resting 48^3 fluid in one octant took 1074 us per
// interval for 347; the FP32 form, which has no ranks to make, gains nothing from it
// and its kernel would spill.
template <typename S>
__device__ __noinline__ void bucket_dense_run(BucketTile<double, S> &sh, const BucketArgs<double> &A, int b0, int n,
                                                 int a, int m, const int *ids)
{
    const int t = threadIdx.x;
    if (m == 0) return;
    if (t < S::kSlots) {
        sh.cstart[t] = a;
        sh.ccount[t] = n;
        if (n > 0) {
            const int slot = A.map.slot_of ? A.map.slot_of[b0 + t] : b0 + t;
            sh.slot[t] = slot;
            if (n > 1) {
                const CellRot<double> o = cell_rotation<double>(slot, A);
                for (int i = 0; i < 9; i++) sh.mat[t][4 * (i / 3) + i % 3] = o.m[i / 3][i % 3];
            }
            for (int k = 0; k < n; k++) sh.cell[a + k] = (unsigned char)t;
        }
    }
    __syncthreads();
    for (int j = t; j < m; j += S::kThreads) {
        const int4 *p = (const int4 *)bucket_record<double>(A.in, b0 + sh.cell[j], ids[j]);
#pragma unroll
        for (int q = 0; q < 4; q++) sh.rec[j][q] = p[q];
    }
    __syncthreads();
    bucket_rank<S>(sh, m);
    __syncthreads();
    bucket_means<S>(sh);
    __syncthreads();
    bucket_move_all<double, S, true>(sh, A, m);
}

// An over-full tile: cell by cell, the records read where they are; FP64 in runs
// of the next cells that fit in shared memory as long as there are any
template <typename R, typename S>
__device__ __noinline__ void bucket_dense_tile(BucketTile<R, S> &sh, const BucketArgs<R> &A, int b0, int n, int a, int np)
{
    constexpr int W = Bucket<R>::kBytes / 4, SL = S::kSlots, CAP = S::kCap;
    const int t = threadIdx.x;
    __shared__ int s_base, s_eff;
    __shared__ int s_first[SL + 1];  // each cell's first particle in the tile
    __shared__ unsigned long long s_sum[3];
    if (t == 0) {
        s_base = atomicAdd(A.in.n_pool + 3, np);
        s_first[SL] = np;
    }
    if (t < SL) s_first[t] = a;
    __syncthreads();
    int *ids = A.ids + s_base, *tmp = A.ids_tmp + s_base;
    if (t < SL) bucket_list(A.in, b0 + t, n, ids + a);
    int run = 1;
    for (int c = 0; c < SL; c += run) {
        const int f = s_first[c];
        if constexpr (sizeof(R) == 8) {
            // (its barrier also ends the run before)
            run = __syncthreads_count(t >= c && t < SL && a + n - f <= CAP);
            if (run > 0) {
                bucket_dense_run<S>(sh, A, b0, t >= c && t < c + run ? n : 0, a - f, s_first[c + run] - f, ids + f);
                continue;
            }
        }
        run = 1;
        const int m = s_first[c + 1] - f, b = b0 + c;
        if (m == 0) continue;
        int *id = ids + f;
        const int slot = A.map.slot_of ? A.map.slot_of[b] : b;
        if (t < 3) s_sum[t] = 0;
        if (t == 0) s_eff = 0;
        __syncthreads();
        int n_eff = 0;
        R lv[3] = {0, 0, 0};
        if constexpr (sizeof(R) == 4) {
            long long s[3] = {0, 0, 0};
            for (int k = t; k < m; k += S::kThreads) {
                const float *v = (const float *)bucket_record<R>(A.in, b, id[k]);
                if (((const int *)v)[3] > 0) {
                    for (int i = 0; i < 3; i++) s[i] += to_fixed(v[i]);
                    n_eff++;
                }
            }
            for (int i = 0; i < 3; i++) atomicAdd(&s_sum[i], (unsigned long long)s[i]);
            atomicAdd(&s_eff, n_eff);
            __syncthreads();
            n_eff = s_eff;
            if (n_eff > 1)
                for (int i = 0; i < 3; i++) lv[i] = fixed_mean((long long)s_sum[i], n_eff);
        } else {
            block_merge_sort(id, tmp + f, m,
                             [&](int q) { return bucket_order<R>(bucket_record<R>(A.in, b, q)); });
            if (t < 3) {
                double s = 0;
                for (int k = 0; k < m; k++) {
                    const double *v = (const double *)bucket_record<R>(A.in, b, id[k]);
                    if (((const int *)v)[6] > 0) {
                        s = s + v[t];
                        n_eff++;
                    }
                }
                s_sum[t] = (unsigned long long)__double_as_longlong(n_eff > 1 ? s / n_eff : 0.0);
                if (t == 0) s_eff = n_eff;
            }
            __syncthreads();
            n_eff = s_eff;
            for (int i = 0; i < 3; i++) lv[i] = __longlong_as_double((long long)s_sum[i]);
        }
        CellRot<R> rot;
        if (n_eff > 1) rot = cell_rotation<R>(slot, A);
        for (int k = t; k < m; k += S::kThreads) {
            alignas(16) int w[W];
            const int *p = (const int *)bucket_record<R>(A.in, b, id[k]);
            for (int i = 0; i < W; i++) w[i] = p[i];
            R *v = (R *)w, *x = (R *)w + 4;
            if (n_eff > 1) cell_rotate(v[0], v[1], v[2], lv, rot);
            const int key = bucket_stream_values<R>(A, x[0], x[1], x[2], v[0], v[1], v[2], w[7]);
            if constexpr (sizeof(R) == 8) {
                w[14] = k;
                w[15] = slot;
            }
            int *o = (int *)bucket_place<R, true>(A.out, key, atomicAdd(A.out.count + key, 1));
            for (int i = 0; i < W; i++) o[i] = w[i];
        }
        __syncthreads();
    }
}

// The tile's records into shared memory: thread t < kSlots starts the copy of
// cell t's n records to place a (records beyond the bucket are fetched from its
// list) and notes the particles' cell.  bucket_arrived has to follow.
template <typename R, typename S>
__device__ __forceinline__ void bucket_load(BucketTile<R, S> &sh, const BucketGrid &g, int b, int n, int a)
{
    constexpr int B = Bucket<R>::kBytes;
    if (threadIdx.x >= S::kSlots) return;
    const int mb = n > 0 ? min(n, g.cap_of(b)) : 0;
    mbar_arrive_expect_tx(&sh.bar, mb * B);
    if (mb) bulk_copy_to_smem(&sh.rec[a][0], g.rec + (size_t)b * g.cap * B, mb * B, &sh.bar);
    sh.cstart[threadIdx.x] = a;
    sh.ccount[threadIdx.x] = n;
    for (int k = 0; k < n; k++) sh.cell[a + k] = (unsigned char)threadIdx.x;
    if (n > mb) {
        int node = g.head[b];
        for (int k = mb; k < n; k++) {
            const int4 *p = (const int4 *)(g.pool + (size_t)node * B);
            for (int q = 0; q < B / 16; q++) sh.rec[a + k][q] = p[q];
            node = g.link[node];
        }
    }
}

// Waits for the copies of bucket_load, with a barrier.  Copies that do not
// arrive in time are reported, and their records loaded directly; a late copy
// brings the same values, which nothing changes in shared memory, and the block
// waits for it again before it exits (bucket_drained).
template <typename R, typename S>
__device__ __forceinline__ bool bucket_arrived(BucketTile<R, S> &sh, const BucketGrid &g, int b, int n, int a,
                                               unsigned *err)
{
    const int late = !mbar_wait_bounded(&sh.bar, 0, kBulkPolls);
    if (!__syncthreads_or(late)) return true;
    if (late) atomicOr(err, DEV_ERR_BULK_WAIT);
    if (threadIdx.x < S::kSlots && n > 0) {
        const int mb = min(n, g.cap_of(b));
        const int4 *p = (const int4 *)(g.rec + (size_t)b * g.cap * Bucket<R>::kBytes);
        for (int q = 0; q < mb * Bucket<R>::kChunks; q++) (&sh.rec[a][0])[q] = p[q];
    }
    __syncthreads();
    return false;
}

template <typename R, typename S>
__device__ __forceinline__ void bucket_drained(BucketTile<R, S> &sh, bool arrived, unsigned *err)
{
    if (!arrived && !mbar_wait_bounded(&sh.bar, 0, kBulkPolls)) atomicOr(err, DEV_ERR_BULK_UNDRAINED);
}

// Bound by the round trips of each particle (cell table, counting atomic), the
// load/store pipe (69 % of its cycles at 128x64x64 FP32) and issue (67 %), not by HBM
// (3.4 TB/s at 128^3), so occupancy decides: one particle per thread in flight,
// 40 registers, 48 warps per SM (two per thread with 32 warps: 128^3 FP32 566 us
// for 531).  With the cell's collision on one thread per cell, copies by cp.async
// and the moved records put back in shared memory, 64^3 FP32 took 94 us for 78,
// and 72 % of the load/store pipe.
template <typename R, typename S>
__global__ void __launch_bounds__(S::kThreads, S::kMinBlocks) k_bucket_interval(const __grid_constant__ BucketArgs<R> A)
{
    constexpr int SL = S::kSlots, CAP = S::kCap;
    static_assert(SL <= 256 && CAP <= 65535, "tile-local indices");
    extern __shared__ __align__(16) unsigned char smem[];
    BucketTile<R, S> &sh = *reinterpret_cast<BucketTile<R, S> *>(smem);
    const int t = threadIdx.x, lane = t & 31;
    const int b0 = blockIdx.x * SL, b = b0 + t;
    // the last warps draw the cells' rotations: thread t that of cell c
    const int c = S::kThreads - 1 - t;
    int n = 0, nc = 0;
    if (t == 0) mbar_init(&sh.bar, SL);
    if (c < SL && b0 + c < A.S) nc = A.in.count[b0 + c];
    if (t < SL && b < A.S) {
        n = A.in.count[b];
        A.count_clear[b] = 0;
        A.head_clear[b] = -1;
    }
    if (blockIdx.x == 0 && t == 0) A.n_pool_clear[0] = A.n_pool_clear[3] = 0;
    int np;
    const int a = tile_scan<S::kThreads>(n, sh.wsum, np);
    if (np == 0) return;
    auto slot_of_bucket = [&](int q) { return A.map.slot_of ? A.map.slot_of[q] : q; };
    if (np > CAP) {
        bucket_dense_tile<R, S>(sh, A, b0, n, a, np);
        return;
    }
    bucket_load<R, S>(sh, A.in, b, n, a);
    if (nc > 0) {
        const int s = slot_of_bucket(b0 + c);
        if constexpr (sizeof(R) == 8) sh.slot[c] = s;
        if (nc > 1) {
            const CellRot<R> o = cell_rotation<R>(s, A);
#pragma unroll
            for (int i = 0; i < 9; i++) sh.mat[c][4 * (i / 3) + i % 3] = o.m[i / 3][i % 3];
        }
    }
    const bool arrived = bucket_arrived<R, S>(sh, A.in, b, n, a, A.err);
    if constexpr (sizeof(R) == 8) {
        bucket_rank<S>(sh, np);
        __syncthreads();
    }
    bucket_means<S>(sh);
    __syncthreads();
    bucket_move_all<R, S, false>(sh, A, np);
    bucket_drained<R, S>(sh, arrived, A.err);
}

// The sorted SoA arrays into the buckets of the current grid, whose counts
// are those of the slots; clears the counts and lists of the next one.  A warp
// per slot in turn; FP64 order = place.
template <typename R>
__global__ void __launch_bounds__(kFusedThreads)
    k_soa_to_buckets(PView<R> v, BucketGrid g, BucketMap map, int S, const int *__restrict__ count,
                     const int *__restrict__ start, int *count_next, int *head_next, int *n_pool_next)
{
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * kFusedThreads + threadIdx.x) >> 5, warps = gridDim.x * (kFusedThreads / 32);
    if (blockIdx.x == 0 && threadIdx.x == 0) n_pool_next[0] = n_pool_next[3] = 0;
    for (int s = blockIdx.x * kFusedThreads + threadIdx.x; s < S; s += gridDim.x * kFusedThreads) {
        count_next[s] = 0;
        head_next[s] = -1;
    }
    for (int s = warp; s < S; s += warps) {
        const int n = count[s], a = start[s];
        const int b = map.of_slot ? map.of_slot[s] : s, cap = g.cap_of(b);
        int last = -1;  // the list of the slot, built by this warp alone
        for (int k0 = 0; k0 < n; k0 += 32) {
            const int k = k0 + lane, i = a + k;
            int node = -1;
            if (k < n && k >= cap) node = atomicAdd(g.n_pool, 1);
            if (k < n) {
                unsigned char *p = k < cap ? g.rec + ((size_t)b * g.cap + k) * Bucket<R>::kBytes
                                           : g.pool + (size_t)node * Bucket<R>::kBytes;
                if constexpr (sizeof(R) == 4) {
                    store_record(p, make_int4(__float_as_int(v.vel.x[i]), __float_as_int(v.vel.y[i]),
                                              __float_as_int(v.vel.z[i]), v.species[i]),
                                 make_int4(__float_as_int(v.pos.x[i]), __float_as_int(v.pos.y[i]),
                                           __float_as_int(v.pos.z[i]), i));
                } else {
                    const double vz = v.vel.z[i], pz = v.pos.z[i];
                    store_record(p, as_int4(v.vel.x[i], v.vel.y[i]),
                                 make_int4(__double2loint(vz), __double2hiint(vz), v.species[i], i));
                    store_record(p + 32, as_int4(v.pos.x[i], v.pos.y[i]),
                                 make_int4(__double2loint(pz), __double2hiint(pz), k, s));
                }
            }
            if (k0 + 32 > cap) {
                for (int l = 0; l < 32; l++) {
                    const int nd = __shfl_sync(0xffffffffu, node, l);
                    if (nd < 0) continue;
                    if (lane == 0) g.link[nd] = last;
                    last = nd;
                }
            }
        }
        if (lane == 0) {
            g.count[b] = n;
            g.head[b] = last;
        }
    }
}

// counts by bucket -> counts by slot
__global__ void k_bucket_counts_to_slots(const int *__restrict__ by_bucket, const int *__restrict__ slot_of, int S,
                                         int *__restrict__ by_slot)
{
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < S; b += gridDim.x * blockDim.x)
        by_slot[slot_of[b]] = by_bucket[b];
}

// The buckets of the final grid into the API arrays, each cell's particles in
// order: FP32 by their position when the run started (a canonical order, since
// the intervals keep none), FP64 by their order words.  image, flags and id
// come from the position-at-start idx.
template <typename R, typename S>
__global__ void __launch_bounds__(S::kThreads, S::kMinBlocks)
    k_buckets_to_soa(BucketGrid g, BucketMap map, int S_, const int *__restrict__ count,
                     const int *__restrict__ start, PView<R> side, PView<R> d, int *ids, int *ids_tmp,
                     unsigned *err)
{
    constexpr int SL = S::kSlots, CAP = S::kCap;
    extern __shared__ __align__(16) unsigned char smem[];
    BucketTile<R, S> &sh = *reinterpret_cast<BucketTile<R, S> *>(smem);
    const int t = threadIdx.x;
    const int b0 = blockIdx.x * SL, b = b0 + t;
    const int slot = t < SL && b < S_ ? (map.slot_of ? map.slot_of[b] : b) : -1;
    const int n = slot >= 0 ? count[slot] : 0;  // counts and starts are those of the slots
    if (t == 0) mbar_init(&sh.bar, SL);
    // each cell's first place in the sorted arrays
    __shared__ int s_out[SL];
    int np;
    const int a = tile_scan<S::kThreads>(n, sh.wsum, np);
    if (t < SL) s_out[t] = slot >= 0 ? start[slot] : 0;
    auto side_fields = [&](int j, int idx) {
        d.ix[j] = side.ix[idx];
        d.iy[j] = side.iy[idx];
        d.iz[j] = side.iz[idx];
        d.flags[j] = side.flags[idx];
        d.id[j] = side.id[idx];
    };
    if (np > CAP) {
        // over-full: each cell's indices are put in order in its own range of ids
        if (t < SL) {
            sh.ccount[t] = n;
            bucket_list(g, b, n, ids + s_out[t]);
        }
        __syncthreads();
        for (int c = 0; c < SL; c++) {
            const int m = sh.ccount[c];
            int *id = ids + s_out[c];
            block_merge_sort(id, ids_tmp + s_out[c], m,
                             [&](int q) { return bucket_order<R>(bucket_record<R>(g, b0 + c, q)); });
            for (int k = t; k < m; k += S::kThreads) {
                const int j = s_out[c] + k;
                const unsigned char *p = bucket_record<R>(g, b0 + c, id[k]);
                const R *w = (const R *)p;
                d.vel.x[j] = w[0];
                d.vel.y[j] = w[1];
                d.vel.z[j] = w[2];
                d.pos.x[j] = w[4];
                d.pos.y[j] = w[5];
                d.pos.z[j] = w[6];
                d.species[j] = ((const int *)p)[sizeof(R) == 4 ? 3 : 6];
                side_fields(j, ((const int *)p)[7]);
            }
        }
        return;
    }
    if (np == 0) return;
    bucket_load<R, S>(sh, g, b, n, a);
    const bool arrived = bucket_arrived<R, S>(sh, g, b, n, a, err);
    if constexpr (sizeof(R) == 8) {
        bucket_rank<S>(sh, np);
        __syncthreads();
        for (int q = t; q < np; q += S::kThreads) {
            const int j = sh.ord[q];
            const int c = sh.cell[j], o = s_out[c] + sh.rank[j];
            const double2 v = as_double2(sh.rec[j][0]), p = as_double2(sh.rec[j][2]);
            const int4 c1 = sh.rec[j][1], c3 = sh.rec[j][3];
            d.vel.x[o] = v.x;
            d.vel.y[o] = v.y;
            d.vel.z[o] = __hiloint2double(c1.y, c1.x);
            d.pos.x[o] = p.x;
            d.pos.y[o] = p.y;
            d.pos.z[o] = __hiloint2double(c3.y, c3.x);
            d.species[o] = c1.z;
            side_fields(o, c1.w);
        }
    } else {
        // a warp per slot: lane l holds record l, its place is its idx's rank
        const int lane = t & 31;
        for (int c = t >> 5; c < SL; c += S::kThreads / 32) {
            const int m = sh.ccount[c], st = sh.cstart[c];
            for (int k = lane; k < m; k += 32) {
                const int4 c0 = sh.rec[st + k][0], c1 = sh.rec[st + k][1];
                int r = 0;
                for (int q = 0; q < m; q++) r += sh.rec[st + q][1].w < c1.w;
                const int o = s_out[c] + r;
                d.vel.x[o] = __int_as_float(c0.x);
                d.vel.y[o] = __int_as_float(c0.y);
                d.vel.z[o] = __int_as_float(c0.z);
                d.pos.x[o] = __int_as_float(c1.x);
                d.pos.y[o] = __int_as_float(c1.y);
                d.pos.z[o] = __int_as_float(c1.z);
                d.species[o] = c0.w;
                side_fields(o, c1.w);
            }
        }
    }
    bucket_drained<R, S>(sh, arrived, err);
}

}  // namespace rmpcd
