// MPCD on the GPU (src/mpcd.f90): SRD and MPC-AT collisions, the Lamura wall
// rule, temperature, cell rescaling, streaming with periodic and wall
// boundaries, and bulk reactions.  Collisions run one thread per Hilbert
// slot over the sorted particle ranges (cells hold ~10 particles), staged in
// shared memory tile by tile.
#include <cmath>

#include "cellops.cuh"
#include "hilbert.cuh"
#include "keys.cuh"
#include "rng.cuh"
#include "stepops.cuh"
#include "timers.cuh"

namespace rmpcd {

// The collision kernels below work on tiles of up to kCellTile consecutive slots,
// whose particles are one contiguous range: the block brings the range's
// velocities and species into shared memory with coalesced loads, one thread
// per slot runs the cell's sequential sums and updates there, and the block
// writes the velocities back coalesced.  A thread per slot on global memory
// touches 32 cells' ranges per warp load (64^3 at density 10: 79 us FP64 for
// the SRD step against 30 us of HBM traffic); the cell's own chain of adds
// then sets its pace.  64 slots per 128-thread block leave 8 (FP64) or 16
// (FP32) blocks per SM, so that one block's loads overlap another's sums; a
// denser fluid's tiles have the slots that kCellCap holds (cell_tile).
//
// A tile of an uneven fluid with more than kCellCap particles takes the same cell
// bodies on global memory.  Two FP64 kernels with long cell bodies, whose staging
// leaves too few threads per SM for that, go run by run instead, each the next cells
// that fit, when no cell has more than kRunCell particles (48^3 fluid in one octant,
// MPC-AT step: 153 us, 278 on global memory; in the SRD kernel the second copy of
// the body costs registers, 27 us for 23 at density 10).
constexpr int kCellTile = 64;
constexpr int kCellThreads = 128;
constexpr int kCellCap = 832;
constexpr int kRunCell = kCellCap / 5;

struct CellRange {
    int n, a;          // this thread's cell: particles, first particle (n = 0: no cell)
    int a0, np;        // the tile's particles
    int s0, cells;     // the tile's slots
    __device__ CellRange(const int *__restrict__ count, const int *__restrict__ start, int S, int per)
    {
        s0 = blockIdx.x * per;
        cells = min(per, S - s0);
        const int s = s0 + (int)threadIdx.x, last = s0 + cells - 1;
        n = 0;
        a = 0;
        if ((int)threadIdx.x < cells) {
            n = count[s];
            a = start[s];
        }
        a0 = start[s0];
        np = start[last] + count[last] - a0;
    }
};

// The cells of a tile: run(n, a, a0, np) for the particles [a0, a0 + np) in shared
// memory, called by every thread, with the thread's cell, n = 0 when that is not
// of the run; direct() by the threads of a tile that takes its cells on global
// memory.  Returns the sum of the thread's results.
template <bool kRuns, typename Run, typename Direct>
__device__ __forceinline__ double cell_bodies(const CellRange &c, const int *__restrict__ count,
                                              const int *__restrict__ start, Run run, Direct direct)
{
    if (c.np <= kCellCap) return run(c.n, c.a - c.a0, c.a0, c.np);
    if constexpr (kRuns) {
        if (!__syncthreads_or(c.n > kRunCell)) {
            const int t = threadIdx.x;
            double r = 0;
            for (int c0 = 0, k; c0 < c.cells; c0 += k) {
                const int a0 = start[c.s0 + c0];
                // (its barrier also ends the run before)
                k = __syncthreads_count(t >= c0 && t < c.cells && c.a + c.n - a0 <= kCellCap);
                const int last = c.s0 + c0 + k - 1;
                r += run(t >= c0 && t < c0 + k ? c.n : 0, c.a - a0, a0, start[last] + count[last] - a0);
            }
            return r;
        }
    }
    return c.n > 0 ? direct() : 0;
}

// K arrays src[k][a0 .. a0 + np) to or from rows of kCellCap of shared memory
template <typename T, int K>
__device__ __forceinline__ void tile_in(T (*dst)[kCellCap], const T *const (&src)[K], int a0, int np)
{
#pragma unroll 2
    for (int j = threadIdx.x; j < np; j += kCellThreads) {
#pragma unroll
        for (int k = 0; k < K; k++) dst[k][j] = src[k][a0 + j];
    }
}
template <typename T, int K>
__device__ __forceinline__ void tile_out(T *const (&dst)[K], T (*src)[kCellCap], int a0, int np)
{
#pragma unroll 2
    for (int j = threadIdx.x; j < np; j += kCellThreads) {
#pragma unroll
        for (int k = 0; k < K; k++) dst[k][a0 + j] = src[k][j];
    }
}

// simple_mpcd_step, src/mpcd.f90:71-183
template <typename R, bool kStaged>
__global__ void __launch_bounds__(kCellThreads)
    k_simple_mpcd(const int *__restrict__ count, const int *__restrict__ start, int S, int per, R *vx, R *vy, R *vz,
                  const int *__restrict__ species, SrdParams q)
{
    const long long slot = (long long)blockIdx.x * (kStaged ? per : kCellThreads) + threadIdx.x;
    if constexpr (!kStaged) {
        if (slot < S) srd_slot<R>(count[slot], start[slot], slot, 0, vx, vy, vz, species, q);
    } else {
        __shared__ R sv[3][kCellCap];
        __shared__ int ss[1][kCellCap];
        const CellRange c(count, start, S, per);
        auto run = [=](int n, int a, int a0, int np) {
            tile_in<R, 3>(sv, {vx, vy, vz}, a0, np);
            tile_in<int, 1>(ss, {species}, a0, np);
            __syncthreads();
            srd_slot<R>(n, a, slot, -(long long)a0, sv[0], sv[1], sv[2], ss[0], q);
            __syncthreads();
            tile_out<R, 3>({vx, vy, vz}, sv, a0, np);
            return 0.0;
        };
        auto direct = [=] {
            srd_slot<R>(c.n, c.a, slot, 0, vx, vy, vz, species, q);
            return 0.0;
        };
        cell_bodies<false>(c, count, start, run, direct);
    }
}

// The MPC-AT normals of simple_mpcd_step (src/mpcd.f90:144-160) and
// wall_mpcd_step (:268-290): for every particle i with species > 0 (for every
// particle when species is null), (R)(rng::normal(seed, step, i, k) * t_factor)
// for k = 0, 1, 2 into n[k][i].  Each deviate is the first accepted of the
// attempts t = 0, 1, ... of rng::normal, so the values are rng::normal's.  A
// warp takes kAtChunks chunks of 32 particles at a time and deals the
// attempts of their deviates to its lanes: first every lane's attempt 0 of
// its particles' deviates, then the attempts that rejections queue in a ring
// in shared memory, 32 at a time, so no lane waits while another repeats a
// rejection (a deviate drawn by one thread costs its warp the slowest lane's
// attempts) and the last few rejections of a pass leave few lanes idle.
constexpr int kAtThreads = 256;
constexpr int kAtChunks = 8;    // 32-particle chunks per warp pass
constexpr int kAtQueue = 1024;  // ring of queued attempts per warp: at least 96 * kAtChunks

__device__ inline unsigned at_job(int p, int k, int t) { return (unsigned)p | ((unsigned)k << 8) | ((unsigned)t << 10); }

template <typename R>
__global__ void __launch_bounds__(kAtThreads) k_at_normals(const int *__restrict__ species, long long N, SrdParams q,
                                                           R *nx, R *ny, R *nz)
{
    static_assert(kAtChunks * 32 <= 256 && 96 * kAtChunks <= kAtQueue && (kAtQueue & (kAtQueue - 1)) == 0,
                  "job fields and ring size");
    __shared__ unsigned ring[kAtThreads / 32][kAtQueue];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned below = lanemask_lt();
    unsigned *qr = ring[w];
    R *out[3] = {nx, ny, nz};
    const long long warps = (long long)gridDim.x * (kAtThreads / 32);
    const long long span = 32LL * kAtChunks;
    for (long long base = ((long long)blockIdx.x * (kAtThreads / 32) + w) * span; base < N; base += warps * span) {
        // round 0: every lane the attempt 0 of its own particles' deviates
        int tail = 0;
        for (int c = 0; c < kAtChunks; c++) {
            const long long i = base + c * 32 + lane;
            const bool act = i < N && (!species || species[i] > 0);
            for (int k = 0; k < 3; k++) {
                double z = 0;
                const bool ok = act && rng::normal_attempt(q.seed, q.step, (uint32_t)i, (uint32_t)k, 0u, &z);
                if (ok) out[k][i] = (R)(z * q.t_factor);
                const unsigned rej = __ballot_sync(0xffffffffu, act && !ok);
                if (act && !ok) qr[(tail + __popc(rej & below)) & (kAtQueue - 1)] = at_job(c * 32 + lane, k, 1);
                tail += __popc(rej);
            }
        }
        __syncwarp();
        // then the queued attempts, 32 at a time; a rejected one queues the
        // deviate's next attempt behind the others (at most 96 * kAtChunks
        // are queued at once, so the ring never overwrites an unread one)
        int head = 0;
        while (head < tail) {
            const int n = min(32, tail - head);
            const bool have = lane < n;
            const unsigned jb = have ? qr[(head + lane) & (kAtQueue - 1)] : 0u;
            head += n;
            const int p = jb & 255, k = (jb >> 8) & 3, t = (int)(jb >> 10);
            const long long ii = base + p;
            double z = 0;
            bool ok = false;
            if (have) {
                // rng::normal gives 0 once its attempts are spent
                ok = t >= (int)rng::kNormalAttempts ||
                     rng::normal_attempt(q.seed, q.step, (uint32_t)ii, (uint32_t)k, (uint32_t)t, &z);
                if (ok) out[k][ii] = (R)(z * q.t_factor);
            }
            const unsigned rej = __ballot_sync(0xffffffffu, have && !ok);
            if (have && !ok) qr[(tail + __popc(rej & below)) & (kAtQueue - 1)] = at_job(p, k, t + 1);
            tail += __popc(rej);
            __syncwarp();
        }
    }
}

// the thermostat branch of srd_slot (src/mpcd.f90:126-160) for the n
// particles from a, with each normal read instead of drawn; vel = normal + dv
// (hydro) or the normal, as srd_slot's store and later add
template <typename R>
__device__ __forceinline__ void at_cell(int n, int a, R *vx, R *vy, R *vz, const int *species, int hydro,
                                        const R *nx, const R *ny, const R *nz)
{
    if (n <= 1) return;
    int n_eff = 0;
    CellSum<R> sx, sy, sz, wx, wy, wz;
    for (int i = a; i < a + n; i++) {
        if (species[i] > 0) {
            sx.add(vx[i]);
            sy.add(vy[i]);
            sz.add(vz[i]);
            wx.add(nx[i]);
            wy.add(ny[i]);
            wz.add(nz[i]);
            n_eff++;
        }
    }
    if (n_eff <= 1) return;
    const R lv[3] = {sx.value() / n_eff, sy.value() / n_eff, sz.value() / n_eff};
    const R dv[3] = {lv[0] - wx.value() / n_eff, lv[1] - wy.value() / n_eff, lv[2] - wz.value() / n_eff};
    for (int i = a; i < a + n; i++) {
        if (species[i] <= 0) continue;
        vx[i] = hydro ? nx[i] + dv[0] : nx[i];
        vy[i] = hydro ? ny[i] + dv[1] : ny[i];
        vz[i] = hydro ? nz[i] + dv[2] : nz[i];
    }
}

// simple_mpcd_step with the MPC-AT thermostat given the normals of
// k_at_normals
template <typename R, bool kStaged>
__global__ void __launch_bounds__(kCellThreads)
    k_at_cells(const int *__restrict__ count, const int *__restrict__ start, int S, int per, R *vx, R *vy, R *vz,
               const int *__restrict__ species, int hydro, const R *__restrict__ nx, const R *__restrict__ ny,
               const R *__restrict__ nz)
{
    if constexpr (!kStaged) {
        const long long slot = (long long)blockIdx.x * kCellThreads + threadIdx.x;
        if (slot < S) at_cell<R>(count[slot], start[slot], vx, vy, vz, species, hydro, nx, ny, nz);
    } else {
        __shared__ R sv[6][kCellCap];
        __shared__ int ss[1][kCellCap];
        const CellRange c(count, start, S, per);
        auto run = [=](int n, int a, int a0, int np) {
            tile_in<R, 6>(sv, {vx, vy, vz, nx, ny, nz}, a0, np);
            tile_in<int, 1>(ss, {species}, a0, np);
            __syncthreads();
            at_cell<R>(n, a, sv[0], sv[1], sv[2], ss[0], hydro, sv[3], sv[4], sv[5]);
            __syncthreads();
            tile_out<R, 3>({vx, vy, vz}, sv, a0, np);
            return 0.0;
        };
        auto direct = [=] {
            at_cell<R>(c.n, c.a, vx, vy, vz, species, hydro, nx, ny, nz);
            return 0.0;
        };
        cell_bodies<sizeof(R) == 8>(c, count, start, run, direct);
    }
}

struct WallArgs {
    int M0, M1, M2, L2;
    int has_wall;
    double wt0, wt1;
    int wn0, wn1;
    int do_cell_v;
};

// wall_mpcd_step of slot s (src/mpcd.f90:193-337), its n particles from a;
// with the thermostat, nx, ny, nz hold the particles' normals
template <typename R>
__device__ __forceinline__ void wall_cell(int n, int a, int s, R *vx, R *vy, R *vz, const R *nx, const R *ny,
                                          const R *nz, const SrdParams &q, const WallArgs &w)
{
    if (n <= 1) return;
    const int M[3] = {w.M0, w.M1, w.M2};
    int cell[3];
    hilbert::compact_point(s, M, cell);
    int wall_idx = -1;
    if (w.has_wall && cell[2] + 1 == 1) wall_idx = 0;
    else if (w.has_wall && cell[2] + 1 == w.L2) wall_idx = 1;
    int n_virtual = 0;
    double vv[3] = {0, 0, 0};
    int wn = wall_idx == 0 ? w.wn0 : w.wn1;
    if (wall_idx >= 0 && n < wn) {
        n_virtual = wn - n;
        for (int k = 0; k < 3; k++) vv[k] = rng::normal(q.seed, q.step, (uint32_t)s, (uint32_t)(3 + k));
        double f = sqrt(n_virtual * (wall_idx == 0 ? w.wt0 : w.wt1));
        for (int k = 0; k < 3; k++) vv[k] = vv[k] * f;
    }
    CellSum<R> sx, sy, sz;
    for (int i = a; i < a + n; i++) {
        sx.add(vx[i]);
        sy.add(vy[i]);
        sz.add(vz[i]);
    }
    R lv[3];
    if (n_virtual > 0) {
        lv[0] = (R)(((double)sx.value() + vv[0]) / wn);
        lv[1] = (R)(((double)sy.value() + vv[1]) / wn);
        lv[2] = (R)(((double)sz.value() + vv[2]) / wn);
    } else {
        lv[0] = sx.value() / n;
        lv[1] = sy.value() / n;
        lv[2] = sz.value() / n;
    }
    if (q.thermostat) {
        R dv[3] = {0, 0, 0};
        if (w.do_cell_v) {
            CellSum<R> wx, wy, wz;
            for (int i = a; i < a + n; i++) {
                wx.add(nx[i]);
                wy.add(ny[i]);
                wz.add(nz[i]);
            }
            dv[0] = lv[0] - wx.value() / (R)n;
            dv[1] = lv[1] - wy.value() / (R)n;
            dv[2] = lv[2] - wz.value() / (R)n;
        }
        for (int i = a; i < a + n; i++) {
            vx[i] = w.do_cell_v ? nx[i] + dv[0] : nx[i];
            vy[i] = w.do_cell_v ? ny[i] + dv[1] : ny[i];
            vz[i] = w.do_cell_v ? nz[i] + dv[2] : nz[i];
        }
    } else {
        double n0, n1, n2;
        rng::sphere(q.seed, q.step, (uint32_t)s, n0, n1, n2);
        Rot o = srd_matrix(n0, n1, n2, q.sin_a, q.cos_a);
        for (int i = a; i < a + n; i++) {
            R x = vx[i], y = vy[i], z = vz[i];
            srd_rotate(x, y, z, lv, o);
            vx[i] = x;
            vy[i] = y;
            vz[i] = z;
        }
    }
}

// wall_mpcd_step, src/mpcd.f90:193-337.  kAT: the thermostat's normals come
// from k_at_normals, which deals the rejection attempts of a whole warp to its
// lanes; drawn inside the cell loop they took a 1.2 M particle channel (FP64)
// 148 us, one thread per cell.
template <typename R, bool kAT, bool kStaged>
__global__ void __launch_bounds__(kCellThreads)
    k_wall_mpcd(const int *__restrict__ count, const int *__restrict__ start, int S, int per, R *vx, R *vy, R *vz,
                const R *__restrict__ nx, const R *__restrict__ ny, const R *__restrict__ nz, SrdParams q, WallArgs w)
{
    const int slot = blockIdx.x * (kStaged ? per : kCellThreads) + (int)threadIdx.x;
    if constexpr (!kStaged) {
        if (slot < S) wall_cell<R>(count[slot], start[slot], slot, vx, vy, vz, nx, ny, nz, q, w);
    } else {
        __shared__ R sv[kAT ? 6 : 3][kCellCap];
        const CellRange c(count, start, S, per);
        auto run = [=](int n, int a, int a0, int np) {
            if constexpr (kAT) tile_in<R, 6>(sv, {vx, vy, vz, nx, ny, nz}, a0, np);
            else tile_in<R, 3>(sv, {vx, vy, vz}, a0, np);
            __syncthreads();
            wall_cell<R>(n, a, slot, sv[0], sv[1], sv[2], sv[kAT ? 3 : 0], sv[kAT ? 4 : 1], sv[kAT ? 5 : 2], q, w);
            __syncthreads();
            tile_out<R, 3>({vx, vy, vz}, sv, a0, np);
            return 0.0;
        };
        auto direct = [=] {
            wall_cell<R>(c.n, c.a, slot, vx, vy, vz, nx, ny, nz, q, w);
            return 0.0;
        };
        cell_bodies<false>(c, count, start, run, direct);
    }
}

// compute_temperature, src/mpcd.f90:342-407, of the n particles from a: the
// cell's contribution to the sum of temperatures (0 for cells that add none)
template <typename R>
__device__ __forceinline__ double cell_temperature(int n, int a, const R *vx, const R *vy, const R *vz,
                                                   const int *species)
{
    if (n <= 1) return 0;
    int n_eff = 0;
    CellSum<R> sx, sy, sz;
    for (int i = a; i < a + n; i++) {
        if (species[i] > 0) {
            sx.add(vx[i]);
            sy.add(vy[i]);
            sz.add(vz[i]);
            n_eff++;
        }
    }
    if (n_eff <= 1) return 0;
    // local_v = local_v / n  (divides by n, not n_effective, as written)
    double l0 = (double)(sx.value() / (R)n), l1 = (double)(sy.value() / (R)n), l2 = (double)(sz.value() / (R)n);
    double kin = 0;
    for (int i = a; i < a + n; i++) {
        if (species[i] > 0) {
            double d0 = (double)vx[i] - l0, d1 = (double)vy[i] - l1, d2 = (double)vz[i] - l2;
            kin = kin + (d0 * d0 + d1 * d1 + d2 * d2);
        }
    }
    return kin / (double)(3 * (n_eff - 1));
}

// per-block partial sums (te, count) over the block's cells, for the fixed-order
// sum of k_temperature_final
template <typename R, bool kStaged>
__global__ void __launch_bounds__(kCellThreads)
    k_temperature(const int *__restrict__ count, const int *__restrict__ start, int S, int per, const R *vx,
                  const R *vy, const R *vz, const int *__restrict__ species, double *part)
{
    double te = 0, cnt = 0;
    if constexpr (!kStaged) {
        const long long slot = (long long)blockIdx.x * kCellThreads + threadIdx.x;
        if (slot < S) {
            te = cell_temperature<R>(count[slot], start[slot], vx, vy, vz, species);
            cnt = count[slot] > 1 ? 1 : 0;
        }
    } else {
        __shared__ R sv[3][kCellCap];
        __shared__ int ss[1][kCellCap];
        const CellRange c(count, start, S, per);
        auto run = [=](int n, int a, int a0, int np) {
            tile_in<R, 3>(sv, {vx, vy, vz}, a0, np);
            tile_in<int, 1>(ss, {species}, a0, np);
            __syncthreads();
            return cell_temperature<R>(n, a, sv[0], sv[1], sv[2], ss[0]);
        };
        auto direct = [=] { return cell_temperature<R>(c.n, c.a, vx, vy, vz, species); };
        te = cell_bodies<false>(c, count, start, run, direct);
        cnt = c.n > 1 ? 1 : 0;
    }
    constexpr int W = kCellThreads / 32;
    __shared__ double s_te[W], s_cnt[W];
    for (int o = 16; o > 0; o >>= 1) {
        te += __shfl_xor_sync(0xffffffffu, te, o);
        cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    }
    if ((threadIdx.x & 31) == 0) {
        s_te[threadIdx.x >> 5] = te;
        s_cnt[threadIdx.x >> 5] = cnt;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        // (a tile's 64 slots are the first two warps')
        for (int w = 1; w < W; w++) {
            te += s_te[w];
            cnt += s_cnt[w];
        }
        part[2 * (size_t)blockIdx.x] = te;
        part[2 * (size_t)blockIdx.x + 1] = cnt;
    }
}

// one block: the partials by a fixed tree (thread t adds t, t + 1024, ...)
__global__ void __launch_bounds__(1024) k_temperature_final(const double *part, int nb, double *out)
{
    __shared__ double ste[32], sc[32];
    double te = 0, cnt = 0;
    for (int b = threadIdx.x; b < nb; b += 1024) {
        te += part[2 * (size_t)b];
        cnt += part[2 * (size_t)b + 1];
    }
    for (int o = 16; o > 0; o >>= 1) {
        te += __shfl_xor_sync(0xffffffffu, te, o);
        cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    }
    if ((threadIdx.x & 31) == 0) {
        ste[threadIdx.x >> 5] = te;
        sc[threadIdx.x >> 5] = cnt;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        te = ste[threadIdx.x];
        cnt = sc[threadIdx.x];
        for (int o = 16; o > 0; o >>= 1) {
            te += __shfl_xor_sync(0xffffffffu, te, o);
            cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        }
        if (threadIdx.x == 0) out[0] = te / cnt;
    }
}

// rescale_cells, src/mpcd.f90:748-801, of the n particles from a
template <typename R>
__device__ __forceinline__ void rescale_cell(int n, int a, R *vx, R *vy, R *vz, const int *species, double T)
{
    if (n <= 1) return;
    int n_eff = 0;
    CellSum<R> sx, sy, sz;
    for (int i = a; i < a + n; i++) {
        if (species[i] > 0) {
            sx.add(vx[i]);
            sy.add(vy[i]);
            sz.add(vz[i]);
            n_eff++;
        }
    }
    if (n_eff <= 1) return;
    R lv[3] = {sx.value() / n_eff, sy.value() / n_eff, sz.value() / n_eff};
    double kin = 0;
    for (int i = a; i < a + n; i++) {
        if (species[i] > 0) {
            double d0 = (double)(vx[i] - lv[0]), d1 = (double)(vy[i] - lv[1]), d2 = (double)(vz[i] - lv[2]);
            kin = kin + (d0 * d0 + d1 * d1 + d2 * d2);
        }
    }
    R tf = (R)sqrt((3 * (n_eff - 1)) * T / kin);
    for (int i = a; i < a + n; i++) {
        if (species[i] > 0) {
            vx[i] = lv[0] + tf * (vx[i] - lv[0]);
            vy[i] = lv[1] + tf * (vy[i] - lv[1]);
            vz[i] = lv[2] + tf * (vz[i] - lv[2]);
        }
    }
}

template <typename R, bool kStaged>
__global__ void __launch_bounds__(kCellThreads)
    k_rescale(const int *__restrict__ count, const int *__restrict__ start, int S, int per, R *vx, R *vy, R *vz,
              const int *__restrict__ species, double T)
{
    if constexpr (!kStaged) {
        const long long slot = (long long)blockIdx.x * kCellThreads + threadIdx.x;
        if (slot < S) rescale_cell<R>(count[slot], start[slot], vx, vy, vz, species, T);
    } else {
        __shared__ R sv[3][kCellCap];
        __shared__ int ss[1][kCellCap];
        const CellRange c(count, start, S, per);
        auto run = [=](int n, int a, int a0, int np) {
            tile_in<R, 3>(sv, {vx, vy, vz}, a0, np);
            tile_in<int, 1>(ss, {species}, a0, np);
            __syncthreads();
            rescale_cell<R>(n, a, sv[0], sv[1], sv[2], ss[0], T);
            __syncthreads();
            tile_out<R, 3>({vx, vy, vz}, sv, a0, np);
            return 0.0;
        };
        auto direct = [=] {
            rescale_cell<R>(c.n, c.a, vx, vy, vz, species, T);
            return 0.0;
        };
        cell_bodies<sizeof(R) == 8>(c, count, start, run, direct);
    }
}

// mpcd_stream_periodic, src/mpcd.f90:440-457
template <typename R>
__global__ void k_stream_periodic(PView<R> v, double e0, double e1, double e2, R dt)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < v.N;
         i += (long long)gridDim.x * blockDim.x) {
        R x = v.pos.x[i] + v.vel.x[i] * dt;
        R y = v.pos.y[i] + v.vel.y[i] * dt;
        R z = v.pos.z[i] + v.vel.z[i] * dt;
        int jx = floor_div_edge((double)x, e0), jy = floor_div_edge((double)y, e1), jz = floor_div_edge((double)z, e2);
        if (jx) v.ix[i] += jx;
        if (jy) v.iy[i] += jy;
        if (jz) v.iz[i] += jz;
        v.pos.x[i] = x - (R)(jx * e0);
        v.pos.y[i] = y - (R)(jy * e1);
        v.pos.z[i] = z - (R)(jz * e2);
    }
}

// yzwall_collision, src/mpcd.f90:511-589 (0-based dims y=1, z=2); the wall
// loop stops after 64 crossings and reports it instead of spinning
__device__ inline void yzwall_collision(const double x0[3], const double v0[3], double x[3],
                                        double v[3], const double L[3], double t, const int bc[3],
                                        double gx, unsigned *err)
{
    double gvec[3] = {gx, 0, 0};
    int im[3] = {0, 0, 0};
    int cd = -1;
    double tc = 1.7976931348623157e308;
    for (int i = 1; i <= 2; i++) {
        double tt = v0[i] > 0 ? (L[i] - x0[i]) / v0[i] : -x0[i] / v0[i];
        if ((tt > 0) && (tt < tc)) {
            tc = tt;
            cd = i;
        }
    }
    if (cd < 0) return;
    double tr = t - tc;
    for (int k = 0; k < 3; k++) {
        x[k] = x0[k] + v0[k] * tc + gvec[k] * (tc * tc) / 2;
        v[k] = v0[k] + gvec[k] * tc;
    }
    for (int iter = 0;; iter++) {
        if (bc[cd] == BOUNCE_BACK_BC) {
            for (int k = 0; k < 3; k++) v[k] = -v[k];
        } else if (bc[cd] == SPECULAR_BC) {
            v[cd] = -v[cd];
        } else if (bc[cd] == PERIODIC_BC) {
            int jump = ifloor(x[cd] / L[cd]);
            x[cd] = x[cd] - jump * L[cd];
            im[cd] = im[cd] + jump;
        }
        if (iter >= 64) {
            atomicOr(err, DEV_ERR_WALL_LOOP);
            break;
        }
        cd = cd == 1 ? 2 : 1;
        tc = v[cd] > 0 ? (L[cd] - x[cd]) / v[cd] : -x[cd] / v[cd];
        if ((tc < 0) || (tc > tr)) break;
        for (int k = 0; k < 3; k++) {
            x[k] = x[k] + v[k] * tc + gvec[k] * (tc * tc) / 2;
            v[k] = v[k] + gvec[k] * tc;
        }
        tr = tr - tc;
    }
    tc = tr;
    for (int k = 0; k < 3; k++) {
        x[k] = x[k] + v[k] * tc + gvec[k] * (tc * tc) / 2 + im[k] * L[k];
        v[k] = v[k] + gvec[k] * tc;
    }
}

// mpcd_stream_xforce_yzwall, src/mpcd.f90:464-506
template <typename R>
__global__ void k_stream_yzwall(PView<R> v, double L0, double L1, double L2, int bc0, int bc1, int bc2,
                                double dt, double g, unsigned *err)
{
    double L[3] = {L0, L1, L2};
    int bc[3] = {bc0, bc1, bc2};
    double gvec[3] = {g, 0, 0};
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < v.N;
         i += (long long)gridDim.x * blockDim.x) {
        double op[3] = {(double)v.pos.x[i], (double)v.pos.y[i], (double)v.pos.z[i]};
        double ov[3] = {(double)v.vel.x[i], (double)v.vel.y[i], (double)v.vel.z[i]};
        double np[3], nv[3];
        for (int k = 0; k < 3; k++) {
            np[k] = op[k] + ov[k] * dt + gvec[k] * (dt * dt) / 2;
            nv[k] = ov[k];
        }
        bool y_out = (np[1] < 0) || (np[1] > L[1]);
        bool z_out = (np[2] < 0) || (np[2] > L[2]);
        if (((bc[1] == PERIODIC_BC) && z_out) || ((bc[1] != PERIODIC_BC) && (y_out || z_out))) {
            yzwall_collision(op, ov, np, nv, L, dt, bc, g, err);
            v.flags[i] |= (1 << WALL_BIT);
            v.vel.x[i] = (R)nv[0];
            v.vel.y[i] = (R)nv[1];
            v.vel.z[i] = (R)nv[2];
        }
        v.pos.x[i] = (R)np[0];
        v.pos.y[i] = (R)np[1];
        v.pos.z[i] = (R)np[2];
    }
}

// mpcd_stream_nogravity_zwall, src/mpcd.f90:702-745
template <typename R>
__global__ void k_stream_zwall(PView<R> v, double Lz, double dt)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < v.N;
         i += (long long)gridDim.x * blockDim.x) {
        double op[3] = {(double)v.pos.x[i], (double)v.pos.y[i], (double)v.pos.z[i]};
        double ov[3] = {(double)v.vel.x[i], (double)v.vel.y[i], (double)v.vel.z[i]};
        double f[3] = {(double)v.force.x[i], (double)v.force.y[i], (double)v.force.z[i]};
        double np[3], nv[3];
        for (int k = 0; k < 3; k++) np[k] = op[k] + ov[k] * dt + f[k] * (dt * dt) / 2;
        bool bounce = false;
        double t_c = 0;
        if (np[2] < 0) {
            t_c = -op[2] / ov[2];
            bounce = true;
        } else if (np[2] > Lz) {
            t_c = (Lz - op[2]) / ov[2];
            bounce = true;
        } else {
            for (int k = 0; k < 3; k++) nv[k] = ov[k];
        }
        if (bounce) {
            for (int k = 0; k < 3; k++) {
                np[k] = np[k] - ov[k] * 2 * (dt - t_c);
                nv[k] = -ov[k];
            }
            v.flags[i] |= (1 << WALL_BIT);
        }
        v.pos.x[i] = (R)np[0];
        v.pos.y[i] = (R)np[1];
        v.pos.z[i] = (R)np[2];
        v.vel.x[i] = (R)nv[0];
        v.vel.y[i] = (R)nv[1];
        v.vel.z[i] = (R)nv[2];
    }
}

// bulk_reaction, src/mpcd.f90:605-643
__global__ void k_bulk_reaction(const int *__restrict__ count, const int *__restrict__ start,
                                const unsigned char *__restrict__ is_reac, int S, int *species,
                                int from, int to, double rate, double tau, uint64_t seed, uint64_t step)
{
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < S; s += gridDim.x * blockDim.x) {
        if ((count[s] <= 1) || !is_reac[s]) continue;
        int a = start[s], n = count[s];
        double local_rate = 0;
        int pick = -1;
        for (int i = a; i < a + n; i++)
            if (species[i] == from) {
                local_rate = local_rate + 1;
                pick = i;
            }
        local_rate = local_rate * rate;
        double u0, u1;
        rng::uniform2(seed, step, (uint32_t)s, rng::BULK, 0, u0, u1);
        if (u0 < (1 - exp(-local_rate * tau)) && pick >= 0) species[pick] = to;
    }
}

// bulk_reaction_endothermic, src/mpcd.f90:645-700: the reaction needs
// kin = sum |v - com_v|^2 / 2 > delta_u in the cell and, when it fires, takes
// delta_u from the cell's relative kinetic energy by scaling v - com_v.  Sums
// run in the cell's particle order, as the reference's per-cell loop does.
template <typename R>
__global__ void k_bulk_reaction_endo(const int *__restrict__ count, const int *__restrict__ start,
                                     const unsigned char *__restrict__ is_reac, int S, PView<R> v, int from,
                                     int to, double rate, double tau, double delta_u, uint64_t seed,
                                     uint64_t step)
{
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < S; s += gridDim.x * blockDim.x) {
        if ((count[s] <= 1) || !is_reac[s]) continue;
        int a = start[s], n = count[s];
        double local_rate = 0;
        int pick = -1;
        double cx = 0, cy = 0, cz = 0;
        for (int i = a; i < a + n; i++) {
            if (v.species[i] == from) {
                local_rate = local_rate + 1;
                pick = i;
            }
            cx = cx + (double)v.vel.x[i];
            cy = cy + (double)v.vel.y[i];
            cz = cz + (double)v.vel.z[i];
        }
        cx = cx / n;
        cy = cy / n;
        cz = cz / n;
        double kin = 0;
        for (int i = a; i < a + n; i++) {
            double dx = (double)v.vel.x[i] - cx, dy = (double)v.vel.y[i] - cy, dz = (double)v.vel.z[i] - cz;
            kin = kin + ((dx * dx + dy * dy) + dz * dz);
        }
        kin = kin / 2;
        if ((local_rate > 0) && (kin > delta_u)) {
            local_rate = local_rate * rate;
            double u0, u1;
            rng::uniform2(seed, step, (uint32_t)s, rng::BULK, 0, u0, u1);
            if (u0 < (1 - exp(-local_rate * tau))) {
                v.species[pick] = to;
                double factor = sqrt((kin - delta_u) / kin);
                for (int i = a; i < a + n; i++) {
                    v.vel.x[i] = (R)(cx + factor * ((double)v.vel.x[i] - cx));
                    v.vel.y[i] = (R)(cy + factor * ((double)v.vel.y[i] - cy));
                    v.vel.z[i] = (R)(cz + factor * ((double)v.vel.z[i] - cz));
                }
            }
        }
    }
}

static SrdParams srd_params(rmpcd_particles *p, rmpcd_cells *c, rmpcd_rng *r, int has_alpha,
                            double alpha, int thermostat, double T, int hydro)
{
    SrdParams q;
    q.sin_a = 1;
    q.cos_a = 0;
    if (has_alpha) {
        q.sin_a = sin(alpha);
        q.cos_a = cos(alpha);
    }
    q.t_factor = thermostat ? sqrt(T) : 0.0;
    q.thermostat = thermostat ? 1 : 0;
    q.hydro = hydro ? 1 : 0;
    q.seed = r ? r->seed : 0;
    q.step = r ? r->step : 0;
    q.axes = c->axes;
    q.gauss = p->gauss;
    return q;
}

static int at_blocks(long long N) { return grid_full((N + 32 * kAtChunks - 1) / (32 * kAtChunks) * 32, kAtThreads); }

// Slots per tile of the collision kernels: what kCellCap holds of a uniform fluid
// of this density with four standard deviations to spare, at most kCellTile.  0: no
// staging, a thread per slot on global memory, kCellThreads slots per block, where
// a tile would have fewer than four slots (kMinTile: also what k_temperature's
// partial sums have room for), from 178 particles per cell on.  us at 48^3 FP64 (SRD
// step, MPC-AT step, rescaling) with 64 slots whatever the density, with these, and
// with a thread per slot on global memory: density 15: 77 190 179, 38 108 37, 81 154
// 96; 30: 174 519 437, 81 213 78, 180 360 237; 100: - , 288 785 346, 648 1287 881; 150: - ,
// 555 1403 702, 966 1933 1364.
constexpr int kMinTile = 4;
static int cell_tile(const rmpcd_particles *p, const rmpcd_cells *c)
{
    const double mean = (double)p->N / ((double)c->L[0] * c->L[1] * c->L[2]);
    int per = kCellTile;
    while (per >= kMinTile && per * mean + 4 * sqrt(per * mean) > kCellCap) per--;
    return per >= kMinTile ? per : 0;
}
static int cell_blocks(int S, int per)
{
    if (per == 0) per = kCellThreads;
    return (S + per - 1) / per;
}

// with the thermostat, the normals go into the sort target's velocity arrays
// (free between sorts) first
template <typename R>
static void simple_launches(rmpcd_particles *p, rmpcd_cells *c, const SrdParams &q)
{
    cudaStream_t s = stream();
    const int per = cell_tile(p, c);
    const int g = cell_blocks(c->S, per);
    PView<R> v = cur<R>(p), t = alt<R>(p);
    if (q.thermostat && !q.gauss && p->N > 0) {
        k_at_normals<R><<<at_blocks(p->N), kAtThreads, 0, s>>>(v.species, p->N, q, t.vel.x, t.vel.y, t.vel.z);
        auto *k = per ? k_at_cells<R, true> : k_at_cells<R, false>;
        k<<<g, kCellThreads, 0, s>>>(c->count, c->start, c->S, per, v.vel.x, v.vel.y, v.vel.z, v.species, q.hydro, t.vel.x,
                                     t.vel.y, t.vel.z);
    } else {
        auto *k = per ? k_simple_mpcd<R, true> : k_simple_mpcd<R, false>;
        k<<<g, kCellThreads, 0, s>>>(c->count, c->start, c->S, per, v.vel.x, v.vel.y, v.vel.z, v.species, q);
    }
}

template <typename R>
static void wall_launches(rmpcd_particles *p, rmpcd_cells *c, const SrdParams &q, const WallArgs &w)
{
    cudaStream_t s = stream();
    const int per = cell_tile(p, c);
    const bool at = q.thermostat && p->N > 0;
    PView<R> v = cur<R>(p), t = alt<R>(p);
    if (at) k_at_normals<R><<<at_blocks(p->N), kAtThreads, 0, s>>>(nullptr, p->N, q, t.vel.x, t.vel.y, t.vel.z);
    auto *k = at ? (per ? k_wall_mpcd<R, true, true> : k_wall_mpcd<R, true, false>)
                 : (per ? k_wall_mpcd<R, false, true> : k_wall_mpcd<R, false, false>);
    k<<<cell_blocks(c->S, per), kCellThreads, 0, s>>>(c->count, c->start, c->S, per, v.vel.x, v.vel.y, v.vel.z, t.vel.x,
                                                    t.vel.y, t.vel.z, q, w);
}

template <typename R>
static void temperature_launches(rmpcd_particles *p, rmpcd_cells *c, double *part, double *out)
{
    const int per = cell_tile(p, c);
    const int nb = cell_blocks(c->S, per);
    PView<R> v = cur<R>(p);
    auto *k = per ? k_temperature<R, true> : k_temperature<R, false>;
    k<<<nb, kCellThreads, 0, stream()>>>(c->count, c->start, c->S, per, v.vel.x, v.vel.y, v.vel.z, v.species, part);
    k_temperature_final<<<1, 1024, 0, stream()>>>(part, nb, out);
}

template <typename R>
static void rescale_launch(rmpcd_particles *p, rmpcd_cells *c, double T)
{
    const int per = cell_tile(p, c);
    PView<R> v = cur<R>(p);
    auto *k = per ? k_rescale<R, true> : k_rescale<R, false>;
    k<<<cell_blocks(c->S, per), kCellThreads, 0, stream()>>>(c->count, c->start, c->S, per, v.vel.x, v.vel.y, v.vel.z,
                                                           v.species, T);
}

}  // namespace rmpcd

using namespace rmpcd;

#define DISPATCH_R(p, CALL_F, CALL_D)        \
    do {                                      \
        if ((p)->precision == RMPCD_FP32) {   \
            CALL_F;                           \
        } else {                              \
            CALL_D;                           \
        }                                     \
    } while (0)

extern "C" {

int rmpcd_simple_mpcd_step(rmpcd_particles *p, rmpcd_cells *c, rmpcd_rng *r, int has_alpha,
                           double alpha, int thermostat, double T, int hydro)
{
    RMPCD_ARG(p && c && r, "null argument");
    if (!hydro && !thermostat)
        return fail(RMPCD_ERR_STOP, "requiring .not.do_hydro without thermostat in simple_mpcd_step");
    PhaseTimer t("step");
    SrdParams q = srd_params(p, c, r, has_alpha, alpha, thermostat, T, hydro);
    DISPATCH_R(p, simple_launches<float>(p, c, q), simple_launches<double>(p, c, q));
    RMPCD_CHECK_LAUNCH();
    r->step++;
    return RMPCD_OK;
}

int rmpcd_wall_mpcd_step(rmpcd_particles *p, rmpcd_cells *c, rmpcd_rng *r,
                         const double wall_temperature[2], const double wall_v[6], const int wall_n[2],
                         int thermostat, double bulk_temperature, int has_alpha, double alpha,
                         int keep_cell_v)
{
    RMPCD_ARG(p && c && r, "null argument");
    bool all_present = wall_temperature && wall_v && wall_n;
    bool all_absent = !wall_temperature && !wall_v && !wall_n;
    if (!(all_present || all_absent))
        return fail(RMPCD_ERR_STOP, "wall parameters must be all present or all absent in wall_mpcd_step");
    if (!keep_cell_v && !thermostat)
        return fail(RMPCD_ERR_STOP, "requiring .not. keep_cell_v and .not. thermostat in wall_mpcd_step");
    SrdParams q = srd_params(p, c, r, has_alpha, alpha, thermostat, bulk_temperature, 1);
    const WallArgs w{c->M[0], c->M[1], c->M[2], c->L[2], all_present ? 1 : 0, all_present ? wall_temperature[0] : 0,
                     all_present ? wall_temperature[1] : 0, all_present ? wall_n[0] : 0, all_present ? wall_n[1] : 0,
                     keep_cell_v ? 1 : 0};
    PhaseTimer t("step");
    DISPATCH_R(p, wall_launches<float>(p, c, q, w), wall_launches<double>(p, c, q, w));
    RMPCD_CHECK_LAUNCH();
    r->step++;
    return RMPCD_OK;
}

int rmpcd_compute_temperature(rmpcd_particles *p, rmpcd_cells *c, double *te)
{
    RMPCD_ARG(p && c && te, "null argument");
    PhaseTimer t("compute_temperature");
    cudaStream_t s = stream();
    // two doubles per tile of slots, in the slots' scatter cursors (rewritten by
    // the next count_particles or sort before they are read)
    double *part = (double *)c->cursor, *out = c->d_red;
    DISPATCH_R(p, temperature_launches<float>(p, c, part, out), temperature_launches<double>(p, c, part, out));
    RMPCD_CHECK_LAUNCH();
    RMPCD_CUDA_TRY(cudaMemcpyAsync(te, out, sizeof(double), cudaMemcpyDeviceToHost, s));
    return sync();
}

int rmpcd_rescale_cells(rmpcd_particles *p, rmpcd_cells *c, rmpcd_rng *, double T)
{
    RMPCD_ARG(p && c, "null argument");
    PhaseTimer t("step");
    DISPATCH_R(p, rescale_launch<float>(p, c, T), rescale_launch<double>(p, c, T));
    RMPCD_CHECK_LAUNCH();
    return RMPCD_OK;
}

int rmpcd_mpcd_stream_periodic(rmpcd_particles *p, rmpcd_cells *c, double dt)
{
    RMPCD_ARG(p && c, "null argument");
    if (p->N == 0) return RMPCD_OK;
    PhaseTimer t("stream");
    cudaStream_t s = stream();
    int g = grid_for(p->N, 256);
    DISPATCH_R(p,
               (k_stream_periodic<float><<<g, 256, 0, s>>>(cur<float>(p), c->edges[0], c->edges[1], c->edges[2], (float)dt)),
               (k_stream_periodic<double><<<g, 256, 0, s>>>(cur<double>(p), c->edges[0], c->edges[1], c->edges[2], dt)));
    RMPCD_CHECK_LAUNCH();
    return RMPCD_OK;
}

int rmpcd_mpcd_stream_xforce_yzwall(rmpcd_particles *p, rmpcd_cells *c, double dt, double g)
{
    RMPCD_ARG(p && c, "null argument");
    if (p->N == 0) return RMPCD_OK;
    PhaseTimer t("stream");
    cudaStream_t s = stream();
    int gr = grid_for(p->N, 256);
    unsigned *err = dev_error_word();
    DISPATCH_R(p,
               (k_stream_yzwall<float><<<gr, 256, 0, s>>>(cur<float>(p), c->edges[0], c->edges[1], c->edges[2],
                                                          c->bc[0], c->bc[1], c->bc[2], dt, g, err)),
               (k_stream_yzwall<double><<<gr, 256, 0, s>>>(cur<double>(p), c->edges[0], c->edges[1], c->edges[2],
                                                           c->bc[0], c->bc[1], c->bc[2], dt, g, err)));
    RMPCD_CHECK_LAUNCH();
    return RMPCD_OK;
}

int rmpcd_mpcd_stream_nogravity_zwall(rmpcd_particles *p, rmpcd_cells *c, double dt)
{
    RMPCD_ARG(p && c, "null argument");
    if (p->N == 0) return RMPCD_OK;
    PhaseTimer t("stream");
    cudaStream_t s = stream();
    int gr = grid_for(p->N, 256);
    DISPATCH_R(p, (k_stream_zwall<float><<<gr, 256, 0, s>>>(cur<float>(p), c->edges[2], dt)),
               (k_stream_zwall<double><<<gr, 256, 0, s>>>(cur<double>(p), c->edges[2], dt)));
    RMPCD_CHECK_LAUNCH();
    return RMPCD_OK;
}

int rmpcd_bulk_reaction(rmpcd_particles *p, rmpcd_cells *c, int from, int to, double rate, double tau,
                        rmpcd_rng *r)
{
    RMPCD_ARG(p && c && r, "null argument");
    k_bulk_reaction<<<grid_full(c->S, 128), 128, 0, stream()>>>(c->count, c->start, c->is_reac, c->S,
                                                               p->species[p->cur], from, to, rate, tau,
                                                               r->seed, r->step);
    RMPCD_CHECK_LAUNCH();
    r->step++;
    return RMPCD_OK;
}

int rmpcd_bulk_reaction_endothermic(rmpcd_particles *p, rmpcd_cells *c, int from, int to, double rate,
                                    double tau, rmpcd_rng *r, double delta_u)
{
    RMPCD_ARG(p && c && r, "null argument");
    int gr = grid_full(c->S, 128);
    cudaStream_t s = stream();
    DISPATCH_R(p,
               (k_bulk_reaction_endo<float><<<gr, 128, 0, s>>>(c->count, c->start, c->is_reac, c->S, cur<float>(p),
                                                               from, to, rate, tau, delta_u, r->seed, r->step)),
               (k_bulk_reaction_endo<double><<<gr, 128, 0, s>>>(c->count, c->start, c->is_reac, c->S,
                                                                cur<double>(p), from, to, rate, tau, delta_u,
                                                                r->seed, r->step)));
    RMPCD_CHECK_LAUNCH();
    r->step++;
    return RMPCD_OK;
}

}  // extern "C"
