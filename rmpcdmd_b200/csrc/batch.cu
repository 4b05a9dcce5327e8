// Batched single-dimer engine: R independent single_dimer_pbc systems
// (programs/single_dimer_pbc.f90:303-443), each with its own box, seed and
// solvent, advanced together.  Every phase of the program's MD step and MPCD
// interval is one launch over all replicas: solvent work is cut into tiles of
// kTile particles (or slots) that each belong to one replica, colloid work is
// one thread or block per replica.  The replicas' solvents are concatenated
// in one particle system, their slot ranges in one slot space; a replica's
// Hilbert order stays inside its own range, so the sort kernels of a single
// system apply to every replica at once.
//
// MD steps touch only the solvent that can interact.  A particle that is in
// neither bead's neighbor list and carries no MD, PAST_MD, REAC or WALL flag, or
// which has no force still to act and whose way stays clear of the beads, flies
// freely until the next re-sort: no force can reach it before the list is rebuilt, so
// its md_pos steps depend on nothing but its own position and velocity.  Such particles
// stay where they are in memory; the re-sort (or the
// interval's end) advances each by its pending md_pos steps in one pass, adding
// dt * v once per step so that every rounding is that of the steps one by one.
// The others -- the active particles, some 800 per dimer at sigma = 2: those
// with flags and those of the lists whose straight way may take them to a bead
// before the next re-sort -- are advanced by kb_md, one block per replica, which
// runs the MD steps one after another without leaving the kernel: pair forces,
// md_vel, change_species, the colloid sums, velocity-Verlet and RATTLE, the
// next step's md_pos, until the program's re-sort test
// (programs/single_dimer_pbc.f90:323-330) fires or the interval's MD steps are
// done.  The test needs the largest solvent displacement: of the active
// particles the block has it, of the free ones kb_classify has computed the
// first step at which any of them reaches the threshold, by the same additions
// and the same comparison.  Replicas re-sort at steps of their own: a launch of
// kb_md ends when each of its replicas waits for a re-sort or is done, then one
// re-sort serves all that wait (a WHILE node of the captured interval graph).
// The re-sort gathers into the other buffer of the particle system; which one
// is current is kept per replica on the device (BRep::cur), as are the RNG
// step and the grid origins, so one captured interval graph serves every
// interval.
//
// Moving every particle in every MD step costs 56 B (FP32) per particle and
// step: 121 us per step at 96^3 (4.1 TB/s) and 237 us for 48 replicas in boxes
// of 16..48 cells, against 6 us per step for kb_md.
//
// Arithmetic per particle is that of the single-system kernels
// (stepops.cuh, nlist_ops.cuh), so replica r reproduces, bit for bit, the
// same program run alone through the C ABI with its own seed.
#include <climits>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include "keys.cuh"
#include "nlist_ops.cuh"
#include "quotient.cuh"
#include "rmpcd_common.cuh"
#include "rng.cuh"
#include "sortcore.cuh"
#include "sorttile.cuh"
#include "state.cuh"
#include "stepops.cuh"
#include "timers.cuh"

namespace rmpcd {

constexpr int kTile = 1024;  // slots per slot tile
constexpr int kBT = 256;     // threads per tile block

// Engine shapes (rmpcd_dimer_batch_autotune): the particles per tile of the
// sort's particle kernels, the threads of kb_md that move a replica's solvent,
// and the list entries per thread of the kernels that make the active list.  Every shape gives the same
// results bit for bit: they only decide which thread handles which particle.
constexpr int kPartThreads[] = {512, 448, 384, 320, 256};
constexpr int kBVars = 5;
constexpr long long kPTiles[] = {256, 512, 1024, 2048, 4096};  // particles per tile
constexpr int kNPTiles = 5;
// list entries per thread: blocks per colloid are ceil(capacity / (256 x
// this)), at most 64
constexpr int kListPer[] = {1, 4};
constexpr int kNListPer = 2;
constexpr int kBShapes = kNListPer * kBVars * kNPTiles;
// shape s: particle tile kPTiles[s % kNPTiles], threads kPartThreads[(s /
// kNPTiles) % kBVars], list entries per thread kListPer[s / (kNPTiles * kBVars)]
__host__ __device__ inline int shape_tile(int s) { return s % kNPTiles; }
__host__ __device__ inline int shape_var(int s) { return (s / kNPTiles) % kBVars; }
__host__ __device__ inline int shape_list(int s) { return s / (kNPTiles * kBVars); }

struct BTile {
    int r;
    int pad;
    long long begin, end;
};


struct BRep {
    long long off;  // first solvent particle of the replica
    int n;          // its solvent particles
    int soff;       // first slot
    int S;          // its slots
    int cur;        // buffer holding the replica's current solvent arrays
    uint64_t seed;
    double far;     // refuel distance (single-precision expression of the program)
    Grid g;         // cells; origin rewritten on the device by the grid shift
};

// a pair force in global memory: its place in the order of addition and the force
struct MdTerm {
    int e, pad;
    double f[3];
};

}  // namespace rmpcd

struct rmpcd_dimer_batch {
    int R = 0;
    int precision = RMPCD_FP64;
    rmpcd_dimer_params prm{};
    long long Ntot = 0;
    int Stot = 0;
    rmpcd_particles *sol = nullptr;  // all solvents, concatenated (buffer 0 current, 1 = gather target / pos_old)
    rmpcd_particles *col = nullptr;  // all colloids, 2 per replica
    std::vector<rmpcd::BRep> rep_h;
    rmpcd::BRep *rep = nullptr;
    rmpcd::BTile *ptile = nullptr, *stile = nullptr;
    int n_ptile = 0, n_stile = 0;
    int order_slots = 0;  // slots per tile of the re-sort's gather, by the densest replica
    int cap_ptile = 0;  // particle tiles allocated (enough for the smallest tile size)
    int shape = 0;      // engine shape in use (kernel variant, particles per tile)
    int *stile_first = nullptr, *stile_count = nullptr;  // per replica
    int *ptile_first = nullptr, *ptile_count = nullptr;  // per replica
    int *act_p = nullptr, *act_s = nullptr, *n_act = nullptr;  // tiles of the replicas flagged for a re-sort
    int *all_p = nullptr, *all_s = nullptr, *n_all = nullptr;  // every tile
    long long *tile_sum = nullptr, *tile_off = nullptr;  // per slot tile
    int *count = nullptr, *start = nullptr, *cursor = nullptr;
    unsigned char *is_md = nullptr, *is_reac = nullptr;
    std::vector<int *> luts;
    int *stencil = nullptr;
    int n_stencil = 0;
    int Nmax = 0;
    int *list = nullptr, *nn = nullptr;
    // active particles (kb_claim, kb_classify), in the replica's range of act:
    // nl[r] of the neighbor lists first, then nx[r] flagged ones outside them
    int *act = nullptr, *nl = nullptr, *nx = nullptr;
    int *aidx = nullptr;       // per particle: its place in act, -1 when it flies freely
    int *ent = nullptr;        // per listed active particle: an entry of it in list 0 and in list 1, or -1
    int *next = nullptr;       // per list entry: another entry of the same particle in the list, or -1
    int *mult = nullptr;       // per listed active particle: entries in list 0 | entries in list 1 << 16
    // pair forces beyond what kb_md holds in shared memory
    rmpcd::MdTerm *over = nullptr, *terms = nullptr;
    unsigned long long *keys[2] = {nullptr, nullptr};
    int *n_over = nullptr;
    // active particles beyond what kb_md holds in shared memory
    unsigned char *far = nullptr;
    int far_cap = 0;  // per replica
    int *nf = nullptr;         // per replica: flagged particles, listed in sol->key from the replica's first place
    int *s_free = nullptr;     // per replica: first MD step at which a free particle forces a re-sort
    int *adv = nullptr, *base = nullptr;  // per replica: md_pos steps done this interval, and those in memory
    int *fresh = nullptr;      // per replica: pos_old is the caller's (no sort yet)
    bool ran = false;          // an interval has been run
    // whether some solvent species was negative at creation; species change
    // only to 1 or 2 inside the batch, so otherwise every particle passes
    // maximum_displacement's species >= 0 test and species need not be read
    bool read_species = true;
    int *resort = nullptr, *n_extra = nullptr;
    double *rattle[3] = {nullptr, nullptr, nullptr};
    double *vv_mass = nullptr;
    uint64_t *d_step = nullptr;
    uint64_t step = 0;  // host copy of every replica's RNG step
    rmpcd::Masses ms{};
    rmpcd::LJDev lj_sc{}, lj_cc{};
    unsigned *done = nullptr;   // replicas finished in the current kb_md launch (last-block hand-off)
    bool use_graph = true;
    bool capturing = false;
    cudaError_t cap_err = cudaSuccess;
    cudaStream_t body = nullptr;  // captures the body of the re-sort WHILE node
    int *any = nullptr;  // 1 when the last kb_md launch left some replica waiting for a re-sort
    cudaGraphExec_t exec = nullptr;
};

namespace rmpcd {

// ------------------------------------------------------------------ views

template <typename R>
static PView<R> phys(const rmpcd_particles *p, int b)
{
    return view<R>(p, b);
}

// buffer 0 or 1
template <typename R>
__device__ __forceinline__ PView<R> pick(const PView<R> &v0, const PView<R> &v1, int which)
{
    return which ? v1 : v0;
}

// the tiles a re-sort kernel visits: tiles[ids[k]] for k < *n (every tile
// for the interval's sort, the flagged replicas' tiles for an MD step's)
struct TileSet {
    const BTile *tiles;
    const int *ids;
    const int *n;
};

// ------------------------------------------------------------ MD step
//
// Force entries that can be non-zero are known from the flags: MD set means
// the particle received a contribution in the last force evaluation, PAST_MD
// in the one before.  Every other entry is exactly zero.  In memory `force` is
// the last evaluation's force of particles with MD or PAST_MD set and zero
// elsewhere; `force_old` is written by an interval's last MD step only.

constexpr int kActiveBits = (1 << WALL_BIT) | (1 << MD_BIT) | (1 << PAST_MD_BIT) | (1 << REAC_BIT);

__device__ inline bool same_bits(float a, float b) { return __float_as_int(a) == __float_as_int(b); }
__device__ inline bool same_bits(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); }

// md_vel of a particle without force turns a -0 velocity component into +0 in
// the FP64 form, as the reference's does; the FP32 form leaves such
// velocities untouched (a -0 component, which an SRD rotation product can
// round to, stays: equal in value, not in bits)
template <typename R>
__device__ __forceinline__ R md_vel_free(R v, R dt)
{
    const R z = 0;
    return sizeof(R) == 8 ? v + dt * (z + z) / 2 : v;
}

// the tile lists of the replicas flagged for a re-sort
struct ResortLists {
    const int *pfirst, *pcount, *sfirst, *scount;  // per replica
    int *pids, *sids;                              // out: active particle / slot tiles
    int *n;                                        // out: n[0] particle tiles, n[1] slot tiles
};

// exclusive block scan of one int per thread (blocks of up to 1024 threads, a
// multiple of 32); *total gets the block's sum (ws: 33 ints of shared memory)
__device__ inline int block_excl_scan(int v, int *ws, int *total)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) ws[w] = inc;
    __syncthreads();
    if (threadIdx.x == 0) {
        int acc = 0;
        for (int k = 0; k < nw; k++) {
            int y = ws[k];
            ws[k] = acc;
            acc += y;
        }
        ws[32] = acc;
    }
    __syncthreads();
    int ex = ws[w] + inc - v;
    *total = ws[32];
    __syncthreads();
    return ex;
}

// Flagged particles of the replicas at creation (later the re-sort's gather
// lists them); force entries that the flags say are zero are made so.
template <typename R>
__global__ void kb_collect_flagged(TileSet ts, const BRep *rep, PView<R> v, int *key, int *nf)
{
    for (int kt = blockIdx.x; kt < *ts.n; kt += gridDim.x) {
        const BTile t = ts.tiles[ts.ids[kt]];
        for (long long i = t.begin + threadIdx.x; i < t.end; i += blockDim.x) {
            const int f = v.flags[i];
            if (f & kActiveBits) key[rep[t.r].off + atomicAdd(nf + t.r, 1)] = (int)i;
            if (!((f >> MD_BIT) & 1)) v.force.x[i] = v.force.y[i] = v.force.z[i] = 0;
            if (!((f >> PAST_MD_BIT) & 1)) v.force_old.x[i] = v.force_old.y[i] = v.force_old.z[i] = 0;
        }
    }
}

// Whether a particle at p with velocity v may come within `reach` of the point c
// in the next time T of free flight, in a periodic box of edges L (single
// precision; reach holds the margin for it)
__device__ __forceinline__ bool may_meet(const float p[3], const float v[3], const float c[3], const float L[3],
                                         float reach, float T)
{
    float d[3], a = 0, b = 0;
    bool one_image = true;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float x = p[k] - c[k], h = 0.5f * L[k];
        d[k] = x < -h ? x + L[k] : x > h ? x - L[k] : x;
        one_image = one_image && fabsf(d[k]) + T * fabsf(v[k]) < L[k] - reach;
        a += v[k] * v[k];
        b += d[k] * v[k];
    }
    const float t = a > 0 ? fminf(fmaxf(-b / a, 0.0f), T) : 0.0f;
    float m = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float x = d[k] + t * v[k];
        m += x * x;
    }
    return !(one_image && m > reach * reach);
}

// The listed particles of the replicas in flag (every one when null) that may
// come within a cut of a bead before the next re-sort become active, each
// once: its place in act goes to aidx.  Until a re-sort a bead stays within
// skin / 10 of its pos_old (the re-sort test, programs/single_dimer_pbc.f90:324-329),
// and a particle without force flies straight, so that of the ~4,800 listed
// particles of a sigma = 2 dimer some 800 are left.  One with MD or PAST_MD set
// does not: half of its last force is still to change its velocity (and, with MD,
// that force its position), wherever it has gone since, so it is always claimed.
template <typename R>
__global__ void __launch_bounds__(kBT)
    kb_claim(const int *flag, const BRep *rep, PView<R> v0, PView<R> v1, Vec3<double> cold, R dt, float reach,
             float margin, int N_MD, const int *base, const int *list, const int *n, int Nmax, int *aidx, int *act,
             int *nl, int *mult, int *ent)
{
    const int i = blockIdx.y, r = i >> 1;
    if (flag && !flag[r]) return;
    const BRep &rp = rep[r];
    const long long off = rp.off;
    const PView<R> v = pick(v0, v1, rp.cur);
    const int steps = N_MD - base[r];
    float L[3], c[2][3];
    for (int k = 0; k < 3; k++) {
        L[k] = (float)rp.g.edges[k];
        for (int h = 0; h < 2; h++) c[h][k] = (float)cold[k][2 * r + h];
    }
    // the rounding of every addition of the flight, and of this test
    const float far = reach + margin + (1e-5f + (sizeof(R) == 4 ? 2.4e-7f : 4.4e-16f) * (float)steps) * (L[0] + L[1] + L[2]);
    const float T = (float)dt * (float)steps * 1.0001f;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n[i]; e += gridDim.x * blockDim.x) {
        const int idx = list[(size_t)i * Nmax + e];
        const float p[3] = {(float)v.pos.x[idx], (float)v.pos.y[idx], (float)v.pos.z[idx]};
        const float u[3] = {(float)v.vel.x[idx], (float)v.vel.y[idx], (float)v.vel.z[idx]};
        const bool forced = v.flags[idx] & ((1 << MD_BIT) | (1 << PAST_MD_BIT));
        if (!forced && !may_meet(p, u, c[0], L, far, T) && !may_meet(p, u, c[1], L, far, T)) continue;
        if (atomicCAS(aidx + idx, -1, -2) != -1) continue;
        const int a = atomicAdd(nl + r, 1);
        act[off + a] = idx;
        aidx[idx] = a;
        const size_t w = (size_t)2 * r * Nmax + a;
        mult[w] = 0;
        ent[2 * w] = ent[2 * w + 1] = -1;
    }
}

// The first MD step before `best` at whose test the free particle i has moved
// sqrt(d2) >= thr from pos_old (programs/single_dimer_pbc.f90:324-329,
// src/particle_system.f90:357-378), or best.  A particle's earliest possible step
// follows from its speed (reach bounds the distance of one addition, its
// rounding included); only the particles that could be first -- a few per
// replica -- go through their additions one by one.
template <typename R>
__device__ __forceinline__ int free_crossing(const PView<R> &v, const Vec3<R> &old, long long i, R vx, R vy, R vz,
                                              float reach, int fresh, R dt, double thr, int base, int n_rem,
                                              int read_species, const int *aidx, int best)
{
    float left = (float)thr;
    if (fresh) {
        // positions and pos_old are the caller's: any distance, any place
        const double d0 = (double)v.pos.x[i] - (double)old.x[i], d1 = (double)v.pos.y[i] - (double)old.y[i],
                     d2 = (double)v.pos.z[i] - (double)old.z[i];
        left = (float)(thr - sqrt(d0 * d0 + d1 * d1 + d2 * d2)) - 1e-3f * (float)thr;
        reach += (sizeof(R) == 4 ? 2.4e-7f : 4.4e-16f) *
                 (fabsf((float)v.pos.x[i]) + fabsf((float)v.pos.y[i]) + fabsf((float)v.pos.z[i]));
    }
    if (!(reach * (float)n_rem >= left)) return best;
    int lo = left > 0 ? (int)fminf(left / reach, 1e9f) - 1 : 1;  // no crossing before the lo-th addition
    if (lo < 1) lo = 1;
    if (base + lo - 1 >= best) return best;
    if ((v.flags[i] & kActiveBits) || aidx[i] >= 0) return best;
    if (read_species && v.species[i] < 0) return best;
    const R hx = dt * vx, hy = dt * vy, hz = dt * vz;
    R x = v.pos.x[i], y = v.pos.y[i], z = v.pos.z[i];
    const double ox = fresh ? (double)old.x[i] : (double)x, oy = fresh ? (double)old.y[i] : (double)y,
                 oz = fresh ? (double)old.z[i] : (double)z;
    for (int j = 1; j <= n_rem; j++) {
        x = x + hx;
        y = y + hy;
        z = z + hz;
        if (j < lo) continue;
        const double d0 = (double)x - ox, d1 = (double)y - oy, d2 = (double)z - oz;
        if (sqrt(d0 * d0 + d1 * d1 + d2 * d2) >= thr) return min(best, base + j - 1);
    }
    return best;
}

// After kb_claim: the first step at which a free particle forces a re-sort
// (particle tiles), every listed particle's entries in the two lists, counted
// and chained (gx blocks per bead), and the flagged particles outside the lists, which
// become active behind the listed ones (one block per replica).
template <typename R>
__global__ void __launch_bounds__(kBT)
    kb_classify(TileSet ts, int n_tile_blocks, int gx, int R_, const int *flag, const BRep *rep, PView<R> v0,
                PView<R> v1, R dt, double thr, int N_MD, int read_species, const int *base, const int *fresh,
                int *s_free, const int *list, const int *n, int Nmax, int *aidx, int *act, const int *nl, int *nx,
                int *mult, int *ent, int *next, const int *key, const int *nf)
{
    int b = blockIdx.x;
    if (b < n_tile_blocks) {
        for (int kt = b; kt < *ts.n; kt += n_tile_blocks) {
            const BTile t = ts.tiles[ts.ids[kt]];
            const BRep &rp = rep[t.r];
            const PView<R> v = pick(v0, v1, rp.cur);
            const Vec3<R> old = rp.cur ? v0.pos : v1.pos;
            const int b0 = base[t.r], fr = fresh[t.r];
            // three components, each rounded by at most half an ulp of a
            // position inside twice the box
            const float slack =
                (sizeof(R) == 4 ? 2.4e-7f : 4.4e-16f) * (float)(rp.g.edges[0] + rp.g.edges[1] + rp.g.edges[2]);
            // the velocities alone rule out nearly every particle: four per
            // thread and pass, loaded before any is used
            constexpr int K = 4;
            for (long long i0 = t.begin + threadIdx.x; i0 < t.end; i0 += K * kBT) {
                R vx[K], vy[K], vz[K];
                const int so_far = *(volatile int *)(s_free + t.r);  // it only falls
                int best = so_far;
#pragma unroll
                for (int k = 0; k < K; k++) {
                    const long long i = i0 + k * kBT;
                    if (i < t.end) {
                        vx[k] = v.vel.x[i];
                        vy[k] = v.vel.y[i];
                        vz[k] = v.vel.z[i];
                    }
                }
                const float steps = (float)(min(N_MD, so_far) - b0);
#pragma unroll
                for (int k = 0; k < K; k++) {
                    const long long i = i0 + k * kBT;
                    if (i >= t.end) break;
                    const float ux = (float)vx[k], uy = (float)vy[k], uz = (float)vz[k];
                    const float reach = (float)dt * sqrtf(ux * ux + uy * uy + uz * uz) * 1.001f + slack;
                    // (one step more: best is the step of the addition before it)
                    if (fr || reach * (steps + 1.0f) >= (float)thr)
                        best = free_crossing<R>(v, old, i, vx[k], vy[k], vz[k], reach, fr, dt, thr, b0, N_MD - b0,
                                                read_species, aidx, best);
                }
                // one atomic for the threads here, where there is a step to write at
                // all (with a skin that many particles cross, 32^3 and skin 0.1, one
                // per particle took 171 us, 11 so)
                const unsigned here = __activemask();
                best = __reduce_min_sync(here, best);
                if (best < so_far && (int)(threadIdx.x & 31) == __ffs(here) - 1) atomicMin(s_free + t.r, best);
            }
        }
        return;
    }
    b -= n_tile_blocks;
    if (b < gx * 2 * R_) {
        const int i = b / gx, r = i >> 1;
        if (flag && !flag[r]) return;
        for (int e = (b % gx) * blockDim.x + threadIdx.x; e < n[i]; e += gx * blockDim.x) {
            const size_t q = (size_t)i * Nmax + e;
            // (the flagged blocks give places from nl on at the same time: those
            // particles' way is clear of the beads, and mult and ent hold the listed)
            const int a = aidx[list[q]];
            if (a < 0 || a >= nl[r]) continue;
            const size_t w = (size_t)2 * r * Nmax + a;
            atomicAdd(mult + w, (i & 1) ? 1 << 16 : 1);
            next[q] = atomicExch(ent + 2 * w + (i & 1), e);
        }
        return;
    }
    const int r = b - gx * 2 * R_;
    if (flag && !flag[r]) return;
    const long long off = rep[r].off;
    for (int k = threadIdx.x; k < nf[r]; k += blockDim.x) {
        const int idx = key[off + k];
        if (atomicCAS(aidx + idx, -1, -2) != -1) continue;
        const int a = nl[r] + atomicAdd(nx + r, 1);
        act[off + a] = idx;
        aidx[idx] = a;
    }
}

// kb_md's block: the warps that add up the pair forces and move the beads
// (half of them per bead), then those that have the particles; and what it
// holds of a step in shared memory (more terms than fit go to global memory; lists
// of more entries than the map's largest size through md_slow_sums)
constexpr int kMdSum = 256;
constexpr int kMdThreads = kMdSum + 512;
constexpr int kMdQueue = 1024;    // pairs of a particle and a bead that may reach it
constexpr int kMdTerms = 512;     // pair forces per bead
constexpr int kMdMapWords = 6144; // most words of the map of a bead's list entries
constexpr size_t kMdSmem = 224 * 1024;  // dynamic shared memory
// A particle is queued for the next step's pair forces before the beads have
// moved: within this distance more than the cuts, which is far above a bead's
// way in a step; a bead that moves farther makes the queue anew.
constexpr float kMdWay = 0.02f;

template <typename R>
struct MdArgs {
    const BRep *rep;
    PView<R> v0, v1;      // solvent, buffers 0 and 1
    PView<double> c;      // colloids
    Vec3<double> cold;    // colloid pos_old
    double *rat[3];       // pos_rattle
    const double *mass;   // velocity-Verlet masses, 2 per replica
    Masses ms;
    double bond, dt, skin;
    R dt_r, dt_sq_r;
    double cut_c, cut_n, prob;
    float reach;          // the largest cut, with a margin for single precision less than 1e-5 (Lx + Ly + Lz)
    LJDev lj_sc, lj_cc;
    int R_, N_MD, Nmax, start, read_species;
    const uint64_t *d_step;
    const int *n, *next, *ent, *act, *nl, *nx, *mult;
    MdTerm *over, *terms;         // 2 * R * Nmax each: terms beyond the shared ones, terms to be put in order
    unsigned long long *keys[2];  // sort keys of the latter
    int *n_over;                  // per bead, one counter per step parity
    unsigned char *far;           // room for far_cap active particles per replica (MdBox::far)
    int far_cap;
    const int *s_free, *fresh;
    int *adv, *resort, *n_extra;
    ResortLists rl;
    unsigned *done;
    int *any;
    cudaGraphConditionalHandle cond;
    int use_cond;
    unsigned *err;
};

// one active solvent particle
template <typename R>
struct Part {
    R p[3], v[3], o[3]; // position, velocity, pos_old
    R g[3];             // the last evaluation's force (zero without MD and PAST_MD)
    int f, sp;          // flags, species
};

template <typename R>
__host__ __device__ constexpr size_t md_part_bytes()
{
    return 18 * sizeof(R) + 8 * sizeof(int);
}
template <typename R>
__host__ __device__ constexpr size_t md_far_bytes()
{
    return 15 * sizeof(R) + 3 * sizeof(int);  // times an even number: a multiple of sizeof(double)
}

// the fields of a block's particles in shared memory, cap of each
template <typename R>
struct MdParts {
    R *r;    // p[3], v[3], o[3], g[3], then the step's forces of the two beads, cap each
    int *i;  // idx, flags, species, multiplicities, entries in the two lists, what
             // the step has for the particle (bit h: bead h is queued, bit 2:
             // flags), what came of it (bit h: bead h acts, bit 2: REAC)
    int cap;
    __device__ R &real(int field, int s) const { return r[(size_t)field * cap + s]; }
    __device__ int &num(int field, int s) const { return i[(size_t)field * cap + s]; }
};

// What the steps need of the replica and the block
template <typename R>
struct MdBox {
    double L[3];
    float lf[3], hf[3];
    float reach_sq, queue_sq;  // squared reach of a bead, and with kMdWay more
    int cs[2];
    uint64_t seed;
    long long off;
    int r, nl, na;        // replica; listed and active particles
    int run[2];           // entries per leaf of the tree, each bead's list
    int cur;              // buffer of the replica's current arrays
    int words;            // of a bead's map (md_bits)
    bool all_mapped;      // it covers both lists
    MdParts<R> parts;
    // The active particles beyond parts.cap: the next far.cap in global memory, field
    // by field by their place in act (p[3], v[3], o[3], g[3], the step's force; what
    // the step has for the particle, flags, species), so that a warp reads whole lines,
    // and any more where they are.  One dimer of sigma = 5 in 40^3 cells, ms per interval FP64, FP32:
    // 13.2, 8.7 with all of them where they are, 9.5, 5.4 so
    MdParts<R> far;
};

// The beads of a replica in warp 0 of its block 0: lane 3 i + k has component k of
// bead i (the other lanes mirror lane 0), so that the divisions of a
// velocity-Verlet half or a RATTLE correction run side by side.  The divisors
// are kept with their reciprocals: a step is a chain of five quotients and a
// root, each waiting for the one before.
struct MdBead {
    double pos, vel, force, fold;
    Quotient vv, m, kk;  // 2 x own mass; own RATTLE mass; bond^2 (1/m1 + 1/m2)
    double dt_inv_mass;    // dt (1/m1 + 1/m2)
    double L;
    int i, k, sp0, sp1;
};

// What the turn needs of the beads' positions alone, before the step's forces
// are there: separation, its square, the reciprocal of RATTLE's divisor and
// the beads' own force (compute_force_n2, src/neighbor_list.f90:227-264)
struct MdPair {
    double s, rsq, f;
    Quotient g;
    bool acts;
};

// The block's shared memory: the step's bead positions and decisions, the queue
// of particles that need more than free flight; behind it the pair forces
// (MdTotals), the maps of the lists' entries (md_bits, md_base) and the particles,
// field by field (MdParts).
//
// What orders the words that both groups of warps use.  A step k has two points
// between the groups: kBarForces, at which the particles' warps arrive without
// waiting when the step's pair forces are pushed, and kBarTurn, at which all wait.
// A bead warp may thus still be in front of kBarForces(k), its loop test
// included, while the particles are at the second half of step k: a word that they
// write there and a bead warp reads before kBarForces has two places, used in
// turn.
template <typename R>
struct MdShared {
    MdBox<R> box;
    double x[2][6];         // bead positions, by step parity
    double old[6], rat[6];  // pos_old and pos_rattle of the beads
    double f[2][3];         // the beads' force sums
    double wsum[2][3][kNlBlockThreads / 32];
    // re-sort in front of step k's forces: by the beads or s_free (written by warp 0
    // between kBarForces(k - 1) and kBarTurn(k - 1), read by all between kBarTurn(k -
    // 1) and kBarForces(k)); by an active particle's displacement, by step parity
    // (written for step k by the particles between their arrival at kBarForces(k - 1)
    // and kBarTurn(k - 1), read like stop: a slow bead warp reads its step's
    // place, which is not written again before kBarTurn(k))
    int stop, over[2];
    int last;               // this block is the launch's last
    int anew;               // a bead went farther than kMdWay (written like stop, read by the particles before kBarForces)
    // step + 1 of the last one with a term in global memory, and with one whose place
    // is beyond the map (written before kBarForces, read after it)
    int spill, unmapped;
    // by step parity: particles queued for step k (counted by the particles after
    // kBarForces(k - 1), read by them before kBarForces(k), cleared by the beads
    // between that and kBarTurn(k)); pair forces per bead (counted before
    // kBarForces(k), read and cleared by the beads after it)
    int nq[2], cnt[2][2];
    int tot[2];             // slow sums: terms gathered
    int ws[33];
    int q[2][kMdQueue];     // queued particles, by step parity
};

// the pair forces of a step, each with its list entry and the step that wrote
// it, and what puts them in order
struct MdTotals {
    double f[2][3][kMdTerms], g[2][3][kMdTerms];  // as they come, and in order
    int2 te[2][kMdTerms];                         // step + 1, place in the order of addition
};

template <typename R>
__host__ __device__ constexpr size_t md_totals_at()
{
    return (sizeof(MdShared<R>) + 15) & ~(size_t)15;
}
template <typename R>
__host__ __device__ constexpr size_t md_map_at()
{
    return (md_totals_at<R>() + sizeof(MdTotals) + 15) & ~(size_t)15;
}
// Bead i's map: the places in its order of addition that have a term in this step,
// and the terms before each word's places (at offsets from the block's shared memory
// itself, not through a pointer, which would make every access a generic one)
template <typename R>
__device__ __forceinline__ unsigned *md_bits(const MdBox<R> &B, int i)
{
    extern __shared__ __align__(16) unsigned char md_smem[];
    return reinterpret_cast<unsigned *>(md_smem + md_map_at<R>()) + i * B.words;
}
template <typename R>
__device__ __forceinline__ int *md_base(const MdBox<R> &B, int i)
{
    return reinterpret_cast<int *>(md_bits(B, 2 + i));
}

// the block's named barriers: of the summing warps, and between them and the
// particles' warps (arrive: without waiting)
__device__ __forceinline__ void md_sync(int id, int threads)
{
    asm volatile("barrier.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void md_arrive(int id, int threads)
{
    asm volatile("barrier.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
constexpr int kBarSum = 1, kBarPart = 2, kBarForces = 3, kBarTurn = 4, kBarReady = 5;

// md_pos (src/md.f90:61-77), the PAST_MD / MD roll (src/neighbor_list.f90:180-188)
// and whether the particle's displacement is sqrt(d2) >= thr
// (src/particle_system.f90:357-378: not for species < 0); the exact test runs
// where the one in single precision is not clear
template <typename R>
__device__ __forceinline__ bool md_begin(Part<R> &q, R dt, R dt_sq, int read_species, double thr, float near_sq)
{
    const bool md = (q.f >> MD_BIT) & 1;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        if (!md) q.g[k] = 0;
        q.p[k] = q.p[k] + dt * q.v[k] + dt_sq * q.g[k];
    }
    q.f = md ? q.f | (1 << PAST_MD_BIT) : q.f & ~(1 << PAST_MD_BIT);
    q.f &= ~(1 << MD_BIT);
    const float c0 = (float)(q.p[0] - q.o[0]), c1 = (float)(q.p[1] - q.o[1]), c2 = (float)(q.p[2] - q.o[2]);
    if (c0 * c0 + c1 * c1 + c2 * c2 < near_sq) return false;
    if (read_species && q.sp < 0) return false;
    const double d0 = (double)q.p[0] - (double)q.o[0], d1 = (double)q.p[1] - (double)q.o[1],
                 d2 = (double)q.p[2] - (double)q.o[2];
    return sqrt(d0 * d0 + d1 * d1 + d2 * d2) >= thr;
}

__device__ __forceinline__ float md_image_f(float d, float L, float h)
{
    return d < -h ? d + L : d > h ? d - L : d;
}

template <typename R>
__device__ __forceinline__ const PView<R> &md_view(const MdArgs<R> &A, const MdBox<R> &B)
{
    return B.cur ? A.v1 : A.v0;
}
template <typename R>
__device__ __forceinline__ const Vec3<R> &md_old(const MdArgs<R> &A, const MdBox<R> &B)
{
    return B.cur ? A.v0.pos : A.v1.pos;
}

// What a particle at p with flags f has to do besides flying freely: bit h, bead h
// may be within reach (squared; a distance in single precision decides), bit 2,
// it has flags.  Three quarters of the active particles have nothing.
template <typename R>
__device__ __forceinline__ int md_busy(const double *X, const MdBox<R> &B, const R p[3], int f, float reach_sq)
{
    float d[2] = {0, 0};
#pragma unroll
    for (int k = 0; k < 3; k++)
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const float c = md_image_f((float)X[3 * i + k] - (float)p[k], B.lf[k], B.hf[k]);
            d[i] += c * c;
        }
    return (d[0] > reach_sq ? 0 : 1) | (d[1] > reach_sq ? 0 : 2) | ((f & kActiveBits) ? 4 : 0);
}

// where active particle i is kept during the launch
constexpr int kShared = 0, kFar = 1, kInPlace = 2;
template <typename R>
__device__ __forceinline__ int md_tier(const MdBox<R> &B, int i)
{
    return i < B.parts.cap ? kShared : i - B.parts.cap < B.far.cap ? kFar : kInPlace;
}

// from the particle arrays
template <typename R>
__device__ __forceinline__ Part<R> md_read_in_place(const MdBox<R> &B, const MdArgs<R> &A, int idx)
{
    Part<R> q;
    q.f = md_view(A, B).flags[idx];
    q.sp = md_view(A, B).species[idx];
    const bool forced = q.f & ((1 << MD_BIT) | (1 << PAST_MD_BIT));
#pragma unroll
    for (int k = 0; k < 3; k++) {
        q.p[k] = md_view(A, B).pos[k][idx];
        q.v[k] = md_view(A, B).vel[k][idx];
        q.o[k] = md_old(A, B)[k][idx];
        q.g[k] = forced ? md_view(A, B).force[k][idx] : (R)0;
    }
    return q;
}
template <typename R>
__device__ __forceinline__ void md_write_in_place(const MdBox<R> &B, const MdArgs<R> &A, int idx, const Part<R> &q)
{
    md_view(A, B).flags[idx] = q.f;
    md_view(A, B).species[idx] = q.sp;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        md_view(A, B).pos[k][idx] = q.p[k];
        md_view(A, B).vel[k][idx] = q.v[k];
        md_view(A, B).force[k][idx] = q.g[k];
    }
}

// from, and to, where particle i is kept
template <int kTier, typename R>
__device__ __forceinline__ Part<R> md_read(const MdBox<R> &B, const MdArgs<R> &A, int i)
{
    if constexpr (kTier == kInPlace) {
        return md_read_in_place(B, A, A.act[B.off + i]);
    } else {
        const MdParts<R> &m = kTier == kShared ? B.parts : B.far;
        const int s = kTier == kShared ? i : i - B.parts.cap;
        Part<R> q;
        q.f = m.num(1, s);
        q.sp = m.num(2, s);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            q.p[k] = m.real(k, s);
            q.v[k] = m.real(3 + k, s);
            q.o[k] = m.real(6 + k, s);
            q.g[k] = m.real(9 + k, s);
        }
        return q;
    }
}
template <int kTier, typename R>
__device__ __forceinline__ void md_write(const MdBox<R> &B, const MdArgs<R> &A, int i, const Part<R> &q)
{
    if constexpr (kTier == kInPlace) {
        md_write_in_place(B, A, A.act[B.off + i], q);
    } else {
        const MdParts<R> &m = kTier == kShared ? B.parts : B.far;
        const int s = kTier == kShared ? i : i - B.parts.cap;
        m.num(1, s) = q.f;
        m.num(2, s) = q.sp;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            m.real(k, s) = q.p[k];
            m.real(3 + k, s) = q.v[k];
            m.real(9 + k, s) = q.g[k];
        }
    }
}

// multiplicities and entries of particle i in the two lists
template <typename R>
__device__ __forceinline__ int md_entries(const MdBox<R> &B, const MdArgs<R> &A, int i, int e[2])
{
    if (i < B.parts.cap) {
        e[0] = B.parts.num(4, i);
        e[1] = B.parts.num(5, i);
        return B.parts.num(3, i);
    }
    if (i >= B.nl) return 0;
    const size_t w = (size_t)2 * B.r * A.Nmax + i;
    e[0] = A.ent[2 * w];
    e[1] = A.ent[2 * w + 1];
    return A.mult[w];
}

// The place of entry e in the order in which a bead's pair forces are added: list
// order in the FP64 form; in the FP32 form leaf by leaf of colloid_tree_block's
// tree (entries t, t + 256, ... of leaf t in that order), run entries per leaf.
template <typename R>
__device__ __forceinline__ int md_order(int e, int run)
{
    return sizeof(R) == 8 ? e : (e & (kNlBlockThreads - 1)) * run + (e >> 8);
}

// The pair force f of bead i, once for each of the particle's entries in its
// list: the term, and the entry's bit in the bead's map (terms without room to
// global memory)
template <typename R>
__device__ __forceinline__ void md_push(MdShared<R> &sh, const MdBox<R> &B, const MdArgs<R> &A, MdTotals &tot, int i,
                                        int k, int e, int times, double f0, double f1, double f2)
{
    const int par = k & 1;
    for (int t = 0; t < times; t++) {
        const int s = atomicAdd(&sh.cnt[par][i], 1), o = md_order<R>(e, B.run[i]);
        const bool mapped = (o >> 5) < B.words;
        if (mapped) atomicOr(md_bits(B, i) + (o >> 5), 1u << (o & 31));
        if (mapped && s < kMdTerms) {
            tot.te[i][s] = make_int2(k + 1, o);
            tot.f[i][0][s] = f0;
            tot.f[i][1][s] = f1;
            tot.f[i][2][s] = f2;
        } else {
            const int b = 2 * B.r + i;
            const int at = B.all_mapped ? s - kMdTerms : atomicAdd(A.n_over + 2 * b + par, 1);
            MdTerm *g = A.over + (size_t)b * A.Nmax + at;
            g->e = o;
            g->f[0] = f0;
            g->f[1] = f1;
            g->f[2] = f2;
            sh.spill = k + 1;
            if (!mapped) sh.unmapped = k + 1;
        }
        if (t + 1 < times) e = A.next[(size_t)(2 * B.r + i) * A.Nmax + e];
    }
}

// pair forces of a queued particle's list entries (src/neighbor_list.f90:198-219,
// in (bead, entry) order) and flag_particles_nl of the catalytic bead
// (programs/single_dimer_pbc.f90:493-509): the step's force and the flags
template <typename R>
__device__ __forceinline__ int md_forces(MdShared<R> &sh, const MdBox<R> &B, const MdArgs<R> &A, MdTotals &tot, int i,
                                         int k, const R p[3], int sp, int f, R nf[3])
{
    int e[2];
    const int m = md_entries(B, A, i, e);
    const double *X = sh.x[k & 1];
    nf[0] = nf[1] = nf[2] = 0;
    if (!m || sp <= 0) return f;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int times = h ? m >> 16 : m & 0xffff;
        if (!times) continue;
        const double d0 = min_image_d(X[3 * h] - (double)p[0], B.L[0]),
                     d1 = min_image_d(X[3 * h + 1] - (double)p[1], B.L[1]),
                     d2 = min_image_d(X[3 * h + 2] - (double)p[2], B.L[2]);
        const double r_sq = d0 * d0 + d1 * d1 + d2 * d2;
        const int tt = (sp - 1) + A.lj_sc.n1 * (B.cs[h] - 1);
        if (r_sq <= A.lj_sc.cut_sq[tt]) {
            const double fr = lj_force_over_r(r_sq, A.lj_sc.epsilon[tt], A.lj_sc.sigma[tt]);
            const double f0 = fr * d0, f1 = fr * d1, f2 = fr * d2;
            for (int t = 0; t < times; t++) {
                nf[0] = nf[0] - (R)f0;
                nf[1] = nf[1] - (R)f1;
                nf[2] = nf[2] - (R)f2;
            }
            md_push(sh, B, A, tot, h, k, e[h], times, f0, f1, f2);
            f |= (1 << MD_BIT) | (B.cs[h] == 1 ? (1 << CATALYZED_BIT) : 0);
        }
        if (h == 0 && sp == 1 && r_sq < A.cut_c) f |= 1 << REAC_BIT;
    }
    return f;
}

// the pair force of bead h on particle i of the shared memory: to the
// particle's pf, with what came of it, and to the bead's terms
template <typename R>
__device__ __forceinline__ void md_pair_force(MdShared<R> &sh, const MdBox<R> &B, const MdArgs<R> &A, MdTotals &tot,
                                              int i, int h, int k)
{
    const double *X = sh.x[k & 1] + 3 * h;
    const int sp = B.parts.num(2, i), m = B.parts.num(3, i), times = h ? m >> 16 : m & 0xffff;
    if (!times || sp <= 0) return;
    const double d0 = min_image_d(X[0] - (double)B.parts.real(0, i), B.L[0]),
                 d1 = min_image_d(X[1] - (double)B.parts.real(1, i), B.L[1]),
                 d2 = min_image_d(X[2] - (double)B.parts.real(2, i), B.L[2]);
    const double r_sq = d0 * d0 + d1 * d1 + d2 * d2;
    const int tt = (sp - 1) + A.lj_sc.n1 * (B.cs[h] - 1);
    if (r_sq <= A.lj_sc.cut_sq[tt]) {
        const double fr = lj_force_over_r(r_sq, A.lj_sc.epsilon[tt], A.lj_sc.sigma[tt]);
        const double f0 = fr * d0, f1 = fr * d1, f2 = fr * d2;
        md_push(sh, B, A, tot, h, k, B.parts.num(4 + h, i), times, f0, f1, f2);
        B.parts.real(12 + 3 * h, i) = (R)f0;
        B.parts.real(13 + 3 * h, i) = (R)f1;
        B.parts.real(14 + 3 * h, i) = (R)f2;
        atomicOr(&B.parts.num(7, i), 1 << h);
    }
    if (h == 0 && sp == 1 && r_sq < A.cut_c) atomicOr(&B.parts.num(7, i), 4);
}

// md_vel (src/md.f90:219-237) and change_species
// (programs/single_dimer_pbc.f90:511-542) of a queued particle, given the step's
// force nf
template <typename R>
__device__ __forceinline__ void md_end(Part<R> &q, const double *X, const MdBox<R> &B, const MdArgs<R> &A,
                                       const R nf[3], int idx, uint64_t step)
{
    const R dt = A.dt_r;
    if (!((q.f >> WALL_BIT) & 1)) {
        if (q.f & ((1 << MD_BIT) | (1 << PAST_MD_BIT))) {
#pragma unroll
            for (int k = 0; k < 3; k++) q.v[k] = q.v[k] + dt * (nf[k] + q.g[k]) / 2;
        } else {
#pragma unroll
            for (int k = 0; k < 3; k++) q.v[k] = md_vel_free(q.v[k], dt);
        }
    } else {
        q.f &= ~(1 << WALL_BIT);
    }
    if ((q.f >> REAC_BIT) & 1) {
        double d[2];
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const double d0 = min_image_d(X[3 * i] - (double)q.p[0], B.L[0]),
                         d1 = min_image_d(X[3 * i + 1] - (double)q.p[1], B.L[1]),
                         d2 = min_image_d(X[3 * i + 2] - (double)q.p[2], B.L[2]);
            d[i] = d0 * d0 + d1 * d1 + d2 * d2;
        }
        if ((d[0] > A.cut_c) && (d[1] > A.cut_n)) {
            double u0, u1;
            rng::uniform2(B.seed, step, (uint32_t)(idx - B.off), rng::REACT, 0, u0, u1);
            if (u0 <= A.prob) q.sp = 2;
            q.f &= ~(1 << REAC_BIT);
        }
    }
#pragma unroll
    for (int k = 0; k < 3; k++) q.g[k] = nf[k];
}

// a warp's level of the tree of colloid_tree_block: its leaves' sums to wsum
template <typename R>
__device__ __forceinline__ void md_tree_warp(MdShared<R> &sh, double3 leaf, int h, int l)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        leaf.x = leaf.x + __shfl_xor_sync(0xffffffffu, leaf.x, o);
        leaf.y = leaf.y + __shfl_xor_sync(0xffffffffu, leaf.y, o);
        leaf.z = leaf.z + __shfl_xor_sync(0xffffffffu, leaf.z, o);
    }
    if ((l & 31) == 0) {
        sh.wsum[h][0][l >> 5] = leaf.x;
        sh.wsum[h][1][l >> 5] = leaf.y;
        sh.wsum[h][2][l >> 5] = leaf.z;
    }
}

// A list whose entries the map does not cover (more than 196,608: beads of sigma = 12
// at density 10): both beads' terms are put in order in global memory by their places
// and added from there, half of the summing warps per bead (FP32: up to the tree's
// warp level).
template <typename R>
__device__ __noinline__ void md_slow_sums(MdShared<R> &sh, const MdArgs<R> &A, const MdTotals &tt, int r, int k)
{
    constexpr int H = kMdSum / 2;
    const int h = threadIdx.x / H, t = threadIdx.x % H, b = 2 * r + h;
    MdTerm *terms = A.terms + (size_t)b * A.Nmax;
    const MdTerm *over = A.over + (size_t)b * A.Nmax;
    unsigned long long *ka = A.keys[0] + (size_t)b * A.Nmax, *kb = A.keys[1] + (size_t)b * A.Nmax;
    if (threadIdx.x < 2) sh.tot[threadIdx.x] = 0;
    md_sync(kBarSum, kMdSum);
    const int m = *(volatile int *)(A.n_over + 2 * b + (k & 1));
    for (int j = t; j < kMdTerms + m; j += H) {
        MdTerm x;
        if (j < kMdTerms) {
            if (tt.te[h][j].x != k + 1) continue;
            x.e = tt.te[h][j].y;
            for (int c = 0; c < 3; c++) x.f[c] = tt.f[h][c][j];
        } else {
            x.e = __ldcg(&over[j - kMdTerms].e);
            for (int c = 0; c < 3; c++) x.f[c] = __ldcg(&over[j - kMdTerms].f[c]);
        }
        const int at = atomicAdd(&sh.tot[h], 1);
        terms[at] = x;
        ka[at] = ((unsigned long long)x.e << 32) | (unsigned)at;
    }
    md_sync(kBarSum, kMdSum);
    const int n = sh.tot[h], most = max(sh.tot[0], sh.tot[1]);
    for (int w = 1; w < most; w <<= 1) {
        for (int i = t; i < n; i += H) {
            const int run = i / w, r0 = run * w;
            const unsigned long long v = ka[i];
            const int p0 = (run & 1) ? r0 - w : r0 + w, pn = (run & 1) ? w : min(w, max(0, n - p0));
            int lo = 0, hi = pn;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (ka[p0 + mid] < v) lo = mid + 1;
                else hi = mid;
            }
            kb[((run & 1) ? p0 : r0) + (i - r0) + lo] = v;
        }
        md_sync(kBarSum, kMdSum);
        unsigned long long *x = ka;
        ka = kb;
        kb = x;
    }
    if constexpr (sizeof(R) == 8) {
        if (t < 3) {
            double acc = 0;
#pragma unroll 8
            for (int j = 0; j < n; j++) acc = acc + terms[(unsigned)ka[j]].f[t];
            sh.f[h][t] = acc;
        }
    } else {
        // every leaf's run of the sorted keys, then the tree
        const int run = sh.box.run[h];
        for (int q = 0; q < 2; q++) {
            const int l = t + q * H;
            int lo = 0, hi = n;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if ((int)(ka[mid] >> 32) < l * run) lo = mid + 1;
                else hi = mid;
            }
            double3 leaf = make_double3(0, 0, 0);
            for (int j = lo; j < n && (int)(ka[j] >> 32) < (l + 1) * run; j++) {
                const MdTerm &x = terms[(unsigned)ka[j]];
                leaf.x = leaf.x + x.f[0];
                leaf.y = leaf.y + x.f[1];
                leaf.z = leaf.z + x.f[2];
            }
            md_tree_warp(sh, leaf, h, l);
        }
    }
}

// acc and the m terms g[0, m) one after another
__device__ __forceinline__ double md_chain(double acc, const double *g, int m)
{
    int j = 0;
    if (m >= 8) {
        double v[8], u[8];
#pragma unroll
        for (int c = 0; c < 8; c++) v[c] = g[c];
        for (; j + 16 <= m; j += 8) {
#pragma unroll
            for (int c = 0; c < 8; c++) u[c] = g[j + 8 + c];
#pragma unroll
            for (int c = 0; c < 8; c++) acc = acc + v[c];
#pragma unroll
            for (int c = 0; c < 8; c++) v[c] = u[c];
        }
#pragma unroll
        for (int c = 0; c < 8; c++) acc = acc + v[c];
        j += 8;
    }
    for (; j < m; j++) acc = acc + g[j];
    return acc;
}

// sh.f[h] = the sum of bead h's pair forces (src/neighbor_list.f90:214-218), half
// of the summing warps per bead.  The bit map gives every term its place among
// the step's terms; the FP64 form adds them one after another in list order,
// one thread per component, as the reference does; the FP32 form adds each
// leaf's terms and then up colloid_tree_block's tree.  In order they stand in shared
// memory, or in the bead's part of A.terms, component by component, in a step with
// more of them (beads larger than sigma = 4 at density 10).
template <typename R>
__device__ __forceinline__ void md_colloid_sums(MdShared<R> &sh, MdTotals &tt, const MdArgs<R> &A, int r, int n0,
                                                int n1, int k)
{
    constexpr int H = kMdSum / 2;
    const int h = threadIdx.x / H, t = threadIdx.x % H, lane = t & 31, w = t >> 5;
    const int n = h ? n1 : n0;
    if (sh.unmapped == k + 1) {
        md_slow_sums<R>(sh, A, tt, r, k);
    } else {
        // terms before each word: a warp per bead, runs of words per lane
        const unsigned *bits = md_bits(sh.box, h);
        int *base = md_base(sh.box, h);
        const int places = sizeof(R) == 8 ? n : kNlBlockThreads * sh.box.run[h];
        const int words = min((places + 31) / 32, sh.box.words), m = sh.cnt[k & 1][h];
        const bool spilled = sh.spill == k + 1;
        double *far = (double *)(A.terms + (size_t)(2 * r + h) * A.Nmax);
        if (w == 0) {
            const int per = (words + 31) / 32, q0 = min(words, lane * per), q1 = min(words, q0 + per);
            int c = 0;
            for (int q = q0; q < q1; q++) c += __popc(bits[q]);
            int inc = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += y;
            }
            int run = inc - c;
            for (int q = q0; q < q1; q++) {
                base[q] = run;
                run += __popc(bits[q]);
            }
        }
        md_sync(kBarSum, kMdSum);
        // the terms before place o
        auto before = [&](int o) { return (o >> 5) >= words ? m : base[o >> 5] + __popc(bits[o >> 5] & ((1u << (o & 31)) - 1u)); };
        // into order
        if (!spilled) {
            for (int j = t; j < m; j += H) {
                const int at = before(tt.te[h][j].y);
                tt.g[h][0][at] = tt.f[h][0][j];
                tt.g[h][1][at] = tt.f[h][1][j];
                tt.g[h][2][at] = tt.f[h][2][j];
            }
        } else {
            const MdTerm *over = A.over + (size_t)(2 * r + h) * A.Nmax;
            for (int j = t; j < m; j += H) {
                const bool in = j < kMdTerms;
                const int at = before(in ? tt.te[h][j].y : __ldcg(&over[j - kMdTerms].e));
                for (int c = 0; c < 3; c++)
                    far[(size_t)c * A.Nmax + at] = in ? tt.f[h][c][j] : __ldcg(&over[j - kMdTerms].f[c]);
            }
        }
        md_sync(kBarSum, kMdSum);
        if constexpr (sizeof(R) == 8) {
            if (!spilled) {
                if (t < 3) sh.f[h][t] = md_chain(0.0, tt.g[h][t], m);
            } else {
                // a part at a time into shared memory: the chain of adds is not to
                // wait for a line from L2 every 16 terms
                const int most = max(sh.cnt[k & 1][0], sh.cnt[k & 1][1]);
                double acc = 0;
                for (int c0 = 0; c0 < most; c0 += kMdTerms) {
                    const int mc = min(kMdTerms, m - c0);
                    for (int j = t; j < mc; j += H)
                        for (int c = 0; c < 3; c++) tt.g[h][c][j] = far[(size_t)c * A.Nmax + c0 + j];
                    md_sync(kBarSum, kMdSum);
                    if (t < 3) acc = md_chain(acc, tt.g[h][t], mc);
                    md_sync(kBarSum, kMdSum);
                }
                if (t < 3) sh.f[h][t] = acc;
            }
        } else {
            const int run = sh.box.run[h];
            for (int q = 0; q < 2; q++) {
                const int l = t + q * H;
                const int lo = run ? before(l * run) : 0, hi = run && l < kNlBlockThreads - 1 ? before((l + 1) * run) : m;
                double3 leaf = make_double3(0, 0, 0);
                if (!spilled) {
                    for (int j = lo; j < hi; j++) {
                        leaf.x = leaf.x + tt.g[h][0][j];
                        leaf.y = leaf.y + tt.g[h][1][j];
                        leaf.z = leaf.z + tt.g[h][2][j];
                    }
                } else {
                    for (int j = lo; j < hi; j++) {
                        leaf.x = leaf.x + far[j];
                        leaf.y = leaf.y + far[(size_t)A.Nmax + j];
                        leaf.z = leaf.z + far[2 * (size_t)A.Nmax + j];
                    }
                }
                md_tree_warp(sh, leaf, h, l);
            }
        }
    }
    if constexpr (sizeof(R) == 4) {
        md_sync(kBarSum, kMdSum);
        if (w == 0) {
            constexpr int NW = kNlBlockThreads / 32;
            double b0 = lane < NW ? sh.wsum[h][0][lane] : 0.0, b1 = lane < NW ? sh.wsum[h][1][lane] : 0.0,
                   b2 = lane < NW ? sh.wsum[h][2][lane] : 0.0;
#pragma unroll
            for (int o = NW / 2; o > 0; o >>= 1) {
                b0 = b0 + __shfl_xor_sync(0xffffffffu, b0, o);
                b1 = b1 + __shfl_xor_sync(0xffffffffu, b1, o);
                b2 = b2 + __shfl_xor_sync(0xffffffffu, b2, o);
            }
            if (lane == 0) {
                sh.f[h][0] = b0;
                sh.f[h][1] = b1;
                sh.f[h][2] = b2;
            }
        }
    }
    md_sync(kBarSum, kMdSum);
}

__device__ __forceinline__ double md_lane(double x, int l) { return __shfl_sync(0xffffffffu, x, l); }
// x . y of values whose components lanes l0, l0 + 1, l0 + 2 hold
__device__ __forceinline__ double md_dot(double x, double y, int l0)
{
    const double p = x * y;
    return md_lane(p, l0) + md_lane(p, l0 + 1) + md_lane(p, l0 + 2);
}

template <typename R>
__device__ __forceinline__ MdPair md_pair(const MdBead &b, const MdArgs<R> &A)
{
    MdPair p;
    p.s = min_image_d(md_lane(b.pos, b.k) - md_lane(b.pos, b.k + 3), b.L);
    p.rsq = md_dot(p.s, p.s, 0);
    p.g.set(b.dt_inv_mass * p.rsq);
    p.acts = p.rsq <= A.lj_cc.cut_sq[(b.sp0 - 1) + A.lj_cc.n1 * (b.sp1 - 1)];
    p.f = 0;
    if (p.acts) {
        const int tt = (b.sp1 - 1) + A.lj_cc.n1 * (b.sp0 - 1);
        p.f = lj_force_over_r(p.rsq, A.lj_cc.epsilon[tt], A.lj_cc.sigma[tt]) * p.s;
    }
    return p;
}

// compute_force_n2, the colloid velocity half and RATTLE's velocity correction
// (src/neighbor_list.f90:227-264, programs/single_dimer_pbc.f90:356-359,
// src/md.f90:298-319), the arithmetic of force_n2_one, colloid_vv_vel_one and
// rattle_vel_dimer
template <typename R>
__device__ __forceinline__ void md_colloid_end(MdBead &b, const MdPair &p, const MdArgs<R> &A)
{
    if (p.acts) b.force = b.i == 0 ? b.force + p.f : b.force - p.f;
    b.vel = b.vel + b.vv.of(A.dt * (b.force + b.fold));
    const double dv = md_lane(b.vel, b.k) - md_lane(b.vel, b.k + 3);
    const double kk = b.kk.of(md_dot(dv, p.s, 0));
    const double c = b.m.of(kk * p.s);
    b.vel = b.i == 0 ? b.vel - c : b.vel + c;
}

// the colloid position half, RATTLE (colloid_vv_pos_one, rattle_pos_dimer) and
// switch_force (programs/single_dimer_pbc.f90:311-322); returns the beads' largest
// displacement
template <typename R>
__device__ __forceinline__ double md_colloid_begin(MdShared<R> &sh, MdBead &b, const MdPair &p, const MdArgs<R> &A)
{
    if (threadIdx.x < 6) sh.rat[threadIdx.x] = b.pos;
    b.pos = b.pos + A.dt * b.vel + b.vv.of(A.dt * A.dt * b.force);
    const double s = min_image_d(md_lane(b.pos, b.k) - md_lane(b.pos, b.k + 3), b.L);
    const double ssq = md_dot(s, s, 0), rs = md_dot(p.s, s, 0);
    const double disc = rs * rs - p.rsq * (ssq - A.bond * A.bond);
    if (disc < 0 && threadIdx.x == 0) atomicOr(A.err, DEV_ERR_RATTLE);
    const double g = p.g.of(rs - sqrt(disc));
    const double dp = b.m.of(g * A.dt * p.s), dv = b.m.of(g * p.s);
    b.pos = b.i == 0 ? b.pos - dp : b.pos + dp;
    b.vel = b.i == 0 ? b.vel - dv : b.vel + dv;
    const double d = b.pos - sh.old[3 * b.i + b.k];
    const double q0 = md_dot(d, d, 0), q1 = md_dot(d, d, 3);
    const double m0 = b.sp0 < 0 ? 0 : q0, m1 = b.sp1 < 0 ? 0 : q1;
    b.fold = b.force;
    b.force = 0;
    return sqrt(m0 > m1 ? m0 : m1);
}

// warp 0: the end of MD step k - 1 (end), the colloid position half and the beads'
// part of the re-sort test of step k (begin; programs/single_dimer_pbc.f90:311-330),
// then the bead positions and the decision for all warps
template <typename R>
__device__ __forceinline__ void md_turn(MdShared<R> &sh, MdBead &b, const MdPair &p, const MdArgs<R> &A, int k,
                                        int s_free, bool end, bool begin)
{
    const int lane = threadIdx.x;
    if (end) {
        b.force = b.force + sh.f[b.i][b.k];
        md_colloid_end<R>(b, p, A);
    }
    if (begin) {
        const double from = b.pos;
        const double co = md_colloid_begin<R>(sh, b, p, A);
        // (not "less than": a NaN makes the queue anew as well)
        const bool far = __any_sync(0xffffffffu, !((float)fabs(b.pos - from) < 0.5f * kMdWay));
        if (lane < 6) sh.x[k & 1][lane] = b.pos;
        if (lane == 6) sh.stop = (co >= A.skin * 0.1) || k >= s_free;
        if (lane == 7) sh.anew = far;
    }
}

// The MD steps of every replica (start) or of those that were re-sorted
// (resort[r]), one block per replica, each until its next re-sort or the
// interval's end.  A step: the queued particles -- those a bead may reach, by a
// distance in single precision, and those with flags -- get their pair forces;
// while the first eight warps add these in order and move the beads, the
// others move the particles and queue those of the next step.  Latency bound:
// one pair force, the ordered sum and the beads' chain of quotients, one after
// the other, at an instruction every ~6 cycles of a code that no warp runs
// twice in a row; FP64 throughput and memory play no part.  (A cluster of eight
// blocks per replica spent two cluster barriers of ~2,000 cycles per step.)
template <typename R>
__global__ void __launch_bounds__(kMdThreads, 1) kb_md(const __grid_constant__ MdArgs<R> A)
{
    extern __shared__ __align__(16) unsigned char md_smem[];
    MdShared<R> &sh = *reinterpret_cast<MdShared<R> *>(md_smem);
    constexpr size_t kMap = md_map_at<R>();
    static_assert(kMap + 16 * (size_t)kMdMapWords + 32 * 1024 <= kMdSmem, "room for particles");
    MdTotals &totals = *reinterpret_cast<MdTotals *>(md_smem + md_totals_at<R>());
    const int r = blockIdx.x;
    const int t = threadIdx.x;
    const int all = blockDim.x;
    if (A.start || A.resort[r]) {
        const BRep &rp = A.rep[r];
        MdBox<R> &W = sh.box;
        if (t == 0) {
            W.off = rp.off;
            W.seed = rp.seed;
            W.r = r;
            for (int k = 0; k < 3; k++) {
                W.L[k] = rp.g.edges[k];
                W.lf[k] = (float)rp.g.edges[k];
                W.hf[k] = 0.5f * (float)rp.g.edges[k];
            }
            for (int i = 0; i < 2; i++) W.cs[i] = A.c.species[2 * r + i];
            // single precision of positions inside twice the box: 1e-5 of the
            // edges is far above the rounding of a distance
            const float reach = A.reach + 1e-5f * (float)(rp.g.edges[0] + rp.g.edges[1] + rp.g.edges[2]);
            W.reach_sq = reach * reach;
            W.queue_sq = (reach + kMdWay) * (reach + kMdWay);
            W.cur = rp.cur;
            W.nl = A.nl[r];
            W.na = W.nl + A.nx[r];
            for (int h = 0; h < 2; h++) W.run[h] = (A.n[2 * r + h] + kNlBlockThreads - 1) / kNlBlockThreads;
            // (the FP32 form's leaves are of whole runs)
            const int places = kNlBlockThreads * max(W.run[0], W.run[1]);
            W.words = min(kMdMapWords, places / 32);
            W.all_mapped = 32 * W.words == places;
            const size_t parts = kMap + 16 * (size_t)W.words;
            W.parts.cap = (int)((kMdSmem - parts) / md_part_bytes<R>());
            W.parts.r = reinterpret_cast<R *>(md_smem + parts);
            W.far.cap = A.far_cap;
            W.far.r = reinterpret_cast<R *>(A.far + (size_t)r * A.far_cap * md_far_bytes<R>());
            W.far.i = reinterpret_cast<int *>(W.far.r + 15 * (size_t)A.far_cap);
            W.parts.i = reinterpret_cast<int *>(W.parts.r + 18 * (size_t)W.parts.cap);
            sh.stop = sh.over[0] = sh.over[1] = sh.spill = sh.unmapped = 0;
            sh.anew = 1;
            for (int p = 0; p < 2; p++) {
                sh.nq[p] = sh.cnt[p][0] = sh.cnt[p][1] = 0;
                A.n_over[4 * r + 2 * p] = A.n_over[4 * r + 2 * p + 1] = 0;
            }
        }
        for (int q = t; q < 2 * kMdTerms; q += all) (&totals.te[0][0])[q] = make_int2(0, 0);
        __syncthreads();
        const MdBox<R> &B = sh.box;
        for (int q = t; q < 2 * B.words; q += all) md_bits(B, 0)[q] = 0;  // used after kBarReady
        const int s_free = A.s_free[r];
        int k = A.start ? 0 : A.adv[r] - 1;
        if (t < kMdSum) {
            // ---- the beads ----
            const int n0 = A.n[2 * r], n1 = A.n[2 * r + 1];
            MdBead b{};
            MdPair pair{};
            if (t < 32) {
                b.i = t < 6 ? t / 3 : 0;
                b.k = t < 6 ? t % 3 : 0;
                const int c = 2 * r + b.i;
                b.pos = A.c.pos[b.k][c];
                b.vel = A.c.vel[b.k][c];
                b.force = A.c.force[b.k][c];
                b.fold = A.c.force_old[b.k][c];
                if (t < 6) {
                    sh.old[t] = A.cold[b.k][c];
                    sh.rat[t] = A.rat[b.k][c];
                }
                __syncwarp();
                b.sp0 = B.cs[0];
                b.sp1 = B.cs[1];
                const double m1 = bead_mass(A.ms, B.cs, 0, A.err), m2 = bead_mass(A.ms, B.cs, 1, A.err);
                const double inv_mass = 1 / m1 + 1 / m2;
                b.vv.set(2 * A.mass[c]);
                b.m.set(b.i == 0 ? m1 : m2);
                b.kk.set(A.bond * A.bond * inv_mass);
                b.dt_inv_mass = A.dt * inv_mass;
                b.L = B.L[b.k];
                pair = md_pair<R>(b, A);
                if (A.start) {
                    md_turn<R>(sh, b, pair, A, k, s_free, false, true);
                    pair = md_pair<R>(b, A);
                } else if (t < 6) {
                    // resumed after a re-sort: the step's forces come next
                    sh.x[k & 1][t] = b.pos;
                }
                __syncwarp();
                if (t == 0) sh.anew = 1;  // there is no queue yet
            }
            md_sync(kBarReady, all);
            while (!(sh.stop | sh.over[k & 1])) {
                const bool last = k + 1 == A.N_MD;
                md_sync(kBarForces, all);
                md_colloid_sums<R>(sh, totals, A, r, n0, n1, k);
                if (t < 32) {
                    md_turn<R>(sh, b, pair, A, k + 1, s_free, true, !last);
                } else {
                    // ready for the step after the next forces
                    for (int q = t - 32; q < 2 * B.words; q += kMdSum - 32) md_bits(B, 0)[q] = 0;
                    if (t < 34) {
                        sh.cnt[k & 1][t - 32] = 0;
                        A.n_over[2 * (2 * r + t - 32) + (k & 1)] = 0;
                    }
                    if (t == 34) sh.nq[k & 1] = 0;
                }
                md_sync(kBarTurn, all);
                // in the shadow of the forces: what the next turn needs of the
                // positions
                if (t < 32) pair = md_pair<R>(b, A);
                k++;
                if (last) break;
            }
            if (t < 6) {
                const int c = 2 * r + b.i;
                A.c.pos[b.k][c] = b.pos;
                A.c.vel[b.k][c] = b.vel;
                A.c.force[b.k][c] = b.force;
                A.c.force_old[b.k][c] = b.fold;
                A.rat[b.k][c] = sh.rat[t];
            }
            if (t == 0) {
                const int need = k < A.N_MD;  // stopped in front of step k's forces
                A.adv[r] = need ? k + 1 : A.N_MD;
                A.resort[r] = need;
                if (need) A.n_extra[r] += 1;
            }
        } else {
            // ---- the particles ----
            const int me = t - kMdSum, threads = all - kMdSum;
            const bool fresh = A.fresh[r] != 0;
            const double thr = A.skin * 0.89;
            const float near_sq = 0.99f * (float)thr * (float)thr;
            const uint64_t step0 = *A.d_step;
            for (int i = me; i < B.na; i += threads) {
                const int idx = A.act[B.off + i], tier = md_tier(B, i);
                Part<R> q = md_read_in_place(B, A, idx);
                if (!fresh)
                    for (int c = 0; c < 3; c++) {
                        q.o[c] = q.p[c];
                        if (tier == kInPlace) md_old(A, B)[c][idx] = q.p[c];
                    }
                if (A.start) {
                    // force_old of the last interval's end is no longer current
                    if ((q.f >> PAST_MD_BIT) & 1)
                        for (int c = 0; c < 3; c++) md_view(A, B).force_old[c][idx] = 0;
                    if (md_begin(q, A.dt_r, A.dt_sq_r, A.read_species, thr, near_sq)) sh.over[k & 1] = 1;
                }
                if (i < B.parts.cap) {
                    B.parts.num(0, i) = idx;
                    int m = 0, e[2] = {0, 0};
                    if (i < B.nl) {
                        const size_t w = (size_t)2 * r * A.Nmax + i;
                        m = A.mult[w];
                        e[0] = A.ent[2 * w];
                        e[1] = A.ent[2 * w + 1];
                    }
                    B.parts.num(3, i) = m;
                    B.parts.num(4, i) = e[0];
                    B.parts.num(5, i) = e[1];
                    for (int c = 0; c < 3; c++) B.parts.real(6 + c, i) = q.o[c];
                    md_write<kShared>(B, A, i, q);
                } else if (tier == kFar) {
                    for (int c = 0; c < 3; c++) B.far.real(6 + c, i - B.parts.cap) = q.o[c];
                    md_write<kFar>(B, A, i, q);
                } else {
                    md_write_in_place(B, A, idx, q);
                }
            }
            md_sync(kBarReady, all);
            while (!(sh.stop | sh.over[k & 1])) {
                const bool last = k + 1 == A.N_MD;
                const int par = k & 1;
                const double *X = sh.x[par];
                const int shared = min(B.na, B.parts.cap);
                if (sh.anew || sh.nq[par] > kMdQueue) {
                    // no queue (the first step, a bead that leapt) or one too long
                    for (int i = me; i < shared; i += threads) {
                        const R p[3] = {B.parts.real(0, i), B.parts.real(1, i), B.parts.real(2, i)};
                        const int m = md_busy(X, B, p, B.parts.num(1, i), B.queue_sq);
                        B.parts.num(6, i) = m;
                        B.parts.num(7, i) = 0;
                        if (m & 1) md_pair_force(sh, B, A, totals, i, 0, k);
                        if (m & 2) md_pair_force(sh, B, A, totals, i, 1, k);
                    }
                } else {
                    const int nq = sh.nq[par];
                    for (int s = me; s < nq; s += threads) {
                        const int e = sh.q[par][s];
                        md_pair_force(sh, B, A, totals, e >> 1, e & 1, k);
                    }
                }
                // the particles that the shared memory does not hold
                const int beyond = min(B.na, B.parts.cap + B.far.cap);
                for (int i = B.parts.cap + me; i < beyond; i += threads) {
                    const int s = i - B.parts.cap;
                    int m = B.far.num(0, s);
                    if (sh.anew) {
                        const R p[3] = {B.far.real(0, s), B.far.real(1, s), B.far.real(2, s)};
                        B.far.num(0, s) = m = md_busy(X, B, p, B.far.num(1, s), B.queue_sq);
                    }
                    if (!m) continue;
                    const R p[3] = {B.far.real(0, s), B.far.real(1, s), B.far.real(2, s)};
                    R nf[3];
                    B.far.num(1, s) = md_forces(sh, B, A, totals, i, k, p, B.far.num(2, s), B.far.num(1, s), nf);
                    for (int c = 0; c < 3; c++) B.far.real(12 + c, s) = nf[c];
                }
                // (those in place: the forces wait in force_old, whose entry is written
                // again below)
                for (int i = beyond + me; i < B.na; i += threads) {
                    const int idx = A.act[B.off + i];
                    const Part<R> q = md_read_in_place(B, A, idx);
                    if (!md_busy(X, B, q.p, q.f, B.reach_sq)) continue;
                    R nf[3];
                    md_view(A, B).flags[idx] = md_forces(sh, B, A, totals, i, k, q.p, q.sp, q.f, nf);
                    for (int c = 0; c < 3; c++) md_view(A, B).force_old[c][idx] = nf[c];
                }
                md_arrive(kBarForces, all);
                md_sync(kBarPart, threads);  // the forces are written
                // every particle's end of step k and beginning of step k + 1
                auto advance = [&](int i, auto tier_of, Part<R> q, int busy) {
                    constexpr int T = decltype(tier_of)::value;
                    const int s = i - B.parts.cap;  // in far
                    const bool past = (q.f >> PAST_MD_BIT) & 1;
                    const R gl[3] = {past ? q.g[0] : (R)0, past ? q.g[1] : (R)0, past ? q.g[2] : (R)0};
                    auto idx = [&] {
                        if constexpr (T == kShared) return B.parts.num(0, i);
                        else return A.act[B.off + i];
                    };
                    if (busy) {
                        R nf[3] = {0, 0, 0};
                        if constexpr (T == kShared) {
                            const int came = B.parts.num(7, i), m = B.parts.num(3, i);
#pragma unroll
                            for (int h = 0; h < 2; h++)
                                if ((came >> h) & 1) {
                                    q.f |= (1 << MD_BIT) | (B.cs[h] == 1 ? (1 << CATALYZED_BIT) : 0);
                                    for (int u = 0; u < (h ? m >> 16 : m & 0xffff); u++)
                                        for (int c = 0; c < 3; c++) nf[c] = nf[c] - B.parts.real(12 + 3 * h + c, i);
                                }
                            if (came & 4) q.f |= 1 << REAC_BIT;
                        } else if constexpr (T == kFar) {
                            for (int c = 0; c < 3; c++) nf[c] = B.far.real(12 + c, s);
                        } else {
                            for (int c = 0; c < 3; c++) nf[c] = md_view(A, B).force_old[c][idx()];
                        }
                        md_end(q, X, B, A, nf, idx(), step0 + (uint64_t)k);
                        if (T == kInPlace && !last)
                            for (int c = 0; c < 3; c++) md_view(A, B).force_old[c][idx()] = 0;
                    } else {
                        for (int c = 0; c < 3; c++) q.v[c] = md_vel_free(q.v[c], A.dt_r);
                    }
                    if (last) {
                        // the interval's last step leaves force_old behind
                        for (int c = 0; c < 3; c++) md_view(A, B).force_old[c][idx()] = gl[c];
                    } else {
                        if (md_begin(q, A.dt_r, A.dt_sq_r, A.read_species, thr, near_sq)) sh.over[1 - par] = 1;
                        if constexpr (T != kInPlace) {
                            const int m = md_busy(X, B, q.p, q.f, B.queue_sq);
                            if constexpr (T == kFar) {
                                B.far.num(0, s) = m;
                            } else {
                                B.parts.num(6, i) = m;
                                B.parts.num(7, i) = 0;
                                if (m & 3) {
                                    const int at = atomicAdd(&sh.nq[1 - par], (m & 1) + (m >> 1 & 1));
                                    const int e = 2 * i + (m & 1 ? 0 : 1);
                                    if (at < kMdQueue) sh.q[1 - par][at] = e;
                                    if ((m & 3) == 3 && at + 1 < kMdQueue) sh.q[1 - par][at + 1] = 2 * i + 1;
                                }
                            }
                        }
                    }
                    md_write<T>(B, A, i, q);
                };
                for (int i = me; i < shared; i += threads)
                    advance(i, std::integral_constant<int, kShared>(), md_read<kShared>(B, A, i), B.parts.num(6, i));
                for (int i = B.parts.cap + me; i < beyond; i += threads)
                    advance(i, std::integral_constant<int, kFar>(), md_read<kFar>(B, A, i), B.far.num(0, i - B.parts.cap));
                for (int i = beyond + me; i < B.na; i += threads) {
                    const Part<R> q = md_read<kInPlace>(B, A, i);
                    // (forces only add flags, so the test gives what it gave)
                    advance(i, std::integral_constant<int, kInPlace>(), q, md_busy(X, B, q.p, q.f, B.reach_sq));
                }
                md_sync(kBarTurn, all);
                k++;
                if (last) break;
            }
            for (int i = me; i < min(B.na, B.parts.cap); i += threads)
                md_write_in_place(B, A, B.parts.num(0, i), md_read<kShared>(B, A, i));
            for (int i = B.parts.cap + me; i < min(B.na, B.parts.cap + B.far.cap); i += threads)
                md_write_in_place(B, A, A.act[B.off + i], md_read<kFar>(B, A, i));
        }
        __syncthreads();
    }
    // the last replica to finish lists the tiles of those to re-sort and sets
    // the graph's loop condition
    if (t == 0) {
        __threadfence();
        sh.last = atomicAdd(A.done, 1u) == (unsigned)A.R_ - 1u;
    }
    __syncthreads();
    if (!sh.last) return;
    __threadfence();
    int any = 0, base_p = 0, base_s = 0;
    for (int r0 = 0; r0 < A.R_; r0 += all) {
        const int q = r0 + t;
        const int nd = q < A.R_ ? __ldcg(A.resort + q) : 0;
        any |= nd;
        const int np = nd ? A.rl.pcount[q] : 0, ns = nd ? A.rl.scount[q] : 0;
        int tp, ts;
        const int ep = base_p + block_excl_scan(np, sh.ws, &tp);
        const int es = base_s + block_excl_scan(ns, sh.ws, &ts);
        for (int c = 0; c < np; c++) A.rl.pids[ep + c] = A.rl.pfirst[q] + c;
        for (int c = 0; c < ns; c++) A.rl.sids[es + c] = A.rl.sfirst[q] + c;
        base_p += tp;
        base_s += ts;
    }
    any = __syncthreads_or(any);
    if (t == 0) {
        A.rl.n[0] = base_p;
        A.rl.n[1] = base_s;
        *A.any = any;
        *A.done = 0;
        if (A.use_cond) cudaGraphSetConditional(A.cond, any ? 1u : 0u);
        __threadfence();
    }
}

// ------------------------------------------------------ re-sort / sort

// count = 0, is_md = 0, is_reac = 1 over the active replicas' slots; for the
// interval's sort, block 0 also draws every replica's grid shift (random_shift, src/cell_system.f90:153-163)
__global__ void kb_zero_slots(TileSet ts, int *count, unsigned char *is_md,
                              unsigned char *is_reac, int R, BRep *rep, const uint64_t *d_step,
                              int shift_step_off)
{
    if (blockIdx.x == 0 && shift_step_off >= 0) {
        const uint64_t step = *d_step + (uint64_t)shift_step_off;
        for (int r = threadIdx.x; r < R; r += blockDim.x) {
            double u0, u1, u2, u3;
            rng::uniform2(rep[r].seed, step, 0, rng::SHIFT, 0, u0, u1);
            rng::uniform2(rep[r].seed, step, 1, rng::SHIFT, 0, u2, u3);
            rep[r].g.origin[0] = u0 - 1;
            rep[r].g.origin[1] = u1 - 1;
            rep[r].g.origin[2] = u2 - 1;
        }
    }
    for (int k = blockIdx.x; k < *ts.n; k += gridDim.x) {
        const BTile t = ts.tiles[ts.ids[k]];
        for (long long s = t.begin + threadIdx.x; s < t.end; s += blockDim.x) {
            count[s] = 0;
            is_md[s] = 0;
            is_reac[s] = 1;
        }
    }
}

// The pending md_pos steps of the free particles (adv - base of the replica,
// added one by one: each step's rounding is kept), the end of their md_vel
// steps, apply_pbc (src/md.f90:202-217), then key = replica's first slot + the
// particle's slot, histogram with one atomic per distinct key per warp.  Ends
// the active particles' places (aidx).
template <typename R>
__global__ void __launch_bounds__(kBT)
    kb_advance_key_count(TileSet ts, const BRep *rep, PView<R> v0, PView<R> v1, int *aidx, const int *adv,
                         const int *base, R dt, int *key, int *count)
{
    const int lane = threadIdx.x & 31;
    for (int kt = blockIdx.x; kt < *ts.n; kt += gridDim.x) {
        const BTile t = ts.tiles[ts.ids[kt]];
        const BRep &rp = rep[t.r];
        const Grid g = rp.g;
        const PView<R> v = pick(v0, v1, rp.cur);
        const int steps = adv[t.r] - base[t.r];
        constexpr int K = 2;  // particles per thread and pass, loaded before any is moved
        for (long long b = t.begin; b < t.end; b += K * kBT) {
            R x[K], y[K], z[K], vx[K], vy[K], vz[K];
            int act[K];
#pragma unroll
            for (int c = 0; c < K; c++) {
                const long long i = b + c * kBT + threadIdx.x;
                if (i < t.end) {
                    x[c] = v.pos.x[i];
                    y[c] = v.pos.y[i];
                    z[c] = v.pos.z[i];
                    vx[c] = v.vel.x[i];
                    vy[c] = v.vel.y[i];
                    vz[c] = v.vel.z[i];
                    act[c] = aidx[i];
                }
            }
#pragma unroll
            for (int c = 0; c < K; c++) {
                const long long i = b + c * kBT + threadIdx.x;
                const bool ok = i < t.end;
                int k = -1;
                if (ok) {
                    bool moved = false;
                    if (act[c] < 0) {
                        const R hx = dt * vx[c], hy = dt * vy[c], hz = dt * vz[c];
#pragma unroll 4
                        for (int j = 0; j < steps; j++) {
                            x[c] = x[c] + hx;
                            y[c] = y[c] + hy;
                            z[c] = z[c] + hz;
                        }
                        // md_pos adds the zero force term too: -0 becomes +0
                        moved = steps > 0;
                        x[c] = moved ? x[c] + (R)0 : x[c];
                        y[c] = moved ? y[c] + (R)0 : y[c];
                        z[c] = moved ? z[c] + (R)0 : z[c];
                        const R nx = md_vel_free(vx[c], dt), ny = md_vel_free(vy[c], dt), nz = md_vel_free(vz[c], dt);
                        if (!same_bits(nx, vx[c]) || !same_bits(ny, vy[c]) || !same_bits(nz, vz[c])) {
                            v.vel.x[i] = nx;
                            v.vel.y[i] = ny;
                            v.vel.z[i] = nz;
                        }
                    } else {
                        aidx[i] = -1;
                    }
                    const int jx = floor_div_edge((double)x[c], g.edges[0]), jy = floor_div_edge((double)y[c], g.edges[1]),
                              jz = floor_div_edge((double)z[c], g.edges[2]);
                    if (jx) {
                        v.ix[i] += jx;
                        x[c] = x[c] - (R)(jx * g.edges[0]);
                    }
                    if (jy) {
                        v.iy[i] += jy;
                        y[c] = y[c] - (R)(jy * g.edges[1]);
                    }
                    if (jz) {
                        v.iz[i] += jz;
                        z[c] = z[c] - (R)(jz * g.edges[2]);
                    }
                    if (moved || jx || jy || jz) {
                        v.pos.x[i] = x[c];
                        v.pos.y[i] = y[c];
                        v.pos.z[i] = z[c];
                    }
                    k = rp.soff + slot_of(g, (double)x[c], (double)y[c], (double)z[c]);
                    key[i] = k;
                }
                unsigned peers = __match_any_sync(0xffffffffu, k);
                if (ok && lane == __ffs(peers) - 1) atomicAdd(count + k, __popc(peers));
            }
        }
    }
}

__device__ inline long long block_sum_ll(long long v)
{
    __shared__ long long ws[kBT / 32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
    __syncthreads();
    long long s = 0;
    if (threadIdx.x == 0)
        for (int w = 0; w < kBT / 32; w++) s += ws[w];
    return s;
}

__global__ void __launch_bounds__(kBT) kb_scan_reduce(TileSet ts, const int *count, long long *tile_sum)
{
    for (int k = blockIdx.x; k < *ts.n; k += gridDim.x) {
        const int id = ts.ids[k];
        const BTile t = ts.tiles[id];
        long long a = 0;
        for (long long s = t.begin + threadIdx.x; s < t.end; s += blockDim.x) a += count[s];
        long long tot = block_sum_ll(a);
        if (threadIdx.x == 0) tile_sum[id] = tot;
        __syncthreads();
    }
}

// Per replica of the sort (one block): the tile offsets (its first particle +
// the sums of its earlier tiles); the colloids' apply_pbc and pos_old = pos;
// the buffers change places (the gather writes the other one); the lists of
// active particles start anew and the pending md_pos steps are done.
__global__ void __launch_bounds__(kBT)
    kb_scan_reps(const int *flag, BRep *rep, const int *first, const int *ntiles, const long long *tile_sum,
                 long long *tile_off, PView<double> c, Vec3<double> cold, int *adv, int *base, int *nl, int *nx,
                 int *nf, int *s_free, int *fresh)
{
    __shared__ int ws[33];
    const int r = blockIdx.x;
    if (flag && !flag[r]) return;
    long long acc = rep[r].off;
    const int f0 = first[r], nt = ntiles[r];
    for (int k0 = 0; k0 < nt; k0 += kBT) {
        const int k = k0 + threadIdx.x;
        int tot;
        const int ex = block_excl_scan(k < nt ? (int)tile_sum[f0 + k] : 0, ws, &tot);
        if (k < nt) tile_off[f0 + k] = acc + ex;
        acc += tot;
    }
    if (threadIdx.x < 2) {
        const int k = 2 * r + threadIdx.x;
        const double *e = rep[r].g.edges;
        apply_pbc_one(c, k, e[0], e[1], e[2]);
        cold.x[k] = c.pos.x[k];
        cold.y[k] = c.pos.y[k];
        cold.z[k] = c.pos.z[k];
    }
    if (threadIdx.x == 32) {
        rep[r].cur ^= 1;
        if (!flag) adv[r] = 0;  // the interval's sort
        base[r] = adv[r];
        nl[r] = nx[r] = nf[r] = 0;
        s_free[r] = INT_MAX;
        fresh[r] = 0;
    }
}

// start = cursor = exclusive scan inside the tile + the tile's offset
__global__ void __launch_bounds__(kBT) kb_scan_apply(TileSet ts, const int *count, const long long *tile_off,
                                                     int *start, int *cursor)
{
    __shared__ long long ws[kBT / 32 + 1];
    constexpr int PER = kTile / kBT;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int kt = blockIdx.x; kt < *ts.n; kt += gridDim.x) {
        const int id = ts.ids[kt];
        const BTile t = ts.tiles[id];
        const long long b = t.begin + (long long)threadIdx.x * PER;
        int v[PER];
        long long sum = 0;
#pragma unroll
        for (int k = 0; k < PER; k++) {
            v[k] = b + k < t.end ? count[b + k] : 0;
            sum += v[k];
        }
        long long inc = sum;
        for (int o = 1; o < 32; o <<= 1) {
            long long y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        if (lane == 31) ws[w] = inc;
        __syncthreads();
        if (threadIdx.x == 0) {
            long long acc = 0;
            for (int k = 0; k < kBT / 32; k++) {
                long long y = ws[k];
                ws[k] = acc;
                acc += y;
            }
        }
        __syncthreads();
        long long run = tile_off[id] + ws[w] + inc - sum;
#pragma unroll
        for (int k = 0; k < PER; k++) {
            if (b + k < t.end) {
                start[b + k] = (int)run;
                cursor[b + k] = (int)run;
            }
            run += v[k];
        }
        __syncthreads();
    }
}

// place every particle inside its cell (in-cell order fixed by kb_order_gather)
__global__ void __launch_bounds__(kBT) kb_perm(TileSet ts, const int *key, int *cursor, int *perm)
{
    const int lane = threadIdx.x & 31;
    const unsigned lt = lanemask_lt();
    for (int kt = blockIdx.x; kt < *ts.n; kt += gridDim.x) {
        const BTile t = ts.tiles[ts.ids[kt]];
        for (long long base = t.begin; base < t.end; base += blockDim.x) {
            long long i = base + threadIdx.x;
            int k = i < t.end ? key[i] : -1;
            unsigned peers = __match_any_sync(0xffffffffu, k);
            int b = 0;
            if (k >= 0 && lane == __ffs(peers) - 1) b = atomicAdd(cursor + k, __popc(peers));
            b = __shfl_sync(0xffffffffu, b, __ffs(peers) - 1);
            if (k >= 0) perm[b + __popc(peers & lt)] = (int)i;
        }
    }
}

// Every field through perm into the replica's other buffer (current since
// kb_scan_reps), each cell's indices put in order on the way (order_tile).
// Only particles with MD or PAST_MD set have force entries: they are moved and
// zeroed behind, so the buffer that is not current holds none.  Flagged
// particles are listed in flist.
// kFull: tiles of kOrderSlots slots, at compile time (96^3 FP32: 263 us otherwise, 246 so)
template <typename R, bool kFull>
__global__ void __launch_bounds__(kOrderThreads, 4)
    kb_order_gather(TileSet ts, int slots, const BRep *rep, PView<R> v0, PView<R> v1, const int *count,
                    const int *start, int *perm, int *flist, int *nf)
{
    __shared__ OrderTile sh;
    // tiles per slot tile; all of them together are at most the slots (2e9)
    if (kFull) slots = kOrderSlots;
    const int per = (kTile + slots - 1) / slots, all = *ts.n * per;
    for (int kt = blockIdx.x; kt < all; kt += gridDim.x) {
        const BTile t = ts.tiles[ts.ids[kt / per]];
        const long long s0 = t.begin + kt % per * slots;
        if (s0 >= t.end) continue;
        const BRep &rp = rep[t.r];
        const PView<R> d = pick(v0, v1, rp.cur), s = pick(v1, v0, rp.cur);
        int a0, np;
        __syncthreads();  // the last tile's indices are read
        const int *src = order_tile(sh, (int)s0, (int)min(s0 + slots, t.end), count, start, perm, d.id, a0, np);
        for (int q = threadIdx.x; q < np; q += kOrderThreads) {
            const int i = src[q], j = a0 + q;
            R px = s.pos.x[i], py = s.pos.y[i], pz = s.pos.z[i];
            R vx = s.vel.x[i], vy = s.vel.y[i], vz = s.vel.z[i];
            int ix = s.ix[i], iy = s.iy[i], iz = s.iz[i];
            int id = s.id[i], sp = s.species[i], fl = s.flags[i];
            d.pos.x[j] = px;
            d.pos.y[j] = py;
            d.pos.z[j] = pz;
            d.vel.x[j] = vx;
            d.vel.y[j] = vy;
            d.vel.z[j] = vz;
            d.ix[j] = ix;
            d.iy[j] = iy;
            d.iz[j] = iz;
            d.id[j] = id;
            d.species[j] = sp;
            d.flags[j] = fl;
            if (fl & kActiveBits) {
                flist[rp.off + atomicAdd(nf + t.r, 1)] = j;
                if (fl & ((1 << MD_BIT) | (1 << PAST_MD_BIT))) {
                    for (int k = 0; k < 3; k++) {
                        d.force[k][j] = s.force[k][i];
                        d.force_old[k][j] = s.force_old[k][i];
                        s.force[k][i] = 0;
                        s.force_old[k][i] = 0;
                    }
                }
            }
        }
    }
}

// update_list (src/neighbor_list.f90:76-157), one block per colloid; the
// candidate cells of each stencil chunk are staged in nl_stage_bytes<R>() of
// dynamic shared memory by bulk copies (a window may reach into a
// neighbouring replica's particles, which are read and not used)
template <typename R>
__global__ void __launch_bounds__(kNlBlockThreads)
    kb_update_list(const int *flag, const BRep *rep, PView<double> c, PView<R> v0, PView<R> v1, const int *count,
                   const int *start,
                   const int *stencil, int n_stencil, double radiussq, LJDev lj, int Nmax, int *list, int *n,
                   unsigned char *is_md, unsigned char *is_reac, unsigned *err)
{
    extern __shared__ __align__(16) unsigned char nl_stage[];
    __shared__ __align__(8) unsigned long long bar;
    const int i = blockIdx.x, r = i >> 1;
    if (flag && !flag[r]) return;
    const BRep &rp = rep[r];
    const PView<R> s = pick(v0, v1, rp.cur);
    update_list_block<R>(i, rp.g, c.pos.x, c.pos.y, c.pos.z, c.species, s.pos.x, s.pos.y, s.pos.z, s.species,
                         count + rp.soff, start + rp.soff, stencil, n_stencil, radiussq, lj, 1, Nmax, list, n,
                         is_md + rp.soff, is_reac + rp.soff, err, NlStage{nl_stage, &bar});
}

// the kernels with dynamic shared memory above the default limit, set once
// per precision (at batch creation, before any stream capture)
template <typename R>
static int allow_shared()
{
    static bool set = false;
    if (!set) {
        RMPCD_CUDA_TRY(cudaFuncSetAttribute(kb_md<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)kMdSmem));
        RMPCD_CUDA_TRY(cudaFuncSetAttribute(kb_update_list<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)nl_stage_bytes<R>()));
        set = true;
    }
    return RMPCD_OK;
}

// ------------------------------------------------------------ interval

// simple_mpcd_step (src/mpcd.f90:71-183), one thread per slot, and refuel
// (programs/single_dimer_pbc.f90:544-565), one thread per particle: the
// collision writes velocities, refuel reads positions and species only
template <typename R>
__global__ void __launch_bounds__(kBT)
    kb_srd_refuel(const BTile *stiles, int n_stiles, const BTile *ptiles, const BRep *rep, const int *count,
                  const int *start, PView<R> v0, PView<R> v1, PView<double> c, SrdParams q, const uint64_t *d_step,
                  int step_off)
{
    if ((int)blockIdx.x < n_stiles) {
        const BTile t = stiles[blockIdx.x];
        const BRep &rp = rep[t.r];
        const PView<R> v = pick(v0, v1, rp.cur);
        q.seed = rp.seed;
        q.step = *d_step + (uint64_t)step_off;
        for (long long s = t.begin + threadIdx.x; s < t.end; s += blockDim.x)
            srd_slot<R>(count[s], start[s], s - rp.soff, rp.off, v.vel.x, v.vel.y, v.vel.z, v.species, q);
        return;
    }
    const BTile t = ptiles[blockIdx.x - n_stiles];
    const BRep &rp = rep[t.r];
    const PView<R> v = pick(v0, v1, rp.cur);
    const double a[3] = {c.pos.x[2 * t.r], c.pos.y[2 * t.r], c.pos.z[2 * t.r]};
    const double b[3] = {c.pos.x[2 * t.r + 1], c.pos.y[2 * t.r + 1], c.pos.z[2 * t.r + 1]};
    for (long long i = t.begin + threadIdx.x; i < t.end; i += blockDim.x)
        refuel_one(v, i, a, b, rp.g.edges[0], rp.g.edges[1], rp.g.edges[2], rp.far);
}

__global__ void kb_advance(uint64_t *d_step, uint64_t by)
{
    *d_step += by;
}

__global__ void k_add_offset(int *dst, const int *src, long long n, long long delta)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i] = (int)(src[i] + delta);
}

// list entries are particle indices for entries e < n(i) only
__global__ void k_list_offset(int *dst, const int *src, const int *n, int points, int Nmax, long long delta)
{
    long long tot = (long long)points * Nmax;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < tot; q += (long long)gridDim.x * blockDim.x) {
        int i = (int)(q / Nmax), e = (int)(q % Nmax);
        dst[q] = e < n[i] ? (int)(src[q] + delta) : -1;
    }
}

// ----------------------------------------------------------- host side

using Batch = rmpcd_dimer_batch;

static int grid_cap(long long n, int bs)
{
    long long g = (n + bs - 1) / bs;
    if (g < 1) g = 1;
    if (g > 65535) g = 65535;
    return (int)g;
}

// grid of the re-sort kernels, which loop over their tile list
static int resort_grid(int n_tiles)
{
    int g = sm_count() * 8;
    return n_tiles < g ? (n_tiles > 0 ? n_tiles : 1) : g;
}

// the re-sort of the flagged replicas (flag = resort flags, lists = their
// tiles) or of every replica (flag = null, lists = all tiles), then the active
// particles of what was sorted
template <typename R>
static TileSet particle_tiles(const Batch *b, const int *flag)
{
    return TileSet{b->ptile, flag ? b->act_p : b->all_p, flag ? b->n_act : b->n_all};
}

template <typename R>
static void resort_launches(Batch *b, const int *flag, cudaStream_t st, int shift_step_off)
{
    const PView<R> v0 = phys<R>(b->sol, 0), v1 = phys<R>(b->sol, 1);
    const PView<double> cv = phys<double>(b->col, 0);
    const TileSet pts = particle_tiles<R>(b, flag);
    const TileSet sts{b->stile, flag ? b->act_s : b->all_s, (flag ? b->n_act : b->n_all) + 1};
    const int gp = resort_grid(b->n_ptile), gs = resort_grid(b->n_stile);
    const R dt = (R)(b->prm.tau / b->prm.N_MD);
    kb_zero_slots<<<gs, kBT, 0, st>>>(sts, b->count, b->is_md, b->is_reac, b->R, b->rep, b->d_step,
                                      shift_step_off);
    kb_advance_key_count<R><<<gp, kBT, 0, st>>>(pts, b->rep, v0, v1, b->aidx, b->adv, b->base, dt, b->sol->key,
                                                b->count);
    kb_scan_reduce<<<gs, kBT, 0, st>>>(sts, b->count, b->tile_sum);
    kb_scan_reps<<<b->R, kBT, 0, st>>>(flag, b->rep, b->stile_first, b->stile_count, b->tile_sum, b->tile_off, cv,
                                       phys<double>(b->col, 1).pos, b->adv, b->base, b->nl, b->nx, b->nf, b->s_free,
                                       b->fresh);
    kb_scan_apply<<<gs, kBT, 0, st>>>(sts, b->count, b->tile_off, b->start, b->cursor);
    kb_perm<<<gp, kBT, 0, st>>>(pts, b->sol->key, b->cursor, b->sol->perm);
    auto *order = b->order_slots == kOrderSlots ? kb_order_gather<R, true> : kb_order_gather<R, false>;
    order<<<resort_grid(b->n_stile * ((kTile + b->order_slots - 1) / b->order_slots)), kOrderThreads, 0, st>>>(
        sts, b->order_slots, b->rep, v0, v1, b->count, b->start, b->sol->perm, b->sol->key, b->nf);
    kb_update_list<R><<<2 * b->R, kNlBlockThreads, nl_stage_bytes<R>(), st>>>(
        flag, b->rep, cv, v0, v1, b->count, b->start, b->stencil, b->n_stencil,
        b->prm.list_radius * b->prm.list_radius, b->lj_sc, b->Nmax, b->list, b->nn, b->is_md, b->is_reac,
        dev_error_word());
}

static void note(Batch *b, cudaError_t e)
{
    if (e != cudaSuccess && b->cap_err == cudaSuccess) b->cap_err = e;
}

// blocks per colloid of the list kernels: ceil(capacity / (256 x the
// shape's list entries per thread)), at most 64
static int list_gx(const Batch *b)
{
    const int per = 256 * kListPer[shape_list(b->shape)];
    const int gx = (b->Nmax + per - 1) / per;
    return gx > 64 ? 64 : gx < 1 ? 1 : gx;
}

// the active particles of the replicas in flag (every one when null), then
// their MD steps up to the next re-sort or the interval's end
template <typename R>
static void md_launches(Batch *b, const int *flag, cudaStream_t st, cudaGraphConditionalHandle cond)
{
    const PView<R> v0 = phys<R>(b->sol, 0), v1 = phys<R>(b->sol, 1);
    const double dt = b->prm.tau / b->prm.N_MD;
    const int gx = list_gx(b), gp = resort_grid(b->n_ptile);
    double cut_sq = b->prm.cut_sq_C;
    for (double c : b->lj_sc.cut_sq) cut_sq = c > cut_sq ? c : cut_sq;
    const float reach = (float)sqrt(cut_sq) * 1.0001f + 1e-3f;
    kb_claim<R><<<dim3(gx, 2 * b->R), kBT, 0, st>>>(flag, b->rep, v0, v1, phys<double>(b->col, 1).pos, (R)dt, reach,
                                                    (float)(b->prm.skin * 0.1) * 1.0001f, b->prm.N_MD, b->base, b->list,
                                                    b->nn, b->Nmax, b->aidx, b->act, b->nl, b->mult, b->ent);
    kb_classify<R><<<gp + gx * 2 * b->R + b->R, kBT, 0, st>>>(
        particle_tiles<R>(b, flag), gp, gx, b->R, flag, b->rep, v0, v1, (R)dt, b->prm.skin * 0.89, b->prm.N_MD,
        b->read_species ? 1 : 0, b->base, b->fresh, b->s_free, b->list, b->nn, b->Nmax, b->aidx, b->act, b->nl, b->nx,
        b->mult, b->ent, b->next, b->sol->key, b->nf);
    MdArgs<R> a;
    a.rep = b->rep;
    a.v0 = v0;
    a.v1 = v1;
    a.c = phys<double>(b->col, 0);
    a.cold = phys<double>(b->col, 1).pos;
    for (int k = 0; k < 3; k++) a.rat[k] = b->rattle[k];
    a.mass = b->vv_mass;
    a.ms = b->ms;
    a.bond = b->prm.bond;
    a.dt = dt;
    a.skin = b->prm.skin;
    a.dt_r = (R)dt;
    a.dt_sq_r = (R)(dt * dt / 2);
    a.cut_c = b->prm.cut_sq_C;
    a.cut_n = b->prm.cut_sq_N;
    a.prob = b->prm.prob;
    a.lj_sc = b->lj_sc;
    a.lj_cc = b->lj_cc;
    a.R_ = b->R;
    a.N_MD = b->prm.N_MD;
    a.Nmax = b->Nmax;
    a.start = flag ? 0 : 1;
    a.read_species = b->read_species ? 1 : 0;
    a.d_step = b->d_step;
    a.n = b->nn;
    a.next = b->next;
    a.ent = b->ent;
    a.act = b->act;
    a.nl = b->nl;
    a.nx = b->nx;
    a.mult = b->mult;
    a.over = b->over;
    a.terms = b->terms;
    a.keys[0] = b->keys[0];
    a.keys[1] = b->keys[1];
    a.n_over = b->n_over;
    a.far = b->far;
    a.far_cap = b->far_cap;
    a.reach = reach;
    a.s_free = b->s_free;
    a.fresh = b->fresh;
    a.adv = b->adv;
    a.resort = b->resort;
    a.n_extra = b->n_extra;
    a.rl = ResortLists{b->ptile_first, b->ptile_count, b->stile_first, b->stile_count, b->act_p, b->act_s, b->n_act};
    a.done = b->done;
    a.any = b->any;
    a.cond = cond;
    a.use_cond = b->capturing ? 1 : 0;
    a.err = dev_error_word();
    kb_md<R><<<b->R, kMdSum + kPartThreads[shape_var(b->shape)], kMdSmem, st>>>(a);
    note(b, cudaGetLastError());
}

// an interval's MD steps in the graph being captured on st: the steps up to
// every replica's first re-sort, then a WHILE node whose body re-sorts the
// replicas that wait for it and continues them
template <typename R>
static void capture_md(Batch *b, cudaStream_t st)
{
    cudaStreamCaptureStatus cs;
    cudaGraph_t g = nullptr;
    note(b, cudaStreamGetCaptureInfo(st, &cs, nullptr, &g, nullptr, nullptr));
    cudaGraphConditionalHandle cond = 0;
    note(b, cudaGraphConditionalHandleCreate(&cond, g, 0, cudaGraphCondAssignDefault));
    md_launches<R>(b, nullptr, st, cond);
    const cudaGraphNode_t *deps = nullptr;
    size_t nd = 0;
    note(b, cudaStreamGetCaptureInfo(st, &cs, nullptr, nullptr, &deps, &nd));
    cudaGraphNodeParams cp{};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = cond;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t node = nullptr;
    note(b, cudaGraphAddNode(&node, g, deps, nd, &cp));
    if (b->cap_err != cudaSuccess) return;
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    note(b, cudaStreamUpdateCaptureDependencies(st, &node, 1, cudaStreamSetCaptureDependencies));
    note(b, cudaStreamBeginCaptureToGraph(b->body, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    resort_launches<R>(b, b->resort, b->body, -1);
    md_launches<R>(b, b->resort, b->body, cond);
    cudaGraph_t out = nullptr;
    note(b, cudaStreamEndCapture(b->body, &out));
}

template <typename R>
static int interval_launches(Batch *b)
{
    cudaStream_t st = stream();
    const int N_MD = b->prm.N_MD;
    if (b->capturing) {
        capture_md<R>(b, st);
    } else {
        md_launches<R>(b, nullptr, st, 0);
        for (;;) {
            int any = 0;
            if (b->cap_err != cudaSuccess)
                return fail(RMPCD_ERR_CUDA, "dimer batch: %s", cudaGetErrorString(b->cap_err));
            RMPCD_CUDA_TRY(cudaMemcpyAsync(&any, b->any, sizeof(int), cudaMemcpyDeviceToHost, st));
            RMPCD_CUDA_TRY(cudaStreamSynchronize(st));
            if (!any) break;
            resort_launches<R>(b, b->resort, st, -1);
            md_launches<R>(b, b->resort, st, 0);
        }
    }
    resort_launches<R>(b, nullptr, st, N_MD);
    SrdParams q{};
    q.sin_a = 1;
    q.cos_a = 0;
    q.thermostat = b->prm.thermostat ? 1 : 0;
    q.hydro = b->prm.hydro ? 1 : 0;
    q.t_factor = b->prm.thermostat ? sqrt(b->prm.T) : 0.0;
    kb_srd_refuel<R><<<b->n_stile + b->n_ptile, kBT, 0, st>>>(b->stile, b->n_stile, b->ptile, b->rep, b->count,
                                                              b->start, phys<R>(b->sol, 0), phys<R>(b->sol, 1),
                                                              phys<double>(b->col, 0), q, b->d_step, N_MD + 1);
    kb_advance<<<1, 1, 0, st>>>(b->d_step, (uint64_t)N_MD + 2);
    return RMPCD_OK;
}

template <typename R>
static int run_t(Batch *b, int n_intervals)
{
    cudaStream_t st = stream();
    for (int it = 0; it < n_intervals; it++) {
        PhaseTimer t("batch_interval");
        b->ran = true;
        if (!b->use_graph) {
            b->cap_err = cudaSuccess;
            int rc = interval_launches<R>(b);
            if (rc) return rc;
            RMPCD_CHECK_LAUNCH();
        } else {
            if (!b->exec) {
                cudaGraph_t g = nullptr;
                b->cap_err = cudaSuccess;
                RMPCD_CUDA_TRY(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
                b->capturing = true;
                interval_launches<R>(b);
                b->capturing = false;
                cudaError_t e = cudaStreamEndCapture(st, &g);
                if (e == cudaSuccess && b->cap_err != cudaSuccess) e = b->cap_err;
                if (e == cudaSuccess) e = cudaGraphInstantiate(&b->exec, g, 0);
                if (g) cudaGraphDestroy(g);
                if (e != cudaSuccess) {
                    b->exec = nullptr;
                    cudaGetLastError();
                    return fail(RMPCD_ERR_CUDA, "interval graph: %s", cudaGetErrorString(e));
                }
            }
            RMPCD_CUDA_TRY(cudaGraphLaunch(b->exec, st));
        }
        b->step += (uint64_t)b->prm.N_MD + 2;
    }
    return check_dev_error(nullptr);
}

static void free_batch(Batch *b)
{
    if (!b) return;
    cudaStreamSynchronize(stream());
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->body) cudaStreamDestroy(b->body);
    rmpcd_particles_destroy(b->sol);
    rmpcd_particles_destroy(b->col);
    void *ptrs[] = {b->rep, b->ptile, b->stile, b->stile_first, b->stile_count, b->tile_sum, b->tile_off, b->count,
                    b->start, b->cursor, b->is_md, b->is_reac, b->stencil, b->list, b->nn, b->act, b->nl, b->nx,
                    b->aidx, b->next, b->mult, b->ent, b->over, b->terms, b->keys[0], b->keys[1], b->n_over, b->far, b->nf, b->s_free, b->adv, b->base, b->fresh, b->resort,
                    b->n_extra, b->rattle[0], b->rattle[1], b->rattle[2], b->vv_mass, b->d_step,
                    b->done, b->ptile_first, b->ptile_count, b->act_p, b->act_s, b->n_act, b->all_p, b->all_s,
                    b->n_all, b->any};
    for (void *q : ptrs) cudaFree(q);
    for (int *l : b->luts) cudaFree(l);
    delete b;
}

template <typename T>
static int dalloc(T **p, size_t n)
{
    RMPCD_CUDA_TRY(cudaMalloc((void **)p, (n > 0 ? n : 1) * sizeof(T)));
    return RMPCD_OK;
}

// Copies between device arrays that do not overlap, many in one launch: moving
// a replica in or out is some 50 arrays, most of them short, and as single
// copies their launches took four times as long as the bytes (48 replicas of
// 16^3 to 48^3 FP32, four intervals with the copies out: 48.3 ms; one launch per
// replica: 41.0 ms).
constexpr int kCopyMax = 64;
struct CopyList {
    const unsigned char *src[kCopyMax];
    unsigned char *dst[kCopyMax];
    unsigned long long bytes[kCopyMax];
};

template <typename T>
__device__ inline void copy_as(unsigned char *d, const unsigned char *s, unsigned long long bytes)
{
    const long long n = (long long)(bytes / sizeof(T)), step = (long long)gridDim.x * blockDim.x;
    constexpr int U = 4;  // loads in flight
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += U * step) {
        T v[U];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i + u * step < n) v[u] = ((const T *)s)[i + u * step];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i + u * step < n) ((T *)d)[i + u * step] = v[u];
    }
}

// blockIdx.y: the copy
__global__ void __launch_bounds__(256) k_copy_list(const __grid_constant__ CopyList l)
{
    const unsigned char *s = l.src[blockIdx.y];
    unsigned char *d = l.dst[blockIdx.y];
    const unsigned long long n = l.bytes[blockIdx.y];
    const unsigned low = (unsigned)((uintptr_t)s | (uintptr_t)d | n) & 15u;
    if (low == 0) copy_as<int4>(d, s, n);
    else if ((low & 3u) == 0) copy_as<int>(d, s, n);
    else copy_as<unsigned char>(d, s, n);
}

class Copies {
public:
    int add(void *dst, const void *src, size_t bytes)
    {
        if (!bytes) return RMPCD_OK;
        l_.src[n_] = (const unsigned char *)src;
        l_.dst[n_] = (unsigned char *)dst;
        l_.bytes[n_] = bytes;
        most_ = bytes > most_ ? bytes : most_;
        return ++n_ == kCopyMax ? flush() : RMPCD_OK;
    }
    int flush()
    {
        if (n_ == 0) return RMPCD_OK;
        const dim3 grid(grid_cap((long long)(most_ / 64), 256), n_);
        n_ = 0;
        most_ = 0;
        k_copy_list<<<grid, 256, 0, stream()>>>(l_);
        RMPCD_CHECK_LAUNCH();
        return RMPCD_OK;
    }

private:
    CopyList l_;
    int n_ = 0;
    size_t most_ = 0;
};

// *out = 1 if some a[i] < 0
__global__ void k_any_negative(const int *a, long long n, int *out)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        if (a[i] < 0) {
            *out = 1;
            return;
        }
}

// the particle tiles of every replica at `ptile` particles per tile: tile
// list, each replica's first tile and count, and the every-tile id list
static int build_particle_tiles(Batch *b, long long ptile)
{
    std::vector<BTile> pt;
    std::vector<int> pfirst(b->R), pcount(b->R);
    for (int r = 0; r < b->R; r++) {
        const BRep &p = b->rep_h[r];
        pfirst[r] = (int)pt.size();
        for (long long t = 0; t < p.n; t += ptile)
            pt.push_back({r, 0, p.off + t, p.off + (t + ptile < p.n ? t + ptile : p.n)});
        pcount[r] = (int)pt.size() - pfirst[r];
    }
    if ((long long)pt.size() > b->cap_ptile)
        return fail(RMPCD_ERR_CAPACITY, "dimer batch: %zu particle tiles above the %d allocated", pt.size(),
                    b->cap_ptile);
    cudaStream_t st = stream();
    std::vector<int> ids(pt.size());
    for (size_t k = 0; k < ids.size(); k++) ids[k] = (int)k;
    const int n = (int)pt.size();
    if (n) {
        RMPCD_CUDA_TRY(cudaMemcpyAsync(b->ptile, pt.data(), pt.size() * sizeof(BTile), cudaMemcpyHostToDevice, st));
        RMPCD_CUDA_TRY(cudaMemcpyAsync(b->all_p, ids.data(), ids.size() * sizeof(int), cudaMemcpyHostToDevice, st));
    }
    RMPCD_CUDA_TRY(cudaMemcpyAsync(b->ptile_first, pfirst.data(), b->R * sizeof(int), cudaMemcpyHostToDevice, st));
    RMPCD_CUDA_TRY(cudaMemcpyAsync(b->ptile_count, pcount.data(), b->R * sizeof(int), cudaMemcpyHostToDevice, st));
    RMPCD_CUDA_TRY(cudaMemcpyAsync(b->n_all, &n, sizeof(int), cudaMemcpyHostToDevice, st));
    // the host vectors go out of scope: wait for the copies that read them
    RMPCD_CUDA_TRY(cudaStreamSynchronize(st));
    b->n_ptile = n;
    return RMPCD_OK;
}

// copy one particle system's current arrays (and pos_old) to/from buffer bc of
// the batch system at offset off; pos_old is buffer bo's positions
static int move_particles(Copies &cp, rmpcd_particles *big, int bc, int bo, rmpcd_particles *p, long long off,
                          bool to_batch)
{
    const size_t rs = (size_t)big->rsize, n = (size_t)p->N;
    const int pc = p->cur;
    for (int k = 0; k < 3; k++) {
        struct {
            void *a, *b;
            size_t bytes;
        } m[] = {{(char *)big->pos[bc][k] + off * rs, p->pos[pc][k], n * rs},
                 {(char *)big->pos[bo][k] + off * rs, p->pos[1 - pc][k], n * rs},
                 {(char *)big->vel[bc][k] + off * rs, p->vel[pc][k], n * rs},
                 {(char *)big->force[bc][k] + off * rs, p->force[pc][k], n * rs},
                 {(char *)big->force_old[bc][k] + off * rs, p->force_old[pc][k], n * rs},
                 {big->image[bc][k] + off, p->image[pc][k], n * sizeof(int)}};
        for (auto &e : m) {
            int rc = to_batch ? cp.add(e.a, e.b, e.bytes) : cp.add(e.b, e.a, e.bytes);
            if (rc) return rc;
        }
    }
    int *bi[3] = {big->id[bc] + off, big->species[bc] + off, big->flags[bc] + off};
    int *pi[3] = {p->id[pc], p->species[pc], p->flags[pc]};
    for (int k = 0; k < 3; k++) {
        int rc = to_batch ? cp.add(bi[k], pi[k], n * sizeof(int)) : cp.add(pi[k], bi[k], n * sizeof(int));
        if (rc) return rc;
    }
    if (!to_batch) {
        p->force_zero = false;
        p->force_old_zero = false;
    }
    return RMPCD_OK;
}

static int check_inputs(int R, rmpcd_particles *const *sol, rmpcd_particles *const *col, rmpcd_cells *const *cells,
                        rmpcd_nlist *const *nl, const rmpcd_rng *rngs, const rmpcd_dimer_params *prm)
{
    RMPCD_ARG(R >= 1, "dimer batch: n_replicas must be >= 1");
    RMPCD_ARG(sol && col && cells && nl && rngs && prm, "null argument");
    RMPCD_ARG(prm->N_MD >= 1 && prm->tau > 0, "dimer batch: N_MD >= 1 and tau > 0 required");
    for (int r = 0; r < R; r++) {
        if (!(sol[r] && col[r] && cells[r] && nl[r]))
            return fail(RMPCD_ERR_INVALID, "dimer batch: null handle for replica %d", r);
        RMPCD_ARG(sol[r]->precision == sol[0]->precision, "dimer batch: replicas mix solvent precisions");
        if (sol[r]->N < 1) return fail(RMPCD_ERR_INVALID, "dimer batch: replica %d has no solvent", r);
        RMPCD_ARG(col[r]->N == 2 && col[r]->precision == RMPCD_FP64, "dimer batch: colloids must be 2 FP64 beads");
        RMPCD_ARG(col[r]->n_species == col[0]->n_species &&
                      memcmp(col[r]->mass, col[0]->mass, sizeof(col[0]->mass)) == 0,
                  "dimer batch: replicas differ in colloid masses");
        RMPCD_ARG(!cells[r]->has_walls, "dimer batch: periodic boxes only");
        RMPCD_ARG(nl[r]->Npoints == 2 && nl[r]->Nmax == nl[0]->Nmax && nl[r]->stencil,
                  "dimer batch: neighbor lists must have 2 points, one capacity and a stencil");
        RMPCD_ARG(nl[r]->n_stencil == nl[0]->n_stencil, "dimer batch: replicas differ in list stencil");
        RMPCD_ARG(rngs[r].step == rngs[0].step, "dimer batch: replicas must start at the same RNG step");
    }
    return RMPCD_OK;
}

static int create(Batch **out, int R, rmpcd_particles *const *sol, rmpcd_particles *const *col,
                  rmpcd_cells *const *cells, rmpcd_nlist *const *nl, const rmpcd_rng *rngs, const rmpcd_lj *lj_sc,
                  const rmpcd_lj *lj_cc, const rmpcd_dimer_params *prm)
{
    int rc = check_inputs(R, sol, col, cells, nl, rngs, prm);
    if (rc) return rc;
    RMPCD_ARG(lj_sc && lj_cc, "null argument");
    Batch *b = new Batch();
    b->R = R;
    b->precision = sol[0]->precision;
    b->prm = *prm;
    b->step = rngs[0].step;
    b->Nmax = nl[0]->Nmax;
    b->n_stencil = nl[0]->n_stencil;
    b->lj_sc = lj_dev(lj_sc);
    b->lj_cc = lj_dev(lj_cc);
    b->ms.n = col[0]->n_species;
    for (int s = 0; s < RMPCD_MAX_SPECIES; s++) b->ms.m[s] = col[0]->mass[s];
    // replica layout and tiles
    // default shape: 512 threads for a replica's MD steps and the largest particle
    // tiles that give ~2 per SM: each tile's block is a chain of round trips, so
    // fewer, fuller tiles beat more blocks (ms per interval with tiles of 256,
    // 512, 1024, 2048, 4096: one 96^3 dimer FP32 3.3, 2.6, 2.3, 2.1, 2.1; 512
    // replicas FP32 43.8, 36.0, 32.2, 30.7, 30.1; one 32^3 dimer FP64 0.88, 0.88,
    // 0.87, 0.90, 0.92); rmpcd_dimer_batch_autotune times the others
    long long n_total = 0;
    for (int r = 0; r < R; r++) n_total += sol[r]->N;
    int tile_k = kNPTiles - 1;
    while (tile_k > 0 && n_total / kPTiles[tile_k] < 2LL * sm_count()) tile_k--;
    b->shape = tile_k;
    long long cap_p = 0;
    for (int r = 0; r < R; r++) cap_p += (sol[r]->N + kPTiles[0] - 1) / kPTiles[0];
    if (cap_p < 1) cap_p = 1;
    std::vector<BTile> stl;
    std::vector<int> sfirst(R), scount(R);
    std::map<std::vector<int>, int *> lut_of;
    b->rep_h.resize(R);
    long long off = 0;
    long long soff = 0;
    for (int r = 0; r < R; r++) {
        BRep &p = b->rep_h[r];
        rmpcd_cells *c = cells[r];
        p.off = off;
        p.n = sol[r]->N;
        p.soff = (int)soff;
        p.S = c->S;
        p.seed = rngs[r].seed;
        p.cur = 0;
        volatile float lf = (float)c->L[0] * 0.45f;
        volatile float ff = lf * lf;
        p.far = (double)ff;
        p.g = grid_of(c);
        std::vector<int> key = {c->L[0], c->L[1], c->L[2]};
        if (!lut_of.count(key)) {
            int *l = nullptr;
            if (dalloc(&l, (size_t)c->n_lut)) {
                free_batch(b);
                return RMPCD_ERR_CUDA;
            }
            b->luts.push_back(l);
            cudaMemcpyAsync(l, c->lut, (size_t)c->n_lut * sizeof(int), cudaMemcpyDeviceToDevice, stream());
            lut_of[key] = l;
        }
        p.g.lut = lut_of[key];
        sfirst[r] = (int)stl.size();
        for (long long t = 0; t < p.S; t += kTile) stl.push_back({r, 0, soff + t, soff + (t + kTile < p.S ? t + kTile : p.S)});
        scount[r] = (int)stl.size() - sfirst[r];
        off += p.n;
        soff += p.S;
    }
    if (off > 2000000000LL || soff > 2000000000LL) {
        free_batch(b);
        return fail(RMPCD_ERR_CAPACITY, "dimer batch: more than 2e9 particles or slots in total");
    }
    b->Ntot = off;
    b->Stot = (int)soff;
    b->cap_ptile = (int)cap_p;
    b->n_stile = (int)stl.size();
    double densest = 0;
    for (const BRep &p : b->rep_h) {
        const double mean = (double)p.n / ((double)p.g.L[0] * p.g.L[1] * p.g.L[2]);
        densest = mean > densest ? mean : densest;
    }
    b->order_slots = order_slots(densest);
    size_t ne = (size_t)2 * R * b->Nmax;
    // every particle that two full lists could make active; an even number, so that
    // each replica's part (132 B per particle in FP64) begins at a multiple of 8 B
    long long most = 0;
    for (const BRep &p : b->rep_h) most = p.n > most ? p.n : most;
    b->far_cap = (int)(((2LL * b->Nmax < most ? 2LL * b->Nmax : most) + 1) & ~1LL);
    bool ok = !dalloc(&b->rep, R) && !dalloc(&b->ptile, cap_p) && !dalloc(&b->stile, stl.size()) &&
              !dalloc(&b->stile_first, R) && !dalloc(&b->stile_count, R) && !dalloc(&b->tile_sum, stl.size()) &&
              !dalloc(&b->tile_off, stl.size()) && !dalloc(&b->count, soff) && !dalloc(&b->start, soff) &&
              !dalloc(&b->cursor, soff) && !dalloc(&b->is_md, soff) && !dalloc(&b->is_reac, soff) &&
              !dalloc(&b->stencil, 3 * (size_t)b->n_stencil) && !dalloc(&b->list, ne) && !dalloc(&b->nn, 2 * (size_t)R) &&
              !dalloc(&b->act, off) && !dalloc(&b->nl, R) && !dalloc(&b->nx, R) && !dalloc(&b->aidx, off) &&
              !dalloc(&b->next, ne) && !dalloc(&b->mult, ne) && !dalloc(&b->ent, 2 * ne) && !dalloc(&b->over, ne) &&
              !dalloc(&b->terms, ne) && !dalloc(&b->keys[0], ne) && !dalloc(&b->keys[1], ne) &&
              !dalloc(&b->n_over, 4 * (size_t)R) &&
              !dalloc(&b->far, (size_t)R * b->far_cap * (b->precision == RMPCD_FP32 ? md_far_bytes<float>() : md_far_bytes<double>())) &&
              !dalloc(&b->nf, R) && !dalloc(&b->s_free, R) && !dalloc(&b->adv, R) && !dalloc(&b->base, R) &&
              !dalloc(&b->fresh, R) && !dalloc(&b->resort, R) &&
              !dalloc(&b->n_extra, R) &&
              !dalloc(&b->rattle[0], 2 * (size_t)R) && !dalloc(&b->rattle[1], 2 * (size_t)R) &&
              !dalloc(&b->rattle[2], 2 * (size_t)R) && !dalloc(&b->vv_mass, 2 * (size_t)R) && !dalloc(&b->d_step, 1) &&
              !dalloc(&b->done, 1) && cudaStreamCreateWithFlags(&b->body, cudaStreamNonBlocking) == cudaSuccess &&
              !dalloc(&b->any, 1) &&
              !dalloc(&b->ptile_first, R) && !dalloc(&b->ptile_count, R) && !dalloc(&b->act_p, cap_p) &&
              !dalloc(&b->act_s, stl.size()) && !dalloc(&b->n_act, 2) && !dalloc(&b->all_p, cap_p) &&
              !dalloc(&b->all_s, stl.size()) && !dalloc(&b->n_all, 2);
    if (!ok) {
        free_batch(b);
        return RMPCD_ERR_CUDA;
    }
    if (rmpcd_particles_init(&b->sol, (int)off, sol[0]->n_species, sol[0]->mass, b->precision) ||
        rmpcd_particles_init(&b->col, 2 * R, col[0]->n_species, col[0]->mass, RMPCD_FP64)) {
        free_batch(b);
        return RMPCD_ERR_CUDA;
    }
    if ((b->precision == RMPCD_FP32 ? allow_shared<float>() : allow_shared<double>()) != RMPCD_OK) {
        free_batch(b);
        return RMPCD_ERR_CUDA;
    }
    cudaStream_t st = stream();
    std::vector<double> vm(2 * (size_t)R);
    for (int r = 0; r < R; r++) {
        vm[2 * r] = prm->vv_mass[0];
        vm[2 * r + 1] = prm->vv_mass[1];
    }
    RMPCD_CUDA_TRY(cudaMemcpyAsync(b->rep, b->rep_h.data(), R * sizeof(BRep), cudaMemcpyHostToDevice, st));
    RMPCD_CUDA_TRY(cudaMemcpyAsync(b->stile, stl.data(), stl.size() * sizeof(BTile), cudaMemcpyHostToDevice, st));
    RMPCD_CUDA_TRY(cudaMemcpyAsync(b->stile_first, sfirst.data(), R * sizeof(int), cudaMemcpyHostToDevice, st));
    RMPCD_CUDA_TRY(cudaMemcpyAsync(b->stile_count, scount.data(), R * sizeof(int), cudaMemcpyHostToDevice, st));
    std::vector<int> ids_s(stl.size());
    for (size_t k = 0; k < ids_s.size(); k++) ids_s[k] = (int)k;
    const int n_all[2] = {0, (int)stl.size()}, n_none[2] = {0, 0};
    RMPCD_CUDA_TRY(cudaMemcpyAsync(b->all_s, ids_s.data(), ids_s.size() * sizeof(int), cudaMemcpyHostToDevice, st));
    RMPCD_CUDA_TRY(cudaMemcpyAsync(b->n_all, n_all, sizeof(n_all), cudaMemcpyHostToDevice, st));
    {
        int rc = build_particle_tiles(b, kPTiles[shape_tile(b->shape)]);
        if (rc) {
            free_batch(b);
            return rc;
        }
    }
    RMPCD_CUDA_TRY(cudaMemcpyAsync(b->n_act, n_none, sizeof(n_none), cudaMemcpyHostToDevice, st));
    RMPCD_CUDA_TRY(cudaMemcpyAsync(b->vv_mass, vm.data(), vm.size() * sizeof(double), cudaMemcpyHostToDevice, st));
    RMPCD_CUDA_TRY(cudaMemcpyAsync(b->d_step, &b->step, sizeof(uint64_t), cudaMemcpyHostToDevice, st));
    RMPCD_CUDA_TRY(cudaMemsetAsync(b->aidx, 0xff, (size_t)off * sizeof(int), st));
    for (int *z : {b->nl, b->nx, b->nf, b->adv, b->base})
        RMPCD_CUDA_TRY(cudaMemsetAsync(z, 0, (size_t)R * sizeof(int), st));
    const std::vector<int> never(R, INT_MAX), yes(R, 1);
    RMPCD_CUDA_TRY(cudaMemcpyAsync(b->s_free, never.data(), R * sizeof(int), cudaMemcpyHostToDevice, st));
    RMPCD_CUDA_TRY(cudaMemcpyAsync(b->fresh, yes.data(), R * sizeof(int), cudaMemcpyHostToDevice, st));
    RMPCD_CUDA_TRY(cudaMemsetAsync(b->n_extra, 0, (size_t)R * sizeof(int), st));
    RMPCD_CUDA_TRY(cudaMemsetAsync(b->resort, 0, (size_t)R * sizeof(int), st));
    RMPCD_CUDA_TRY(cudaMemsetAsync(b->done, 0, sizeof(unsigned), st));
    RMPCD_CUDA_TRY(cudaMemsetAsync(b->any, 0, sizeof(int), st));
    Copies cp;
    rc = cp.add(b->stencil, nl[0]->stencil, 3 * (size_t)b->n_stencil * sizeof(int));
    for (int r = 0; r < R; r++) {
        const BRep &p = b->rep_h[r];
        if (rc || (rc = move_particles(cp, b->sol, 0, 1, sol[r], p.off, true)) ||
            (rc = move_particles(cp, b->col, 0, 1, col[r], 2 * r, true))) {
            free_batch(b);
            return rc;
        }
        rmpcd_cells *c = cells[r];
        rc = cp.add(b->count + p.soff, c->count, (size_t)p.S * sizeof(int));
        k_add_offset<<<grid_cap(p.S, 256), 256, 0, st>>>(b->start + p.soff, c->start, p.S, p.off);
        if (!rc) rc = cp.add(b->is_md + p.soff, c->is_md, (size_t)p.S);
        if (!rc) rc = cp.add(b->is_reac + p.soff, c->is_reac, (size_t)p.S);
        k_list_offset<<<grid_cap(2 * (long long)b->Nmax, 256), 256, 0, st>>>(b->list + (size_t)2 * r * b->Nmax, nl[r]->list,
                                                                          nl[r]->n, 2, b->Nmax, p.off);
        if (!rc) rc = cp.add(b->nn + 2 * r, nl[r]->n, 2 * sizeof(int));
    }
    if (!rc) rc = cp.flush();
    if (rc) {
        free_batch(b);
        return rc;
    }
    {
        TileSet all{b->ptile, b->all_p, b->n_all};
        const int gp = resort_grid(b->n_ptile);
        if (b->precision == RMPCD_FP32)
            kb_collect_flagged<float><<<gp, kBT, 0, st>>>(all, b->rep, phys<float>(b->sol, 0), b->sol->key, b->nf);
        else
            kb_collect_flagged<double><<<gp, kBT, 0, st>>>(all, b->rep, phys<double>(b->sol, 0), b->sol->key, b->nf);
    }
    {
        int *neg = nullptr, h_neg = 1;
        if (cudaMalloc(&neg, sizeof(int)) == cudaSuccess && cudaMemsetAsync(neg, 0, sizeof(int), st) == cudaSuccess) {
            k_any_negative<<<grid_cap(b->sol->N, 256), 256, 0, st>>>(b->sol->species[0], b->sol->N, neg);
            if (cudaMemcpyAsync(&h_neg, neg, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess) h_neg = 1;
        }
        rc = sync();
        cudaFree(neg);
        b->read_species = h_neg != 0;
    }
    if (rc) {
        free_batch(b);
        return rc;
    }
    *out = b;
    return RMPCD_OK;
}

static int scatter(Batch *b, int r, rmpcd_particles *sol, rmpcd_particles *col, rmpcd_cells *cells, rmpcd_nlist *nl,
                   rmpcd_rng *rng)
{
    RMPCD_ARG(b && r >= 0 && r < b->R, "dimer batch: replica index out of range");
    const BRep &p = b->rep_h[r];
    cudaStream_t st = stream();
    BRep now;
    RMPCD_CUDA_TRY(cudaMemcpyAsync(&now, b->rep + r, sizeof(BRep), cudaMemcpyDeviceToHost, st));
    int rc = sync();
    if (rc) return rc;
    Copies cp;
    if (sol) {
        RMPCD_ARG(sol->N == p.n && sol->precision == b->precision, "dimer batch: solvent handle does not match");
        // an interval ends with its sort, where pos_old = pos
        if ((rc = move_particles(cp, b->sol, now.cur, b->ran ? now.cur : 1, sol, p.off, false))) return rc;
    }
    if (col) {
        RMPCD_ARG(col->N == 2 && col->precision == RMPCD_FP64, "dimer batch: colloid handle does not match");
        if ((rc = move_particles(cp, b->col, 0, 1, col, 2 * r, false))) return rc;
        if (!col->pos_rattle[0])
            for (int k = 0; k < 3; k++) RMPCD_CUDA_TRY(cudaMalloc(&col->pos_rattle[k], 2 * sizeof(double)));
        for (int k = 0; k < 3 && !rc; k++) rc = cp.add(col->pos_rattle[k], b->rattle[k] + 2 * r, 2 * sizeof(double));
        if (rc) return rc;
    }
    if (cells) {
        RMPCD_ARG(cells->S == p.S, "dimer batch: cell handle does not match");
        rc = cp.add(cells->count, b->count + p.soff, (size_t)p.S * sizeof(int));
        k_add_offset<<<grid_cap(p.S, 256), 256, 0, st>>>(cells->start, b->start + p.soff, p.S, -p.off);
        if (!rc) rc = cp.add(cells->is_md, b->is_md + p.soff, (size_t)p.S);
        if (!rc) rc = cp.add(cells->is_reac, b->is_reac + p.soff, (size_t)p.S);
        if (rc) return rc;
        for (int k = 0; k < 3; k++) cells->origin[k] = now.g.origin[k];
    }
    if (nl) {
        RMPCD_ARG(nl->Npoints == 2 && nl->Nmax == b->Nmax, "dimer batch: neighbor list does not match");
        k_list_offset<<<grid_cap(2 * (long long)b->Nmax, 256), 256, 0, st>>>(nl->list, b->list + (size_t)2 * r * b->Nmax,
                                                                          b->nn + 2 * r, 2, b->Nmax, -p.off);
        if ((rc = cp.add(nl->n, b->nn + 2 * r, 2 * sizeof(int)))) return rc;
    }
    if ((rc = cp.flush())) return rc;
    if (rng) rng->step = b->step;
    return sync();
}

// shape in use <- s: kernel variant and particle tiles; the captured interval
// graphs hold the old launches and are dropped (captured again on the next run)
static int set_shape(Batch *b, int s)
{
    RMPCD_CUDA_TRY(cudaStreamSynchronize(stream()));
    int rc = build_particle_tiles(b, kPTiles[shape_tile(s)]);
    if (rc) return rc;
    if (b->exec) {
        cudaGraphExecDestroy(b->exec);
        b->exec = nullptr;
    }
    b->shape = s;
    return RMPCD_OK;
}

// chosen shapes per GPU, precision, N_MD and mix of boxes (batches on
// different host threads may tune at once: the map is guarded)
static std::map<std::string, int> g_batch_tuned;
static std::mutex g_batch_tuned_mu;

static bool tuned_lookup(const std::string &key, int *shape)
{
    std::lock_guard<std::mutex> lk(g_batch_tuned_mu);
    auto hit = g_batch_tuned.find(key);
    if (hit == g_batch_tuned.end()) return false;
    *shape = hit->second;
    return true;
}

static std::string tune_key(const Batch *b)
{
    int dev = 0;
    cudaGetDevice(&dev);
    std::map<std::vector<int>, int> mix;
    for (const BRep &p : b->rep_h) mix[{p.g.L[0], p.g.L[1], p.g.L[2]}]++;
    std::string k = std::to_string(dev) + ":" + std::to_string(b->precision) + ":" + std::to_string(b->prm.N_MD);
    for (auto &m : mix)
        k += ":" + std::to_string(m.first[0]) + "x" + std::to_string(m.first[1]) + "x" + std::to_string(m.first[2]) +
             "*" + std::to_string(m.second);
    return k;
}

static int run_any(Batch *b, int n)
{
    if (b->precision == RMPCD_FP32) return run_t<float>(b, n);
    return run_t<double>(b, n);
}

static int autotune(Batch *b, int n_intervals, int *best, float *ms, int *ran)
{
    *ran = 0;
    const std::string key = tune_key(b);
    int remembered = 0;
    if (tuned_lookup(key, &remembered)) {
        *best = remembered;
        if (ms)
            for (int k = 0; k < kBShapes; k++) ms[k] = -1.0f;
        return set_shape(b, remembered);
    }
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    RMPCD_CUDA_TRY(cudaEventCreate(&e0));
    if (cudaEventCreate(&e1) != cudaSuccess) {
        cudaEventDestroy(e0);
        return fail(RMPCD_ERR_CUDA, "dimer batch autotune: event creation failed");
    }
    int rc = RMPCD_OK, b_best = b->shape;
    float best_ms = 0;
    if (ms)
        for (int k = 0; k < kBShapes; k++) ms[k] = -1.0f;
    // every tile size and kernel variant with one list entry per thread,
    // then the best of them with each other list setting
    std::vector<int> order;
    for (int k = 0; k < kNPTiles * kBVars; k++) order.push_back(k);
    for (size_t oi = 0; !rc; oi++) {
        if (oi == (size_t)kNPTiles * kBVars && order.size() == oi)
            for (int m = 1; m < kNListPer; m++) order.push_back(b_best + m * kNPTiles * kBVars);
        if (oi >= order.size()) break;
        const int k = order[oi];
        rc = set_shape(b, k);
        // one interval captures the shape's graph and warms it up; then the
        // timed ones
        if (!rc) rc = run_any(b, 1);
        if (!rc && cudaEventRecord(e0, stream()) != cudaSuccess) rc = fail(RMPCD_ERR_CUDA, "event record");
        if (!rc) rc = run_any(b, n_intervals);
        if (!rc && cudaEventRecord(e1, stream()) != cudaSuccess) rc = fail(RMPCD_ERR_CUDA, "event record");
        float t = 0;
        if (!rc && (cudaEventSynchronize(e1) != cudaSuccess || cudaEventElapsedTime(&t, e0, e1) != cudaSuccess))
            rc = fail(RMPCD_ERR_CUDA, "dimer batch autotune: event timing failed");
        if (rc) break;
        *ran += 1 + n_intervals;
        t /= (float)n_intervals;
        if (ms) ms[k] = t;
        if (oi == 0 || t < best_ms) {
            best_ms = t;
            b_best = k;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) return rc;
    {
        std::lock_guard<std::mutex> lk(g_batch_tuned_mu);
        g_batch_tuned[key] = b_best;
    }
    *best = b_best;
    return set_shape(b, b_best);
}

}  // namespace rmpcd

using namespace rmpcd;

extern "C" {

int rmpcd_dimer_batch_shapes(int precision, int *n_shapes)
{
    RMPCD_ARG(n_shapes, "null argument");
    RMPCD_ARG(precision == RMPCD_FP32 || precision == RMPCD_FP64, "precision must be RMPCD_FP32 or RMPCD_FP64");
    *n_shapes = kBShapes;
    return RMPCD_OK;
}

int rmpcd_dimer_batch_shape_info(int precision, int shape, int *particles_per_tile, int *per_thread_begin,
                                 int *per_thread_end, int *blocks_per_sm, int *list_entries_per_thread,
                                 int *colloid_block_first)
{
    RMPCD_ARG(precision == RMPCD_FP32 || precision == RMPCD_FP64, "precision must be RMPCD_FP32 or RMPCD_FP64");
    RMPCD_ARG(shape >= 0 && shape < kBShapes, "no such engine shape");
    if (particles_per_tile) *particles_per_tile = (int)kPTiles[shape_tile(shape)];
    if (list_entries_per_thread) *list_entries_per_thread = kListPer[shape_list(shape)];
    if (colloid_block_first) *colloid_block_first = 1;
    const int warps = kPartThreads[shape_var(shape)] / 32;
    if (per_thread_begin) *per_thread_begin = warps;
    if (per_thread_end) *per_thread_end = warps;
    if (blocks_per_sm) *blocks_per_sm = 1;
    return RMPCD_OK;
}

int rmpcd_dimer_batch_set_shape(rmpcd_dimer_batch *b, int shape)
{
    RMPCD_ARG(b, "null argument");
    RMPCD_ARG(shape >= 0 && shape < kBShapes, "no such engine shape");
    return set_shape(b, shape);
}

int rmpcd_dimer_batch_get_shape(const rmpcd_dimer_batch *b, int *shape)
{
    RMPCD_ARG(b && shape, "null argument");
    *shape = b->shape;
    return RMPCD_OK;
}

int rmpcd_dimer_batch_autotune(rmpcd_dimer_batch *b, int n_intervals, int *best, float *ms_per_interval,
                               int *intervals_run)
{
    RMPCD_ARG(b && best && intervals_run, "null argument");
    RMPCD_ARG(n_intervals >= 1, "n_intervals must be >= 1");
    return autotune(b, n_intervals, best, ms_per_interval, intervals_run);
}

int rmpcd_dimer_batch_create(rmpcd_dimer_batch **out, int n_replicas, rmpcd_particles *const *solvent,
                             rmpcd_particles *const *colloids, rmpcd_cells *const *cells,
                             rmpcd_nlist *const *nlists, const rmpcd_rng *rngs, const rmpcd_lj *solvent_colloid,
                             const rmpcd_lj *colloid_colloid, const rmpcd_dimer_params *params)
{
    RMPCD_ARG(out, "null argument");
    *out = nullptr;
    return create(out, n_replicas, solvent, colloids, cells, nlists, rngs, solvent_colloid, colloid_colloid, params);
}

int rmpcd_dimer_batch_destroy(rmpcd_dimer_batch *b)
{
    free_batch(b);
    return RMPCD_OK;
}

int rmpcd_dimer_batch_set_graph(rmpcd_dimer_batch *b, int use_graph)
{
    RMPCD_ARG(b, "null argument");
    b->use_graph = use_graph != 0;
    return RMPCD_OK;
}

int rmpcd_dimer_batch_run(rmpcd_dimer_batch *b, int n_intervals)
{
    RMPCD_ARG(b, "null argument");
    RMPCD_ARG(n_intervals >= 0, "n_intervals must be >= 0");
    if (b->precision == RMPCD_FP32) return run_t<float>(b, n_intervals);
    return run_t<double>(b, n_intervals);
}

int rmpcd_dimer_batch_scatter(rmpcd_dimer_batch *b, int replica, rmpcd_particles *solvent,
                              rmpcd_particles *colloids, rmpcd_cells *cells, rmpcd_nlist *nlist, rmpcd_rng *rng)
{
    return scatter(b, replica, solvent, colloids, cells, nlist, rng);
}

int rmpcd_dimer_batch_info(const rmpcd_dimer_batch *b, int *n_replicas, long long *n_solvent, int *n_extra_sorting)
{
    RMPCD_ARG(b, "null argument");
    if (n_replicas) *n_replicas = b->R;
    if (n_solvent) *n_solvent = b->Ntot;
    if (n_extra_sorting) {
        RMPCD_CUDA_TRY(cudaMemcpyAsync(n_extra_sorting, b->n_extra, (size_t)b->R * sizeof(int), cudaMemcpyDeviceToHost,
                                       stream()));
        return rmpcd::sync();
    }
    return RMPCD_OK;
}

}  // extern "C"
