// Counting and stable cell sort of a particle system (the core of
// count_particles, src/cell_system.f90:86-129, and particle_system_t%sort,
// src/particle_system.f90:304-355).
//
// Schedule (all on the library stream):
//   key/count  one pass over positions: key[i] = slot, warp-aggregated
//              atomic histogram into count[]
//   scan       exclusive scan count -> start, cursor
//   perm       one pass over keys: warp-aggregated cursor atomics give every
//              particle a place inside its cell: perm[place] = i
//   gather     tile by tile, each cell's perm segment is put in ascending
//              order in shared memory, which restores the reference's
//              single-thread order (stable in i), then dst[j] = src[perm[j]]
//              for every field: coalesced writes, reads local in the Hilbert
//              order
#pragma once
#include "state.cuh"

namespace rmpcd {

// key[] and count/start/cursor of p under the current origin of c
int count_and_scan(rmpcd_cells *c, rmpcd_particles *p, bool keep_key);
// perm[] from key[] and cursor[] (cell order fixed, in-cell order arbitrary)
int build_perm_unsorted(rmpcd_cells *c, rmpcd_particles *p, int *cellmap = nullptr);
// ascending sort of every cell's perm segment (uses cursor[] and key[] as scratch)
int sort_perm_segments(rmpcd_cells *c, rmpcd_particles *p);
// both of the above
int build_perm(rmpcd_cells *c, rmpcd_particles *p);
// gather every field through perm (unsorted inside the cells) into the other
// buffer and flip buffers
int gather_all(rmpcd_cells *c, rmpcd_particles *p);
// full sort
int sort_particles(rmpcd_cells *c, rmpcd_particles *p);
// positions of `from` into `to` in cell order (cell_system_t%sort_particles)
int sort_positions(rmpcd_cells *c, const rmpcd_particles *from, rmpcd_particles *to);
// the sort of a wrapped system after its key pass (p->key holds every
// particle's slot in the cells' grid, c->count their counts), for a system in
// which a particle with neither MD nor PAST_MD set has zero force and
// force_old (the state compute_force and its flag roll maintain): scan,
// placement and a gather that moves force entries only where there are any;
// cellmap receives the slot of every particle of the sorted arrays, flagged (N
// entries) their indices that have MD or PAST_MD set, counted in *n_flagged
// (zero on entry)
int sort_keyed_flagged(rmpcd_cells *c, rmpcd_particles *p, int *cellmap, int *flagged, int *n_flagged);
// compute_force_n2 of the colloids run right after compute_force, with the
// colloid sums, on a second stream beside the solvent force application
// (the two branches write disjoint arrays; each array sees the arithmetic
// of the two calls in sequence)
struct ForceN2Branch {
    const rmpcd_lj *lj_cc;      // colloid-colloid parameters of compute_force_n2
    cudaStream_t side;
    cudaEvent_t ev_fork, ev_join;
    const int *gate;            // device word; non-zero: every kernel of the evaluation returns at once (or null)
};
// compute_force (src/neighbor_list.f90:159-225); roll_flags = false leaves
// the PAST_MD/MD roll to the caller (which must then have done it).  n2 (no
// energy only): also compute_force_n2 of ps1, as above.
int compute_force_impl(rmpcd_particles *ps1, rmpcd_particles *ps2, rmpcd_nlist *nl, const double L[3],
                       const rmpcd_lj *lj, double *energy, bool roll_flags, const ForceN2Branch *n2 = nullptr);
// drops the n_colloids loop kept between calls if it refers to `handle` (a
// particle system, cell system or neighbor list being destroyed)
void ncolloids_forget(const void *handle);
}  // namespace rmpcd
