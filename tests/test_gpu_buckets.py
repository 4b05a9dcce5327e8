"""The bucket schedule of the bulk interval where its storage runs out: cells
beyond a bucket's records (linked lists), tiles beyond shared memory (the block
goes cell by cell), densities from below one particle per cell to where the
gather takes over, boxes with more slots than cells, species that take no part."""
import numpy as np
import pytest

from helpers import SOLVENT_FIELDS, assert_cells_same, assert_same, make_pair, upload

pytestmark = pytest.mark.gpu


def crowd(kind, L, N, rng):
    pos = rng.random((N, 3)) * L
    if kind == "one_cell":
        pos[:] = 3.0 + rng.random((N, 3))
    elif kind == "crowded_corner":
        pos[::2] = rng.random((len(pos[::2]), 3)) * [3, 2, 2]
    elif kind == "overflow":
        # 23, 24, 25 and 40 more particles in four cells far apart
        k = 0
        for cell, n in (((1, 1, 1), 23), ((6, 1, 5), 24), ((2, 6, 3), 25), ((7, 5, 6), 40)):
            pos[k:k + n] = np.array(cell) + rng.random((n, 3))
            k += n
    return pos


def pair(rm, oracle, kind, L, N, precision):
    (oc, op), (gc, gp) = make_pair(rm, oracle, L, N, seed=N % 89, precision=precision, n_species=2, sorted_=False)
    rng = np.random.default_rng(N)
    op.pos[:] = crowd(kind, L, N, rng)
    op.species[:] = rng.choice([1, 2, 0], size=N, p=[0.6, 0.3, 0.1])
    upload(gp, op)
    if precision == 32:
        op.pos[:], op.vel[:] = gp.download("pos"), gp.download("vel")
    op.sort(oc)
    gp.sort(gc)
    return (oc, op), (gc, gp)


CASES = [("one_cell", (9, 8, 7), 5040), ("crowded_corner", (9, 8, 7), 5040), ("overflow", (9, 8, 7), 5040),
         ("overflow", (8, 8, 8), 5120), ("uniform", (12, 11, 10), 264), ("uniform", (12, 11, 10), 3960),
         ("uniform", (12, 11, 10), 17160), ("uniform", (1, 1, 2), 20)]


@pytest.mark.parametrize("kind,L,N", CASES)
def test_fp64_equals_the_oracle(rm, oracle, kind, L, N):
    oracle.set_threads(1)
    keep = rm.bulk_shape(64)
    try:
        for shape in [None] + list(range(len(rm.bulk_shapes(64)))):
            (oc, op), (gc, gp) = pair(rm, oracle, kind, L, N, 64)
            if shape is not None:
                rm.set_bulk_shape(64, shape)
            for n in (1, 3, 2):  # runs that start from each of the three grids' arrays
                oracle.bulk_run(op, oc, n, 1.0, 7, 2 * n)
                rm.bulk_run(gp, gc, rm.Rng(7, 2 * n), 1.0, n)
            assert_same(gp, op, SOLVENT_FIELDS)
            assert_cells_same(gc, oc)
    finally:
        rm.set_bulk_shape(64, keep)


@pytest.mark.parametrize("kind,L,N", CASES)
def test_fp32_shapes_agree_and_follow_fp64(rm, oracle, kind, L, N):
    """One interval: a velocity is within 1e-5 of the FP64 one (|v| < 6: some ten
    roundings of 2^-24 relative each).  Four: every shape gives the same arrays."""
    oracle.set_threads(1)
    keep = rm.bulk_shape(32)
    out = []
    try:
        for shape in range(len(rm.bulk_shapes(32))):
            (oc, op), (gc, gp) = pair(rm, oracle, kind, L, N, 32)
            rm.set_bulk_shape(32, shape)
            rm.bulk_run(gp, gc, rm.Rng(7, 0), 1.0, 1)
            oracle.bulk_run(op, oc, 1, 1.0, 7, 0)
            v, o = np.empty((N, 3)), np.empty((N, 3))
            v[gp.download("id") - gp.download("id").min()] = gp.download("vel")
            o[op.id - op.id.min()] = op.vel
            assert np.abs(v - o).max() < 1e-5
            rm.bulk_run(gp, gc, rm.Rng(7, 2), 1.0, 3)
            out.append({f: gp.download(f) for f in SOLVENT_FIELDS} | {"n": gc.cell_count})
        for o in out[1:]:
            for f in o:
                assert np.array_equal(o[f], out[0][f]), f
    finally:
        rm.set_bulk_shape(32, keep)
