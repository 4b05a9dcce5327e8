"""The gather that orders each cell's indices tile by tile (128 slots, 1,792
particles in shared memory, cells of more than 64 ordered by the block): tiles
and cells at those sizes, and force buffers between gated and plain sorts."""
import numpy as np
import pytest

from helpers import assert_cells_same, assert_same, make_pair, upload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("in_tile,in_cell", [(1791, 10), (1792, 64), (1793, 0), (1793, 64), (2000, 65), (2500, 1300),
                                             (1792, 1792), (1793, 1793)])
def test_tile_and_cell_sizes(rm, oracle, precision, in_tile, in_cell):
    """An 8x8x4 box is two tiles of 128 slots in every cell order: one half
    holds in_tile particles, in_cell of them in one cell, shuffled."""
    L, N = [8, 8, 4], 4000
    (oc, op), (gc, gp) = make_pair(rm, oracle, L, N, seed=in_tile + in_cell, precision=precision, sorted_=False)
    rng = np.random.default_rng(in_cell)
    # the cells of each tile, from a system with one particle per cell
    (tc, tp), _ = make_pair(rm, oracle, L, 256, seed=1, sorted_=False)
    tp.pos[:] = np.stack(np.unravel_index(np.arange(256), L), axis=1) + 0.5
    tp.sort(tc)
    assert np.array_equal(tc.cell_count, np.ones(256))
    first, second = np.floor(tp.pos[:128]), np.floor(tp.pos[128:])
    where = np.concatenate([np.repeat(first[3:4], in_cell, axis=0),
                            first[rng.integers(0, len(first), in_tile - in_cell)],
                            second[rng.integers(0, len(second), N - in_tile)]])
    op.pos[:] = rng.permutation(where + 0.05 + 0.9 * rng.random((N, 3)))
    op.force[:] = rng.normal(size=(N, 3))
    upload(gp, op, ("pos", "force"))
    if precision == 32:
        op.pos[:], op.vel[:], op.force[:] = (gp.download(f) for f in ("pos", "vel", "force"))
    op.sort(oc)
    gp.sort(gc)
    assert_cells_same(gc, oc)
    assert_same(gp, op, ("pos", "vel", "image", "id", "species", "flags", "force", "force_old"))


@pytest.mark.parametrize("precision", [64, 32])
def test_force_buffers_between_plain_and_gated_sorts(rm, precision):
    """Caller's sorts with every force set, between native loops whose sorts
    move force entries of flagged particles only."""
    from rmpcdmd_b200.programs import NColloidsPBC

    kw = dict(L=(20, 20, 20), rho=10, N_MD=8, N_colloids=6, seed=12, precision=precision)
    a, b = NColloidsPBC(**kw), NColloidsPBC(**kw)
    for k in range(3):
        for x, native in ((a, False), (b, True)):
            x.thermalise(2, native=native)
            f, fo = x.solvent.download("force"), x.solvent.download("force_old")
            flags, pos_old, origin = x.solvent.download("flags"), x.solvent.download("pos_old"), x.cells.origin
            noise = np.random.default_rng(k).normal(size=f.shape)
            for q in range(k):
                x.solvent.upload("force", noise)
                x.solvent.upload("force_old", -noise)
                x.solvent.sort(x.cells)  # sorted already: the order stays
            x.solvent.upload("force", f)
            x.solvent.upload("force_old", fo)
            x.solvent.upload("pos_old", pos_old)
            assert np.array_equal(x.solvent.download("flags"), flags)
        for fld in ("pos", "vel", "id", "flags", "force", "force_old"):
            assert np.array_equal(a.solvent.download(fld), b.solvent.download(fld)), fld
    assert b.n_extra_sorting > 0 and a.n_extra_sorting == b.n_extra_sorting
