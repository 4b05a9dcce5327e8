"""Over-full tiles of the bulk interval: most of the particles in lists, tiles of
several shared-memory fills, with and without cells larger than one."""
import numpy as np
import pytest

from helpers import SOLVENT_FIELDS, assert_cells_same, assert_same, make_pair, upload

pytestmark = pytest.mark.gpu

L = (10, 8, 8)
N = 6400


def crowd(kind, rng):
    x = rng.random((N, 3)) * L
    if kind == "octant":  # 80 per cell
        x *= 0.5
    elif kind == "cells of 300":
        x[:4800] = rng.integers(0, 2, (4800, 3)) * [3, 2, 1] + rng.random((4800, 3)) + [0, 2, 4]
    elif kind == "small and large":  # 353 to 1,500 in one cell, 80 per cell around it
        x *= 0.5
        x[:1500] = 2.0 + rng.random((1500, 3))
    return x


@pytest.mark.parametrize("kind", ["octant", "cells of 300", "small and large"])
@pytest.mark.parametrize("speed", [0.0, 0.577])
def test_crowds(rm, oracle, kind, speed):
    """FP64 equals the oracle with every shape; the FP32 arrays are the same with every
    shape and, after one interval, within 1e-5 of the FP64 velocities (some ten
    roundings of 2^-24 relative each, |v| < 6)."""
    oracle.set_threads(1)
    for precision in (64, 32):
        keep, first = rm.bulk_shape(precision), None
        try:
            for shape in range(-1, len(rm.bulk_shapes(precision))):
                (oc, op), (gc, gp) = make_pair(rm, oracle, L, N, seed=5, precision=precision, sorted_=False)
                rng = np.random.default_rng(17)
                op.pos[:] = crowd(kind, rng)
                op.vel[:] = rng.normal(size=(N, 3)) * speed
                op.species[:] = rng.choice([1, 2, 0], size=N, p=[0.6, 0.3, 0.1])
                upload(gp, op)
                if precision == 32:
                    op.pos[:], op.vel[:] = gp.download("pos"), gp.download("vel")
                op.sort(oc)
                gp.sort(gc)
                rm.set_bulk_shape(precision, shape)
                step = 0
                for n in (1, 3):
                    rm.bulk_run(gp, gc, rm.Rng(7, step), 1.0, n)
                    if precision == 64 or step == 0:
                        oracle.bulk_run(op, oc, n, 1.0, 7, step)
                    if precision == 32 and step == 0:
                        v, o = np.empty((N, 3)), np.empty((N, 3))
                        v[gp.download("id") - 1], o[op.id - 1] = gp.download("vel"), op.vel
                        assert np.abs(v - o).max() < 1e-5
                    step += 2 * n
                if precision == 64:
                    assert_same(gp, op, SOLVENT_FIELDS)
                    assert_cells_same(gc, oc)
                else:
                    out = {f: gp.download(f) for f in SOLVENT_FIELDS} | {"n": gc.cell_count}
                    first = first or out
                    for f in out:
                        assert np.array_equal(out[f], first[f]), (shape, f)
        finally:
            rm.set_bulk_shape(precision, keep)
