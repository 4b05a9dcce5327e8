"""The automatic tile shape on both sides of its lines (one wave of blocks of 148
SMs) and of the density that a shape's tiles hold: the arrays are those of every
fixed shape."""
import numpy as np
import pytest

from helpers import SOLVENT_FIELDS

pytestmark = pytest.mark.gpu

LINES = [(32, (24, 24, 24), 10), (32, (25, 24, 24), 10), (32, (38, 38, 39), 10), (32, (39, 38, 39), 10),
         (32, (40, 40, 39), 10.6), (32, (40, 40, 39), 11), (32, (41, 40, 39), 10), (32, (18, 18, 18), 11.5),
         (64, (22, 22, 24), 10), (64, (23, 23, 23), 10), (64, (18, 18, 18), 11.2), (64, (18, 18, 18), 12)]


@pytest.mark.parametrize("precision,L,rho", LINES)
def test_automatic_shape(rm, precision, L, rho):
    rng = np.random.default_rng(7)
    n = int(rho * np.prod(L))
    pos, vel = rng.random((n, 3)) * L, rng.normal(size=(n, 3)) * 0.577
    keep, out = rm.bulk_shape(precision), []
    try:
        for shape in (-1, 0, 2):
            rm.set_bulk_shape(precision, shape)
            c, p, g = rm.CellSystem(list(L), 1.0), rm.ParticleSystem(n, 1, None, precision), rm.Rng(3)
            p.pos, p.vel, p.species = pos, vel, 1
            c.random_shift(g)
            p.sort(c)
            rm.bulk_run(p, c, g, 1.0, 3)
            out.append({f: p.download(f) for f in SOLVENT_FIELDS} | {"n": c.cell_count, "a": c.cell_start})
    finally:
        rm.set_bulk_shape(precision, keep)
    for o in out[1:]:
        for f in o:
            assert np.array_equal(o[f], out[0][f]), f
