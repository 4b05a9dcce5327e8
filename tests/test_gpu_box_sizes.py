"""The fused bulk interval at box sizes around the lines of its shape rule and
of the slot scan (tiles of 4096 slots, one launch for up to eight)."""
import numpy as np
import pytest

from helpers import SOLVENT_FIELDS, assert_cells_same, assert_same, make_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [(4, 5, 3), (16, 16, 16), (17, 16, 15), (21, 20, 20), (26, 26, 25), (33, 20, 30),
                               (40, 36, 23)])
def test_bulk_run_box_sizes(rm, oracle, L):
    """FP64 intervals equal the oracle bit for bit; the FP32 form's arrays do
    not depend on the shape that the box selects."""
    N = 10 * int(np.prod(L))
    (oc, op), (gc, gp) = make_pair(rm, oracle, L, N, seed=sum(L), n_species=1)
    oracle.set_threads(1)
    oracle.bulk_run(op, oc, 2, 1.0, 7, 0)
    rm.bulk_run(gp, gc, rm.Rng(7, 0), 1.0, 2)
    assert_same(gp, op, SOLVENT_FIELDS)
    assert_cells_same(gc, oc)
    out = []
    for shape in (None, 2):
        (_, _), (gc, gp) = make_pair(rm, oracle, L, N, seed=sum(L), n_species=1, precision=32)
        keep = rm.bulk_shape(rm.FP32)
        if shape is not None:
            rm.set_bulk_shape(rm.FP32, shape)
        rm.bulk_run(gp, gc, rm.Rng(7, 0), 1.0, 2)
        out.append({f: gp.download(f) for f in SOLVENT_FIELDS})
        if shape is not None:
            rm.set_bulk_shape(rm.FP32, keep)
    for f in SOLVENT_FIELDS:
        assert np.array_equal(out[0][f], out[1][f]), f
