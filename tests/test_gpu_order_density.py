"""The ordering inside the sorts' gathers away from density 10: tiles of fewer slots
for denser fluids (one from 816 particles per cell on), crowded tiles in runs of
cells, by rank (up to 64 particles per cell) or by merging, and cells too large for
shared memory."""
import numpy as np
import pytest

from helpers import assert_cells_same, assert_same, make_pair, upload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,rho", [((9, 8, 7), 0.3), ((9, 8, 7), 12.3), ((9, 8, 7), 13), ((9, 8, 7), 40), ((9, 8, 7), 150),
                                   ((3, 3, 2), 800), ((3, 2, 1), 1640), ((3, 2, 1), 2500)])
def test_even_fluids(rm, oracle, L, rho):
    n = int(rho * np.prod(L))
    (oc, op), (gc, gp) = make_pair(rm, oracle, list(L), n, seed=n, sorted_=True)
    assert_cells_same(gc, oc)
    assert_same(gp, op)


@pytest.mark.parametrize("sizes", [(31, 32, 33, 63, 64, 64, 64, 2000), (65, 66, 1, 127, 128, 129, 300, 1791), (1792,), (1793,),
                                   (700, 700, 700, 700, 64, 65), (1792, 1792, 20), (40000, 5, 4097), (64,) * 40])
@pytest.mark.parametrize("precision", [64, 32])
def test_crowded_cells(rm, oracle, sizes, precision):
    """Cells of these sizes side by side, with one particle in every third other."""
    L = [8, 8, 4]
    rng = np.random.default_rng(len(sizes) + sum(sizes))
    # the cells in slot order, from a system with one particle per cell
    (tc, tp), _ = make_pair(rm, oracle, L, 256, seed=1, sorted_=False)
    tp.pos[:] = np.stack(np.unravel_index(np.arange(256), L), axis=1) + 0.5
    tp.sort(tc)
    cells = np.floor(tp.pos)
    where = np.concatenate([np.repeat(cells[q + 5:q + 6], m, axis=0) for q, m in enumerate(sizes)] + [cells[60::3]])
    n = len(where)
    (oc, op), (gc, gp) = make_pair(rm, oracle, L, n, seed=n, precision=precision, sorted_=False)
    op.pos[:] = rng.permutation(where + 0.05 + 0.9 * rng.random((n, 3)))
    op.force[:] = rng.normal(size=(n, 3))
    upload(gp, op, ("pos", "force"))
    if precision == 32:
        op.pos[:], op.vel[:], op.force[:] = (gp.download(f) for f in ("pos", "vel", "force"))
    op.sort(oc)
    gp.sort(gc)
    assert_cells_same(gc, oc)
    assert_same(gp, op, ("pos", "vel", "image", "id", "species", "flags", "force", "force_old"))


@pytest.mark.parametrize("precision", [64, 32])
def test_dense_replicas(rm, precision):
    """The replica engine's sort at density 20."""
    from rmpcdmd_b200.programs import DimerBatch, SingleDimerPBC
    from test_gpu_batch import assert_dimers_equal

    def replicas():
        return [SingleDimerPBC(L=L, rho=20, N_MD=8, tau=0.4, seed=s, list_capacity=20000, precision=precision)
                for L, s in (((10, 10, 10), 3), ((12, 11, 14), 4))]

    ref, mine = replicas(), replicas()
    b = DimerBatch(mine)
    for d in ref:
        d.interval()
        d.interval()
    b.run(2)
    for r in range(2):
        b.scatter(r)
        assert_dimers_equal(ref[r], mine[r])
    assert sum(d.n_extra_sorting for d in ref) > 0
