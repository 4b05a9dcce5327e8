"""Solvent that the caller flagged, in lists and out of them, in such numbers that
the flagged particles' places among the active ones go beyond the room that the
lists' tables have for a replica."""
import numpy as np
import pytest

from test_gpu_batch import assert_dimers_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
def test_more_flagged_particles_than_list_places(rm, precision):
    from rmpcdmd_b200.programs import DimerBatch, SingleDimerPBC

    def replicas():
        out = []
        for k, L in enumerate([(14, 13, 16), (13, 14, 14)]):
            d = SingleDimerPBC(L=L, rho=10, N_MD=12, tau=0.12, seed=21 + k, list_capacity=6500, precision=precision)
            r = np.random.default_rng(5 + k)
            bits = r.choice([0, 1 << rm.WALL_BIT, 1 << rm.REAC_BIT], size=d.N, p=[0.2, 0.4, 0.4]).astype(np.int32)
            d.solvent.flags = d.solvent.flags | bits
            assert np.count_nonzero(bits) > 2 * 6500
            d.solvent.copy_pos_old()
            d.colloids.copy_pos_old()
            out.append(d)
        return out

    ref, mine = replicas(), replicas()
    b = DimerBatch(mine)
    for d in ref:
        d.interval()
        d.interval()
    b.run(2)
    for r in range(2):
        b.scatter(r)
        assert_dimers_equal(ref[r], mine[r])
    rm.get_status()
