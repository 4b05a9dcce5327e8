"""The collision kernels' shared-memory tiles (64 slots, 832 particles) at their
edges: a box of fewer slots than a tile, ragged boxes, tiles with more
particles than fit (the global-memory path), single particles."""
import numpy as np
import pytest

from helpers import assert_same, make_pair

pytestmark = pytest.mark.gpu

CASES = [((2, 2, 2), 1), ((2, 2, 2), 90), ((5, 7, 9), 3150), ((8, 8, 8), 512 * 13), ((8, 8, 8), 512 * 20),
         ((16, 4, 4), 256 * 14)]


def pair(rm, oracle, L, N, walls=False):
    r = np.random.default_rng(N)
    sp = r.choice([1, 2, 0], size=N, p=[0.6, 0.3, 0.1]).astype(np.int32)
    return make_pair(rm, oracle, list(L), N, seed=N, species=sp, walls=walls,
                     origin=[-0.5, -0.5, 0.0] if walls else [-0.3, -0.8, -0.1])


@pytest.mark.parametrize("L,N", CASES)
@pytest.mark.parametrize("thermostat", [False, True])
def test_collisions_and_temperature(rm, oracle, L, N, thermostat):
    (oc, op), (gc, gp) = pair(rm, oracle, L, N)
    oracle.simple_mpcd_step(op, oc, 11, 3, thermostat=thermostat, T=0.4)
    rm.simple_mpcd_step(gp, gc, rm.Rng(11, 3), thermostat=thermostat, T=0.4)
    assert_same(gp, op, ("vel",))
    if N > 1:
        t_o, t_g = oracle.compute_temperature(op, oc), rm.compute_temperature(gp, gc)
        # sums of the same non-negative cell values in another order
        assert abs(t_g - t_o) <= oc.S * 2.0 ** -52 * abs(t_o)
        v_o, v_g = oracle.velocity_sums(op), rm.velocity_sums(gp)
        assert abs(v_g[0] - v_o[0]) <= N * 2.0 ** -52 * v_o[0]
    oracle.rescale_cells(op, oc, 0.7)
    rm.rescale_cells(gp, gc, None, 0.7)
    assert_same(gp, op, ("vel",))


@pytest.mark.parametrize("L,N", CASES[2:])
@pytest.mark.parametrize("thermostat,keep", [(False, True), (True, True), (True, False)])
def test_wall_collisions(rm, oracle, L, N, thermostat, keep):
    (oc, op), (gc, gp) = pair(rm, oracle, L, N, walls=True)
    wt, wn = [0.8, 1.2], [12, 9]
    oracle.wall_mpcd_step(op, oc, 3, 9, wall_temperature=wt, wall_n=wn, thermostat=thermostat, bulk_temperature=0.6,
                          keep_cell_v=keep)
    rm.wall_mpcd_step(gp, gc, rm.Rng(3, 9), wall_temperature=wt, wall_v=np.zeros((3, 2)), wall_n=wn,
                      thermostat=thermostat, bulk_temperature=0.6, keep_cell_v=keep)
    assert_same(gp, op, ("vel",))
