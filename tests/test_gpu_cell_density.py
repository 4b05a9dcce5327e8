"""The collision kernels from thin to very dense fluids: their tiles have the slots
that 832 particles in shared memory hold at the fluid's mean density (64 up to
11.3 per cell, 4 at 177), beyond 178 a thread per slot on global memory; and uneven
fluids, whose crowded tiles go run by run or on global memory."""
import numpy as np
import pytest

from helpers import assert_same, make_pair, upload

pytestmark = pytest.mark.gpu

L = (7, 5, 9)
CELLS = 7 * 5 * 9


def crowd(kind, n, rng):
    x = rng.random((n, 3)) * L
    if kind == "octant":  # 8 times the mean in 1/8 of the box
        x *= 0.5
    elif kind == "clumps":  # cells of some 200
        x[::2] = rng.integers(0, 2, (len(x[::2]), 3)) * [5, 3, 6] + 0.1 + 0.8 * rng.random((len(x[::2]), 3))
    elif kind == "one_cell":
        x[:1200] = 2.0 + rng.random((1200, 3))
    return x


CASES = [("even", r) for r in (1, 11.4, 11.7, 13, 20, 46, 100, 176, 179, 240)] + [
    ("octant", 6), ("octant", 11), ("clumps", 10), ("one_cell", 10)]


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("walls", [False, True])
@pytest.mark.parametrize("kind,rho", CASES)
def test_density(rm, oracle, precision, walls, kind, rho):
    """FP64 bit for bit; FP32 velocities (|v| < 6) within 1e-5 of the FP64 ones: some
    ten roundings of 2^-24 relative each, the cells' sums being compensated."""
    n = int(rho * CELLS)
    rng = np.random.default_rng(n)
    sp = rng.choice([1, 2, 0], size=n, p=[0.6, 0.3, 0.1]).astype(np.int32)
    (oc, op), (gc, gp) = make_pair(rm, oracle, list(L), n, seed=n, species=sp, walls=walls, precision=precision,
                                   origin=[-0.5, -0.5, 0.0] if walls else [-0.3, -0.8, -0.1], sorted_=False)
    op.pos[:] = crowd(kind, n, rng)
    upload(gp, op)
    if precision == 32:
        op.pos[:], op.vel[:] = gp.download("pos"), gp.download("vel")
    op.sort(oc)
    gp.sort(gc)

    def same(what):
        v, o = gp.download("vel"), op.vel
        assert np.abs(v - o).max() < 1e-5 if precision == 32 else np.array_equal(v, o), what
        op.vel[:] = v

    for thermostat in (False, True):
        if walls:
            kw = dict(wall_temperature=[0.8, 1.2], wall_n=[12, 9], thermostat=thermostat, bulk_temperature=0.4)
            oracle.wall_mpcd_step(op, oc, 3, 9, **kw)
            rm.wall_mpcd_step(gp, gc, rm.Rng(3, 9), wall_v=np.zeros((3, 2)), **kw)
        else:
            oracle.simple_mpcd_step(op, oc, 11, 3, thermostat=thermostat, T=0.4)
            rm.simple_mpcd_step(gp, gc, rm.Rng(11, 3), thermostat=thermostat, T=0.4)
        same(f"collision, thermostat {thermostat}")
    if walls:
        return
    t_o, t_g = oracle.compute_temperature(op, oc), rm.compute_temperature(gp, gc)
    # FP64: sums of the same non-negative cell values in another order; FP32: the
    # cell means are rounded to 2^-24
    assert abs(t_g - t_o) <= (oc.S * 2.0 ** -52 if precision == 64 else 1e-6) * abs(t_o)
    oracle.rescale_cells(op, oc, 0.7)
    rm.rescale_cells(gp, gc, None, 0.7)
    same("rescaling")
