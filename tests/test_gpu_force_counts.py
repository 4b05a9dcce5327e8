"""compute_force leaves its per-particle contribution counts at zero: repeated
evaluations with beads that share no, some, or more solvent particles than one
block sorts (4,096 entries), against the oracle."""
import numpy as np
import pytest

from helpers import assert_same, make_pair, upload
from test_gpu_nlist import dimer_lj

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("sigma,d,rho,shared", [(2.0, 6.0, 10, (0, 0)), (2.0, 2.5, 10, (10, 4096)),
                                                (6.0, 1.0, 8, (4097, 30000))])
def test_repeated_evaluations(rm, oracle, precision, sigma, d, rho, shared):
    L = np.array([24, 24, 24])
    N = int(np.prod(L) * rho)
    (oc, op), (gc, gp) = make_pair(rm, oracle, L, N, seed=5, species=1, sorted_=False, precision=precision)
    ocol, gcol = oracle.Particles(2, 2, np.ones(2)), rm.ParticleSystem(2, 2, np.ones(2))
    ocol.species[:] = [1, 2]
    ocol.pos[:] = [L / 2, L / 2 + [d, 0, 0]]
    upload(gcol, ocol, ("pos", "species"))
    # no particle far inside a bead
    near = np.min([np.linalg.norm(op.pos - b, axis=1) for b in ocol.pos], axis=0) < 0.9 * sigma
    op.pos[near] = 0.5 + 2 * np.random.default_rng(1).random((near.sum(), 3))
    upload(gp, op, ("pos",))
    op.pos[:], op.vel[:] = gp.download("pos"), gp.download("vel")
    op.sort(oc)
    gp.sort(gc)
    glj, olj = dimer_lj(rm, oracle, sigma)
    cut = sigma * 2 ** (1 / 6)
    inside = [np.linalg.norm(op.pos - b, axis=1) <= cut for b in ocol.pos]
    assert shared[0] <= 2 * (inside[0] & inside[1]).sum() <= shared[1]
    onl, gnl = oracle.NeighborList(2, 20000), rm.NeighborList(2, 20000)
    for nl, c, p, col, lj in ((onl, oc, op, ocol, olj), (gnl, gc, gp, gcol, glj)):
        nl.make_stencil(c, cut + 1)
        nl.update_list(col, p, cut + 1, c, lj)
    for k in range(3):
        op.force[:] = ocol.force[:] = 0
        gp.zero_force()
        gcol.zero_force()
        oracle.compute_force(ocol, op, onl, oc.edges, olj)
        rm.compute_force(gcol, gp, gnl, gc.edges, glj, energy=k == 1)
        if precision == 64:
            assert_same(gp, op, ("force", "flags"))
            assert_same(gcol, ocol, ("force",))
        else:
            # one rounding to 24 bits per contribution, two at most
            assert_same(gp, op, ("force",), exact=False, rtol=4 * 2.0 ** -24, atol=2.0 ** -20 * np.abs(op.force).max())
            assert_same(gp, op, ("flags",))
