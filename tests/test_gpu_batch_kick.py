"""A particle whose last force is still to change its velocity: its way is not the
straight one, so the replica engine must have it among the particles that can
meet a bead.  And coarse or hot runs with a small skin, re-sorted in most steps."""
import numpy as np
import pytest

from test_gpu_batch_active import compare, twins

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
def test_kicked_particles_meet_the_bead(rm, precision):
    """Resting particles 2.6 to 3 from the first bead (cut 2.245), half of them
    with MD set and a force that sends them there at speed 1.5."""
    hit = []

    def change(d):
        x = d.solvent.pos - d.colloids.pos[0]
        x -= np.rint(x / d.edges) * d.edges
        r = np.sqrt((x * x).sum(1))
        near = np.nonzero((r > 2.6) & (r < 3.0))[0]
        v, f, flags = d.solvent.vel, d.solvent.download("force"), d.solvent.flags
        v[near] = 0
        kicked = near[::2]
        f[kicked] = -300.0 * x[kicked] / r[kicked, None]
        flags[kicked] |= 1 << rm.MD_BIT
        d.solvent.vel = v
        d.solvent.upload("force", f)
        d.solvent.flags = flags
        d.solvent.copy_pos_old()
        d.colloids.copy_pos_old()
        hit.append(len(kicked))

    ref, mine = twins(change, L=(14, 13, 16), N_MD=60, tau=0.6, seed=9, list_capacity=12000, precision=precision)
    assert hit[0] > 50
    compare(ref, mine, 1)


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("skin,dt,speed", [(0.3, 0.01, 3.0), (0.1, 0.05, 1.0), (2.0, 0.1, 1.0)])
def test_small_skin_and_coarse_steps(rm, precision, skin, dt, speed):
    def change(d):
        d.solvent.vel = d.solvent.vel * speed

    ref, mine = twins(change, L=(14, 13, 16), N_MD=12, tau=12 * dt, seed=2, skin=skin, list_capacity=12000,
                      precision=precision)
    compare(ref, mine, 3)
    assert ref.n_extra_sorting >= 4
