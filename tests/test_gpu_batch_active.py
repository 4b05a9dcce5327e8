"""The replica engine moves only the solvent that can meet a bead in every MD
step; the rest is advanced at the next sort.  Cases at the edges of that split:
lists beyond the shared-memory tables of the MD kernel, flags that the caller
set on particles outside every list, negative species, MD loops of one step."""
import numpy as np
import pytest

from test_gpu_batch import assert_dimers_equal

pytestmark = pytest.mark.gpu


def twins(change=None, **kw):
    from rmpcdmd_b200.programs import SingleDimerPBC

    out = []
    for _ in range(2):
        d = SingleDimerPBC(rho=10, **kw)
        if change:
            change(d)
        out.append(d)
    return out


def compare(ref, mine, intervals):
    from rmpcdmd_b200.programs import DimerBatch

    b = DimerBatch([mine])
    for _ in range(intervals):
        ref.interval()
    b.run(intervals)
    b.scatter(0)
    assert_dimers_equal(ref, mine)


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("sigma,d,L", [(3.0, 6.5, 24), (5.0, 11.0, 36)])
def test_long_lists(rm, precision, sigma, d, L):
    """~6,000 and ~17,000 entries per list; more than 1,024 pair forces per bead
    at sigma = 5."""
    ref, mine = twins(L=(L, L, L), N_MD=12, sigma_C=sigma, sigma_N=sigma, d=d, seed=4, tau=0.12, list_capacity=40000,
                      precision=precision)
    compare(ref, mine, 2)


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("N_MD", [1, 2, 9])
def test_flags_and_species_of_the_caller(rm, precision, N_MD):
    """WALL and REAC bits on particles anywhere in the box, some species
    negative, and an MD loop that ends where it begins."""
    def change(d):
        r = np.random.default_rng(3)
        n = d.N
        d.solvent.flags = d.solvent.flags | r.choice([0, 1 << rm.WALL_BIT, 1 << rm.REAC_BIT], size=n,
                                                     p=[0.8, 0.1, 0.1]).astype(np.int32)
        d.solvent.species = np.where(r.random(n) < 0.05, -1, d.solvent.species).astype(np.int32)
        # the displacement test starts from pos_old = pos, as after a sort
        d.solvent.copy_pos_old()
        d.colloids.copy_pos_old()

    ref, mine = twins(change, L=(14, 13, 16), N_MD=N_MD, tau=0.01 * N_MD, seed=8, list_capacity=12000, precision=precision)
    compare(ref, mine, 3)


@pytest.mark.parametrize("precision", [64, 32])
def test_fast_particles_decide_the_resort(rm, precision):
    """A few particles far above the thermal speed: the engine's re-sort steps
    are those of the call-by-call test of every particle's displacement."""
    def change(d):
        v = d.solvent.vel
        v[::5000] *= 20.0
        d.solvent.vel = v

    ref, mine = twins(change, L=(16, 16, 16), N_MD=40, tau=0.4, seed=5, list_capacity=12000, precision=precision)
    compare(ref, mine, 2)
    assert ref.n_extra_sorting >= 3
