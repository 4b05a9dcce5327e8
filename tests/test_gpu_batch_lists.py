"""Lists and active sets beyond what the replica engine's MD kernel holds in shared
memory: pair forces and particles in global memory, and lists longer than the map
of their entries (196,608)."""
import pytest

from test_gpu_batch import assert_dimers_equal

pytestmark = pytest.mark.gpu


def pair(**kw):
    from rmpcdmd_b200.programs import SingleDimerPBC

    return SingleDimerPBC(**kw), SingleDimerPBC(**kw)


def compare(ref, mine, intervals):
    from rmpcdmd_b200.programs import DimerBatch

    b = DimerBatch([mine])
    for _ in range(intervals):
        ref.interval()
    b.run(intervals)
    b.scatter(0)
    assert_dimers_equal(ref, mine)


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("N_MD,skin", [(1, 2.0), (7, 0.4), (40, 2.0)])
def test_large_beads(rm, precision, N_MD, skin):
    """Some 2,000 pair forces per bead and 8,000 active particles, with and without
    re-sorts, in intervals of one step and of many."""
    ref, mine = pair(L=(34, 36, 35), rho=10, sigma_C=5.0, sigma_N=4.5, d=10.8, N_MD=N_MD, tau=0.02 * N_MD, seed=6, skin=skin,
                     list_capacity=40000, precision=precision)
    compare(ref, mine, 3)
    if skin < 1:
        assert ref.n_extra_sorting >= 3


@pytest.mark.parametrize("precision", [64, 32])
def test_lists_beyond_the_map(rm, precision):
    ref, mine = pair(L=(30, 30, 30), rho=35, sigma_C=3.0, sigma_N=3.0, d=6.8, skin=8.0, N_MD=3, tau=0.03, seed=2,
                     list_capacity=400000, precision=precision)
    assert min(ref.neigh.download()[1]) > 196608
    compare(ref, mine, 2)
