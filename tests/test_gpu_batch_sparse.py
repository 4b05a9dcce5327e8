"""The replica engine where its particle warps have little to do: fluids so thin
that most MD steps have no pair force, with particles fast enough that their own
displacement, decided a step ahead of the beads, ends the MD steps."""
import pytest

from test_gpu_batch_active import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("rho,speed", [(0.02, 1.0), (0.1, 6.0), (0.5, 6.0)])
def test_thin_fluid(rm, precision, rho, speed):
    from rmpcdmd_b200.programs import SingleDimerPBC

    two = []
    for _ in range(2):
        d = SingleDimerPBC(L=(14, 13, 16), rho=rho, N_MD=50, tau=0.5, seed=11, list_capacity=4000, precision=precision)
        d.solvent.vel = d.solvent.vel * speed
        two.append(d)
    compare(*two, 4)
    if speed > 1:
        assert two[0].n_extra_sorting >= 4
