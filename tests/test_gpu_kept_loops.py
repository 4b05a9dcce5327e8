"""rmpcd_ncolloids_run keeps the loops of the last four systems: more systems
than that run in turn give the states of each run by itself, also when some are
dropped in between."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,systems", [(32, 3), (32, 6), (64, 5)])
def test_systems_in_turn(rm, precision, systems):
    from rmpcdmd_b200.programs import NColloidsPBC

    def make(seed):
        return NColloidsPBC(L=(20, 18, 16), rho=10, N_MD=8, N_colloids=5, seed=seed, precision=precision)

    turn = [make(k) for k in range(systems)]
    for k in range(4):
        for i, x in enumerate(turn):
            if x is not None:
                x.thermalise(1)
        if k == 1:
            turn[1] = None  # its handles go while its loop is kept
    for i, x in enumerate(turn):
        if x is None:
            continue
        alone = make(i)
        for k in range(4):
            alone.thermalise(1)
        for f in ("pos", "vel", "image", "id", "flags", "force", "force_old"):
            assert np.array_equal(x.solvent.download(f), alone.solvent.download(f)), f
        assert np.array_equal(x.colloids.download("pos"), alone.colloids.download("pos"))
        assert x.n_extra_sorting == alone.n_extra_sorting
