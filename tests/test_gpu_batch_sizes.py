"""Several replicas whose particle numbers and list capacities are odd: each one's
part of the engine's arrays begins where its elements are aligned."""
import pytest

from test_gpu_batch import assert_dimers_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("rho,capacity,skin", [(15, 60001, 0.5), (15, 12001, 2.0), (9, 7001, 1.0), (3, 1333, 0.5)])
def test_odd_sizes(rm, precision, rho, capacity, skin):
    from rmpcdmd_b200.programs import DimerBatch, SingleDimerPBC

    def replicas():
        return [SingleDimerPBC(L=L, rho=rho, N_MD=9, tau=0.18, seed=s, skin=skin, list_capacity=capacity, precision=precision)
                for L, s in (((13, 17, 13), 3), ((11, 13, 15), 4), ((13, 11, 11), 5))]

    ref, mine = replicas(), replicas()
    b = DimerBatch(mine)
    for d in ref:
        d.interval()
        d.interval()
    b.run(2)
    for r in range(3):
        b.scatter(r)
        assert_dimers_equal(ref[r], mine[r])
    rm.get_status()
