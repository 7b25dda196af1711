"""The batched solver's kernel where its shapes change, against the
single-instance solver (same seeds): candidate lists of every padding (1 ..
32), sizes around the pairs and batches of the scan and the tier threshold,
colonies of a partial warp and of several rounds, demands of one, two and four
bytes, more than 32 vehicles (the repair's groups) and one-customer routes
(the deposit's shared cells).  Routes, costs and epochs are equal exactly."""
import numpy as np
import pytest

from tests.test_gpu_batch import plain
from vehicleroutingproblem_b200 import _native
from vehicleroutingproblem_b200 import instances as I

pytestmark = pytest.mark.gpu


def _tight(n, K, seed, demand_max=100, slack=1.02):
    inst = I.uniform_instance(n, K, seed, demand_max=max(2, demand_max))
    if demand_max == 1:
        inst.demand[1:] = 1
    cap = max(int(np.ceil(inst.demand.sum() / K * slack)), int(inst.demand.max()))
    return I.Instance(inst.name, inst.x, inst.y, inst.demand, K, cap)


def _check(insts, ants, k, epochs, tuning, seed=500):
    with _native.Batch(0) as b:
        b.setup(insts, ants=ants, cand_k=k, seed=seed, epochs=epochs)
        b.set_tuning(*tuning)
        b.solve()
        for i, inst in enumerate(insts):
            nodes, lens, cost, ep = b.best(i)
            rn, rl, rc, re = plain(inst, seed + i, ants, k, epochs)
            assert ep == re and cost == rc, (i, inst.n, cost, rc)
            assert np.array_equal(nodes, rn) and (len(rn) == 0 or np.array_equal(lens, rl)), i


@pytest.mark.parametrize("k", [1, 3, 4, 5, 13, 16, 17, 21, 28, 31, 32])
def test_candidate_lengths(k):
    insts = [_tight(max(k, n), K, 800 + n) for n, K in [(32, 3), (75, 4), (130, 5), (300, 6)]]
    _check(insts, 20, k, 5, (32, 16, 1))


@pytest.mark.parametrize("demand_max", [1, 254, 255, 65534, 65535, 900000])
def test_sizes_and_demands(demand_max):
    sizes = [16, 31, 32, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 700]
    insts = [_tight(n, 1 + n // 50, 820 + n, demand_max) for n in sizes]
    _check(insts, 12, 16, 4, (16, 32, 1))


@pytest.mark.parametrize("ants", [1, 7, 8, 9, 65, 128, 129, 300])
def test_colony_sizes(ants):
    insts = [_tight(90, 4, 840), _tight(61, 3, 841, 1), _tight(201, 6, 842)]
    _check(insts, ants, 16, 4, (16, 16, 0))
    _check(insts, ants, 24, 3, (32, 8, 1))


def test_many_vehicles_and_single_customer_routes():
    insts = [_tight(120, 70, 860, 3), _tight(100, 100, 861, 1, slack=1.0),
             _tight(64, 33, 862, 100, slack=1.3), _tight(90, 95, 863, 2)]
    _check(insts, 24, 16, 8, (16, 64, 1))
    _check(insts, 24, 20, 8, (32, 32, 1))


def test_large_instances_in_few_ants_at_a_time():
    """Rows that leave no room for every ant's elements, or for the pheromone
    levels, beside them."""
    _check([_tight(790, 9, 870), _tight(640, 8, 871)], 64, 32, 3, (32, 16, 1))
    _check([_tight(2046, 20, 872)], 40, 8, 2, (32, 8, 1))
    _check([_tight(1300, 12, 873, 900000)], 40, 16, 2, (32, 8, 1))
