"""The batched solver where the ants' elements leave no room for the whole
colony and bitmaps take their place: the same routes as the single-instance
solver, with demands of every size, partial warps, tight capacities (repairs
of few and of many customers) and small instances beside large ones."""
import pytest

from tests.test_gpu_batch_shapes import _check, _tight

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,ants,demand_max", [
    (2046, 8, 128, 1), (2046, 8, 65, 254), (2017, 12, 61, 255), (1990, 12, 60, 65535),
    (1000, 16, 71, 900000), (992, 16, 65, 65534), (793, 32, 61, 900000), (640, 32, 64, 65535)])
def test_bitmaps_equal_single_instance_solver(n, k, ants, demand_max):
    insts = [_tight(n, 2 + n // 70, 880, demand_max),
             _tight(n - 31, 2 + n // 300, 881, demand_max, slack=1.005),
             _tight(max(k, 33), 2, 882, demand_max), _tight(130, 41, 883, demand_max)]
    _check(insts, ants, k, 3, (32, 8, 1))
