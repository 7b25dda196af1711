"""The construction's per-node elements against the oracle, ant by ant: the
element types at the ends of their demand ranges (1, 2 and 4 bytes), instance
sizes around the 16-byte pieces, the node pairs and the batches of the full
scan, candidate lists shorter than a warp, every table layout, tight
capacities (repair of many vehicles) and the bitmap form (many ants of a
large instance).  Routes, lengths, costs and draws are equal exactly."""
import numpy as np
import pytest

from tests.test_gpu_parity import check_construct, make_ctx, random_tau
from vehicleroutingproblem_b200 import _native
from vehicleroutingproblem_b200 import instances as I

pytestmark = pytest.mark.gpu


def _instance(n, K, demand_max, seed, slack=1.0):
    inst = I.uniform_instance(n, K, seed, demand_max=max(2, demand_max))
    inst.demand[1 + seed % n] = demand_max
    inst.demand[1:] = np.minimum(inst.demand[1:], demand_max)
    cap = int(np.ceil(inst.demand.sum() / K * slack))
    return I.Instance(inst.name, inst.x, inst.y, inst.demand, K, max(cap, demand_max))


@pytest.mark.parametrize("layout", [_native.LAYOUT_SMEM_WEIGHTS, _native.LAYOUT_SMEM_PACKED,
                                    _native.LAYOUT_GLOBAL])
@pytest.mark.parametrize("demand_max", [1, 254, 255, 65534, 65535, 1000000])
def test_element_types(oracle_mod, demand_max, layout):
    for n, K, k in [(15, 2, 8), (16, 3, 16), (257, 5, 20), (600, 9, 32)]:
        inst = _instance(n, K, demand_max, 31 + n, slack=1.02)
        with make_ctx(inst, k, 24, seed=5) as ctx:
            tau = random_tau(n, 3)
            ctx.set_tau(tau)
            ctx.construct(1, layout)
            check_construct(oracle_mod, inst, ctx, 5, 1, tau)


@pytest.mark.parametrize("n,K", [(1, 1), (2, 1), (30, 31), (31, 2), (32, 4), (33, 33), (63, 5),
                                 (64, 5), (127, 40), (128, 6), (255, 70), (256, 8), (511, 9),
                                 (512, 10), (513, 11), (1023, 12), (1024, 13)])
def test_sizes(oracle_mod, n, K):
    inst = _instance(n, K, 90, 700 + n, slack=1.01)
    with make_ctx(inst, min(n, 11 + n % 22), 16, seed=8) as ctx:
        tau = random_tau(n, 4, "mostly_init")
        ctx.set_tau(tau)
        ctx.construct(2)
        check_construct(oracle_mod, inst, ctx, 8, 2, tau)


def test_bitmap_form(oracle_mod):
    """15 ants per block of a 16000-customer instance: their elements do not
    fit in shared memory together, so the block keeps bitmaps."""
    inst = I.uniform_instance(16000, 16, 661)
    with make_ctx(inst, 16, 148 * 15, seed=3) as ctx:
        assert ctx.plan()["smem"] < 64 * 1024
        tau = ctx.tau()
        ctx.construct(0)
        check_construct(oracle_mod, inst, ctx, 3, 0, tau, ants=(0, 1, 1109, 2219))
