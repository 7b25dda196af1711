"""The construction where its tables leave little shared memory: the sizes a
table layout can be forced for (up to the last one, and not beyond), and the
plans with bitmaps in place of per-node elements.  Routes, lengths, costs and
draws equal those of the rows read from global memory, and the oracle's."""
import numpy as np
import pytest

from tests.test_gpu_parity import check_construct, make_ctx, random_tau
from vehicleroutingproblem_b200 import _native as N
from vehicleroutingproblem_b200 import instances as I

pytestmark = pytest.mark.gpu

WEIGHTS, PACKED, GLOBAL = N.LAYOUT_SMEM_WEIGHTS, N.LAYOUT_SMEM_PACKED, N.LAYOUT_GLOBAL


def _instance(n, K, demand_max, slack=1.01):
    inst = I.uniform_instance(n, K, 900 + n, demand_max=max(2, demand_max))
    inst.demand[1:] = np.minimum(inst.demand[1:], demand_max)
    inst.demand[n] = demand_max
    cap = max(int(np.ceil(inst.demand.sum() / K * slack)), demand_max)
    return I.Instance(inst.name, inst.x, inst.y, inst.demand, K, cap)


def _same_ants(a, b):
    for x, y, lens in zip(a[0], b[0], a[1]):
        assert np.array_equal(x[:lens.sum()], y[:lens.sum()])
    assert all(np.array_equal(x, y) for x, y in zip(a[1:], b[1:]))


@pytest.mark.parametrize("n,layout", [(1152, WEIGHTS), (1153, WEIGHTS), (1157, WEIGHTS),
                                      (1158, WEIGHTS), (2197, PACKED), (2198, PACKED),
                                      (2215, PACKED), (2216, PACKED)])
def test_forced_layouts_up_to_their_last_size(n, layout):
    with make_ctx(_instance(n, 9, 1), 32, 128, seed=4) as ctx:
        ctx.set_tau(random_tau(n, 5, "mostly_init"))
        ctx.construct(1, GLOBAL)
        want = ctx.ants()
        ctx.construct(1, layout)
        _same_ants(ctx.ants(), want)


@pytest.mark.parametrize("n,layout", [(1159, WEIGHTS), (2217, PACKED)])
def test_forced_layouts_beyond_are_refused(n, layout):
    with make_ctx(_instance(n, 9, 1), 32, 128, seed=4) as ctx:
        with pytest.raises(N.AcoError) as err:
            ctx.construct(1, layout)
        assert err.value.status == N.ACO_ERR_INVALID_INPUT


@pytest.mark.parametrize("depot_rule", [0, 1])
@pytest.mark.parametrize("n,K,k,m,demand_max,layout",
                         [(2198, 20, 32, 128, 1, PACKED), (2100, 17, 32, 700, 1, PACKED),
                          (1860, 15, 32, 2368, 1, PACKED), (2119, 18, 32, 400, 255, PACKED),
                          (2000, 16, 32, 1024, 255, PACKED), (1990, 40, 32, 400, 65535, PACKED),
                          (3901, 30, 16, 1024, 1000, PACKED), (1860, 15, 32, 2368, 100, GLOBAL),
                          (6144, 30, 9, 300, 100, GLOBAL), (16000, 20, 8, 2368, 1, GLOBAL)])
def test_bitmaps_in_place_of_elements(oracle_mod, n, K, k, m, demand_max, layout, depot_rule):
    inst = _instance(n, K, demand_max)
    with make_ctx(inst, k, m, seed=6, depot_rule=depot_rule) as ctx:
        assert ctx.plan()["layout"] == layout
        tau = random_tau(n, 8, "mostly_init")
        ctx.set_tau(tau)
        ctx.construct(2)
        got = ctx.ants()
        if layout != GLOBAL:
            ctx.construct(2, GLOBAL)
            _same_ants(got, ctx.ants())
        if depot_rule == 0:
            check_construct(oracle_mod, inst, ctx, 6, 2, tau, ants=(0, m // 2, m - 1))
