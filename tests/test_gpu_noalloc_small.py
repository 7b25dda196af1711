"""The allocation-free pheromone update where its one-launch form begins and
ends (customers, routes, no global best), against the context's entry point
on the same inputs, bit for bit."""
import numpy as np
import pytest

from tests.test_gpu_update_edges import _dev
from tests.test_zz_no_alloc import _entry
from vehicleroutingproblem_b200 import _native
from vehicleroutingproblem_b200 import instances as I

pytestmark = pytest.mark.gpu


def _instance(n, K):
    inst = I.uniform_instance(n, K, 950 + n).unit_twin()
    return I.Instance(inst.name, inst.x, inst.y, inst.demand, K, -(-n // K))


@pytest.mark.parametrize("with_global", [True, False])
@pytest.mark.parametrize("n,K", [(1, 1), (3, 3), (16, 16), (17, 17), (90, 12), (384, 16), (385, 16),
                                 (400, 15), (401, 15), (512, 8), (624, 1), (625, 1)])
def test_one_launch_form_equals_context_entry_point(n, K, with_global):
    import torch
    noalloc = _entry()
    tau0 = np.random.RandomState(n + K).randint(0, 256, size=(n + 1) ** 2).astype(np.uint8)
    with _native.Context(0) as ctx:
        ctx.setup_instance(_instance(n, K), ants=16, cand_k=min(n, 20), seed=11)
        ctx.construct(0)
        nodes, lens, cost, feas, _, _ = ctx.ants()
        a, b = 0, ctx.m - 1
        routes = [(nodes[q][:lens[q].sum()].astype(np.int32), lens[q].astype(np.int32))
                  for q in (a, b)]
        dep = [float(np.float32(30.0) / np.float32(cost[a])),
               float(np.float32(70.0) / np.float32(cost[b]))]
        ctx.set_tau(tau0)
        expected = []
        for _ in range(3):
            if with_global:
                ctx.evaporate_deposit(a, dep[0], *routes[1], dep[1])
            else:
                ctx.evaporate_deposit(a, dep[0])
            expected.append(ctx.tau())
    d, *r = _dev(tau0, *routes[0], *routes[1])
    p = [t.data_ptr() for t in r]
    if not with_global:
        p[2:] = [None, None]
    for want in expected:
        assert noalloc(d.data_ptr(), n, K, p[0], p[1], dep[0], p[2], p[3], dep[1], 0.5,
                       torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        assert np.array_equal(d.cpu().numpy(), want)
