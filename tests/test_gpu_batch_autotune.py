"""The batch's autotuner: a solve per queue order, and no choice among shapes
whose launches are the same."""
import pytest

from vehicleroutingproblem_b200 import _native
from vehicleroutingproblem_b200 import instances as I

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,shape", [(16, (16, 32, 1)), (16, (32, 8, 0)), (32, (32, 16, 1))])
def test_shapes_of_one_order_share_their_time(k, shape):
    insts = I.batched_instances(24, seed0=31000)
    with _native.Batch(0) as b:
        b.setup(insts, ants=32, cand_k=k, seed=9, epochs=6)
        b.set_tuning(*shape)
        chosen, ms = b.autotune(trial_epochs=2)
        orders = [1] * (6 if k <= 16 else 3) + [0] * (2 if k <= 16 else 1)
        assert len(ms) == len(orders) and (ms > 0).all()
        times = {o: {float(t) for t, q in zip(ms, orders) if q == o} for o in (0, 1)}
        assert len(times[0]) == len(times[1]) == 1
        assert chosen == b.tuning() and chosen[:2] == shape[:2]
        assert times[chosen[2]] == {float(ms.min())}
