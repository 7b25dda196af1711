"""The fallback's lists where the collection of their keys starts again or
ends early: clumps of customers smaller than the lists with empty space around
them, and many customers at one place, against the oracle's order."""
import numpy as np
import pytest

from vehicleroutingproblem_b200 import _native
from vehicleroutingproblem_b200 import instances as I

pytestmark = pytest.mark.gpu


def _clumps(n, size, width, seed):
    """n customers, `size` to a clump; width 0: all at its place."""
    inst = I.uniform_instance(n, 5, seed)
    rs = np.random.RandomState(seed)
    at = rs.uniform(0, 1000, size=(n // size + 2, 2))
    off = rs.uniform(-1, 1, size=(n + 1, 2)) * width
    pick = rs.permutation(n + 1) // size
    inst.x[:], inst.y[:] = (at[pick] + off).astype(np.float32).T
    return inst


@pytest.mark.parametrize("k", [1, 8, 32])
@pytest.mark.parametrize("n,size,width", [(1500, 33, 0.2), (2500, 40, 0.2), (2500, 100, 1e-3),
                                          (3000, 200, 0.2), (2200, 288, 0.1), (2200, 289, 0.1),
                                          (2500, 60, 0.0), (2500, 256, 0.0), (2500, 289, 0.0),
                                          (3000, 447, 0.0), (3000, 600, 0.0), (1500, 1600, 0.0)])
def test_lists_of_clumped_customers(oracle_mod, n, size, width, k):
    inst = _clumps(n, size, width, n + size)
    with _native.Context(0) as ctx:
        ctx.setup_instance(inst, ants=2, cand_k=k)
        want = oracle_mod.knn(inst.x, inst.y, k + 256).reshape(n + 1, k + 256)
        assert np.array_equal(ctx.candidates()[0].reshape(n + 1, k), want[:, :k])
        assert np.array_equal(ctx.tier().reshape(n + 1, 64), want[:, k:k + 64])
        assert np.array_equal(ctx.tier2().reshape(n + 1, 192), want[:, k + 64:])
