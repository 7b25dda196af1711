"""Candidate and fallback lists where their construction can go wrong: points
on few places (many equal distances, zero distances), dense clusters beside an
almost empty plane (the second tier's collection bound far off at first),
sizes around the groups of four times 32 nodes, against the oracle's order."""
import numpy as np
import pytest

from vehicleroutingproblem_b200 import _native
from vehicleroutingproblem_b200 import instances as I

pytestmark = pytest.mark.gpu


def _places(n, places, seed):
    inst = I.uniform_instance(n, 5, seed)
    rs = np.random.RandomState(seed)
    at = rs.randint(0, 1001, size=(places, 2)).astype(np.float32)
    pick = rs.randint(0, places, size=n + 1)
    inst.x[:], inst.y[:] = at[pick, 0], at[pick, 1]
    return inst


def _outliers(n, far, seed):
    inst = I.uniform_instance(n, 5, seed)
    inst.x[far + 1:] = 500 + inst.x[far + 1:] // 100
    inst.y[far + 1:] = 500 + inst.y[far + 1:] // 100
    return inst


CASES = {
    "one_place": lambda: _places(1600, 1, 1), "three_places": lambda: _places(1700, 3, 2),
    "line": lambda: _places(1536, 400, 3), "outliers": lambda: _outliers(2000, 40, 4),
    "half_out": lambda: _outliers(1800, 900, 5), "clustered": lambda: I.clustered_instance(3001, 9, 6),
    "n1500": lambda: I.uniform_instance(1500, 5, 7), "n1499": lambda: I.uniform_instance(1499, 5, 7),
    "n127": lambda: I.uniform_instance(127, 3, 8), "n128": lambda: I.uniform_instance(128, 3, 8),
    "n129": lambda: I.uniform_instance(129, 3, 8), "n5": lambda: I.uniform_instance(5, 2, 9),
    "n97": lambda: I.uniform_instance(97, 2, 9),
}


@pytest.mark.parametrize("k", [1, 17, 32])
@pytest.mark.parametrize("name", list(CASES))
def test_lists_follow_the_order(oracle_mod, name, k):
    inst = CASES[name]()
    n = inst.n
    with _native.Context(0) as ctx:
        ctx.setup_instance(inst, ants=2, cand_k=k)
        kk = ctx.k
        want = oracle_mod.knn(inst.x, inst.y, kk + 256).reshape(n + 1, kk + 256)
        assert np.array_equal(ctx.candidates()[0].reshape(n + 1, kk), want[:, :kk])
        assert np.array_equal(ctx.tier().reshape(n + 1, 64), want[:, kk:kk + 64])
        if n >= 1500:
            assert np.array_equal(ctx.tier2().reshape(n + 1, 192), want[:, kk + 64:])
