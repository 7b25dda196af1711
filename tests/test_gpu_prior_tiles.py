"""The prior's tensor-core passes where blocks take several tiles of four rows
(two blocks per SM: from 1185 rows on a B200): one tile, two, three and four of
them per block, last tiles that are not full, against the FP64 oracle with
BF16 rounding at the device's points.  The bounds are those of the one-tile
sizes: FP32 sums in another order move the gradient's norm by no more than
n 2^-24 of it, 2e-4 for the longest sum here, a tenth of the bound."""
import numpy as np
import pytest

from vehicleroutingproblem_b200 import instances as I

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def large(native):
    from oracle import prior_oracle as PO
    insts = [I.uniform_instance(1000, 9, 821), I.clustered_instance(1100, 8, 822),
             I.uniform_instance(900, 7, 823, demand_max=1), I.uniform_instance(997, 6, 824)]
    sols = []
    for j, inst in enumerate(insts):
        with native.Context(0) as c:
            c.setup_instance(inst, ants=32, cand_k=16, seed=80 + j)
            c.run(2)
            nodes, lens, _ = c.best()
            sols.append((nodes, lens))
    pr = native.Prior(0, seed=77)
    cnt = pr.set_dataset(insts, sols, cand_k=32)
    rows = sum(x.n + 1 for x in insts)
    bits, kv, sc = pr.rows(0, rows, scores=True)
    yield pr, cnt, PO.bf16_bits_to_float(bits), kv.astype(np.int64), sc
    pr.close()


@pytest.mark.parametrize("count", [1183, 1184, 1185, 2371, 3552, 3557])
def test_gradient(large, count):
    from oracle import prior_oracle as PO
    pr, cnt, X, kv, _ = large
    ids = np.random.RandomState(count).randint(0, cnt, count).astype(np.int32)
    loss, g = pr.gradient(ids)
    ref_loss, ref = PO.loss_grad(pr.params().astype(np.float64), X, kv, pr.examples()[ids],
                                 mimic=True)
    assert abs(loss - ref_loss) <= 1e-4 * max(1.0, abs(ref_loss))
    assert np.linalg.norm(g - ref) / np.linalg.norm(ref) < 2e-3


def test_scores(large):
    from oracle import prior_oracle as PO
    pr, _, X, kv, sc = large
    ref = PO.forward(pr.params().astype(np.float64), X, kv, mimic=True)
    mask = np.arange(32)[None, :] < kv[:, None]
    assert np.abs(sc - ref)[mask].max() <= 2e-3 * np.abs(ref[mask]).max() + 1e-4
