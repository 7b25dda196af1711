"""The pheromone updates on caller-owned memory at sizes around their tiles,
with more routes than threads of a block, and recorded in a CUDA graph (their
launches overlap programmatically) against the same calls made one by one."""
import numpy as np
import pytest

from tests.test_zz_no_alloc import _entry
from vehicleroutingproblem_b200 import _native

pytestmark = pytest.mark.gpu


def _routes(n, K, seed):
    rs = np.random.RandomState(seed)
    perm = rs.permutation(n) + 1
    parts = np.split(perm, np.sort(rs.randint(0, n + 1, size=K - 1)))
    nodes = np.concatenate([np.concatenate([[0], p, [0]]) for p in parts]).astype(np.int32)
    return nodes, np.array([len(p) + 2 for p in parts], np.int32)


def _dev(*arrays):
    import torch
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]


@pytest.mark.parametrize("n,K", [(1, 1), (2, 2), (18, 3), (19, 40), (30, 5), (31, 2), (63, 7),
                                 (89, 90), (127, 3), (355, 6), (356, 500), (700, 4000)])
def test_seq_update_edges(oracle_mod, n, K):
    import torch
    L = _native.load()
    it, gb = _routes(n, K, n), _routes(n, K, n + 1)
    tau = np.random.RandomState(n).uniform(0.01, 2.0, size=(n + 1) ** 2)
    d = _dev(tau, *it, *gb)
    scratch = torch.zeros(L.aco_b200_seq_update_scratch_bytes(n), dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    expected = tau
    for reset in (0, 1):
        expected = oracle_mod.seq_pheromone_update(expected, n, *it, 0.3, *gb, 0.7, 0.1, 0.05, 1.5,
                                                   reset, 1.0)
        rc = L.aco_b200_seq_pheromone_update(
            d[0].data_ptr(), n, K, d[1].data_ptr(), d[2].data_ptr(), 0.3, d[3].data_ptr(),
            d[4].data_ptr(), 0.7, 0.1, 0.05, 1.5, reset, 1.0, scratch.data_ptr(), stream)
        assert rc == 0
        torch.cuda.synchronize()
        assert np.array_equal(d[0].cpu().numpy().view(np.uint64),
                              np.asarray(expected).view(np.uint64))
        assert int(scratch.sum()) == 0


@pytest.mark.parametrize("n,K", [(3, 2), (89, 5), (90, 91), (127, 8), (500, 700)])
def test_graph_replays_equal_calls(n, K):
    import torch
    L, noalloc = _native.load(), _entry()
    it, gb = _routes(n, K, n), _routes(n, K, n + 1)
    rs = np.random.RandomState(n)
    t8, t64 = rs.randint(0, 256, (n + 1) ** 2).astype(np.uint8), rs.uniform(0.01, 2, (n + 1) ** 2)
    d8, d64, *d = _dev(t8, t64, *it, *gb)
    p = [x.data_ptr() for x in d]
    scratch = torch.zeros(L.aco_b200_seq_update_scratch_bytes(n), dtype=torch.uint8, device="cuda")

    def both(stream):
        assert noalloc(d8.data_ptr(), n, K, p[0], p[1], 30.0, p[2], p[3], 70.0, 0.1, stream) == 0
        assert L.aco_b200_seq_pheromone_update(d64.data_ptr(), n, K, p[0], p[1], 0.3, p[2], p[3],
                                               0.7, 0.1, 0.05, 1.5, 0, 1.0, scratch.data_ptr(),
                                               stream) == 0

    for _ in range(3):
        both(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    want8, want64 = d8.cpu().numpy(), d64.cpu().numpy()
    d8.copy_(torch.from_numpy(t8))
    d64.copy_(torch.from_numpy(t64))
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        both(torch.cuda.current_stream().cuda_stream)
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(d8.cpu().numpy(), want8)
    assert np.array_equal(d64.cpu().numpy().view(np.uint64), want64.view(np.uint64))
