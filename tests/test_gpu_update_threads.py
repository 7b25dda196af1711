"""The FP64 pheromone update from two host threads at once, each on a stream
and a matrix of its own, with different numbers of routes that both need more
shared memory for their offsets than a launch has by default."""
import threading

import numpy as np
import pytest

from tests.test_gpu_update_edges import _dev, _routes
from vehicleroutingproblem_b200 import _native

pytestmark = pytest.mark.gpu

CALLS = 400


def test_two_threads_with_many_routes(oracle_mod):
    import torch
    L, n = _native.load(), 50
    jobs = []
    for K in (6144, 8192):
        it, gb = _routes(n, K, K), _routes(n, K, K + 1)
        tau = np.random.RandomState(K).uniform(0.01, 2.0, size=(n + 1) ** 2)
        scratch = torch.zeros(L.aco_b200_seq_update_scratch_bytes(n), dtype=torch.uint8,
                              device="cuda")
        jobs.append(dict(K=K, it=it, gb=gb, tau=tau, dev=_dev(tau, *it, *gb), scratch=scratch,
                         stream=torch.cuda.Stream(), rcs=[]))
    torch.cuda.synchronize()
    start = threading.Barrier(len(jobs))

    def work(j):
        torch.cuda.set_device(0)
        p = [t.data_ptr() for t in j["dev"]]
        start.wait()
        for _ in range(CALLS):
            j["rcs"].append(L.aco_b200_seq_pheromone_update(
                p[0], n, j["K"], p[1], p[2], 0.3, p[3], p[4], 0.7, 0.1, 0.05, 1.5, 0, 1.0,
                j["scratch"].data_ptr(), j["stream"].cuda_stream))

    threads = [threading.Thread(target=work, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for j in jobs:
        assert j["rcs"] == [0] * CALLS
        assert int(j["scratch"].sum()) == 0
        want = j["tau"]
        for _ in range(CALLS):
            want = oracle_mod.seq_pheromone_update(want, n, *j["it"], 0.3, *j["gb"], 0.7, 0.1,
                                                   0.05, 1.5, 0, 1.0)
        got = j["dev"][0].cpu().numpy()
        assert np.array_equal(got.view(np.uint64), np.asarray(want).view(np.uint64))
