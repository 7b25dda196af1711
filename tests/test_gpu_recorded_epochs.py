"""Epochs that a caller recorded in a CUDA graph and replays after a set-up of
the same sizes (the recording stays valid while graph_generation does): run()
counts from the epoch they reached, as if they had been enqueued call by
call."""
import numpy as np
import pytest

from vehicleroutingproblem_b200 import instances as I

pytestmark = pytest.mark.gpu

KW = dict(ants=24, cand_k=16)


def _split_epoch(ctx, send, recv):
    ctx.shard_construct(send.data_ptr())
    recv.copy_(send)
    ctx.shard_update(recv.data_ptr(), 1)


@pytest.mark.parametrize("again", ["same instance", "other instance"])
def test_run_after_replayed_split_epochs(native, again):
    import torch
    first = I.uniform_instance(120, 4, 811)
    second = first if again == "same instance" else I.uniform_instance(120, 4, 812)
    s = torch.cuda.Stream()
    with native.Context(0) as ctx, native.Context(0) as ref:
        ctx.set_stream(s.cuda_stream)
        ctx.setup_instance(first, seed=3, **KW)
        P = ctx.shard_packet_ints()
        send = torch.zeros(P, dtype=torch.int32, device="cuda")
        recv = torch.zeros(P, dtype=torch.int32, device="cuda")
        with torch.cuda.stream(s):
            _split_epoch(ctx, send, recv)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s, capture_error_mode="thread_local"):
            _split_epoch(ctx, send, recv)
        generation = ctx.graph_generation()
        for seed in (4, 5):  # the second round: no library call between set-up and replay
            ctx.setup_instance(second, seed=seed, **KW)
            if ctx.graph_generation() != generation:  # the capacity is a launch argument
                generation = ctx.graph_generation()
                with torch.cuda.graph(graph := torch.cuda.CUDAGraph(), stream=s,
                                      capture_error_mode="thread_local"):
                    _split_epoch(ctx, send, recv)
                ctx.setup_instance(second, seed=seed, **KW)
                assert ctx.graph_generation() == generation
            with torch.cuda.stream(s):
                for _ in range(4):
                    graph.replay()
            st = ctx.run(8)
            ref.setup_instance(second, seed=seed, **KW)
            want = ref.run(12)
            assert (st.epochs, st.total_steps) == (12, want.total_steps) and want.epochs == 12
            assert st.global_best == want.global_best and np.array_equal(ctx.tau(), ref.tau())
            assert all(np.array_equal(a, b) for a, b in zip(ctx.best(), ref.best()))
        del graph
