"""The first kernel of a call is launched so that it can be resident before the work in front of it has finished: whatever
that work is, the call must see its results (weights included), eagerly and in a captured graph."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 4, 16])
def test_call_sees_what_was_enqueued_in_front_of_it(B):
    import ezops_b200 as ez
    from ezops_b200 import _lib
    from ezops_b200 import workloads as wl

    sh, S = wl.QWEN3_0_6B, 300
    args = [t.cuda() for t in wl.decode_layer_inputs(sh, B, S)]
    op = ez.Qwen3DenseDecodeOp(B, S, sh.hidden, sh.inter, sh.num_heads, sh.head_dim, backend="cuda", num_kv_heads=sh.num_kv_heads)
    want = op(*args).clone()
    keep = [t.clone() for t in args]
    side, filler = torch.cuda.Stream(), torch.empty(1 << 22, device="cuda")

    def calls():
        outs = []
        for i in (0, 1, 3, 6):  # hidden, keys, and the weights of the first and of the last projection
            args[i].zero_()
            args[i].copy_(keep[i])
            outs.append(op(*args))
        filler.zero_()
        outs.append(op(*args))
        outs.append(op(*args))  # directly behind another call
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            args[0].fill_(0.5)
            args[0].copy_(keep[0])
        torch.cuda.current_stream().wait_stream(side)
        outs.append(op(*args))
        return outs

    for _ in range(5):
        assert all(torch.equal(o, want) for o in calls())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outs = calls()
    for _ in range(5):
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(o, want) for o in outs)
    assert _lib.device_status() == 0
