"""The scratch of the prefill and of the backward pass: one block per call in flight, a graph's own in a graph, given back when
the allocator needs it."""
import threading

import pytest
import torch

from avelang_b200 import synth
from gpu_util import dev

pytestmark = pytest.mark.gpu


def test_two_threads_on_one_stream(built_lib):
    """Both threads enqueue on the default stream: a call of several launches must not find another call's records."""
    from avelang_b200 import gdn
    work = []
    for seed, T in ((1, 900), (2, 200)):
        b = dev(synth.make_inputs(1, T, 2, 4, 128, 128, seed=seed, gate_scale=0.3))
        p = dev(synth.make_inputs(1, T, 2, 4, 64, 64, seed=seed, gate_scale=0.3))
        d_o = torch.randn_like(b.v)
        def run(b=b, p=p, d_o=d_o):
            return (*gdn.gated_delta_rule_backward(b.q, b.k, b.v, b.g, b.beta, d_o)[:5],
                    *gdn.chunk_gated_delta_rule(p.q, p.k, p.v, p.g, p.beta, output_final_state=True))
        work.append((run, run()))
    torch.cuda.synchronize()
    wrong, go = [], threading.Barrier(2)

    def loop(run, want):
        go.wait()
        for _ in range(40):
            for x, y in zip(run(), want):
                if not torch.equal(x, y):
                    wrong.append(x.shape)

    threads = [threading.Thread(target=loop, args=w) for w in work]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not wrong and gdn.read_status() == 0


def test_a_graph_keeps_its_scratch(built_lib):
    """A captured call, then a larger one on the same stream, then tensors that take what that leaves: replays still give the
    same result and write into none of the tensors."""
    from avelang_b200 import gdn
    small = dev(synth.make_inputs(1, 500, 2, 4, 128, 128, seed=3))
    large = dev(synth.make_inputs(1, 4000, 2, 4, 128, 128, seed=4))
    run = lambda g, out: gdn.chunk_gated_delta_rule(g.q, g.k, g.v, g.g, g.beta, out=out)
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st):
        out, want = torch.empty_like(small.v), torch.empty_like(small.v)
        run(small, want)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            run(small, out)
        run(large, torch.empty_like(large.v))
        held, reserved = [], torch.cuda.memory_reserved()
        while torch.cuda.memory_reserved() == reserved and len(held) < 4096:  # until no freed block is left to hand out
            held.append(torch.zeros(1 << 20, device="cuda"))
        out.zero_()
        graph.replay()
        assert torch.equal(out, want)
        assert not any(bool(t.any()) for t in held)
    st.synchronize()


def test_scratch_goes_back_when_memory_is_short(built_lib):
    from avelang_b200 import gdn
    g = dev(synth.make_inputs(1, 2048, 8, 16, 128, 128, seed=5))
    d_o = torch.randn_like(g.v)
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):  # no earlier call has left scratch here
        before = torch.cuda.memory_allocated()
        gdn.gated_delta_rule_backward(g.q, g.k, g.v, g.g, g.beta, d_o)  # takes about 140 MB
        kept = torch.cuda.memory_allocated() - before
        assert kept > 100 << 20, "the scratch stays for the next call"
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        total = torch.cuda.get_device_properties(0).total_memory
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (64 << 20)) / total)
        try:
            x = torch.zeros(kept + (32 << 20), dtype=torch.uint8, device="cuda")  # fits only if the scratch makes room
        finally:
            torch.cuda.set_per_process_memory_fraction(1.0)
        assert torch.cuda.memory_allocated() - before <= x.numel() + (2 << 20)
