"""The backward pass and offset tables that are not monotone inside [0, T]: such a batch is skipped and flagged as a whole, like
in the forward pass, because its chunk records have no places of their own."""
import pytest
import torch

from avelang_b200 import synth
from gpu_util import dev

pytestmark = pytest.mark.gpu


# sequences that overlap, one that goes backwards and others that are valid by themselves, offsets outside [0, T]
@pytest.mark.parametrize("bad", [[0, 200, 100, 300], [150, 300, 0, 150], [0, 100, 5000, 100, 300], [-64, 100, 300], [0, 100, 301]])
def test_backward_rejects_a_bad_offset_table(built_lib, checker, bad):
    from avelang_b200 import gdn
    O, _ = checker
    T, n = 300, len(bad) - 1
    inp = synth.make_inputs(1, T, 1, 2, 128, 128, seed=91, n_states=n, gate_scale=0.3)
    d_o = torch.randn(inp.v.shape, generator=torch.Generator().manual_seed(92)).bfloat16()
    g = dev(inp)
    mark = 123.0
    f32 = dict(dtype=torch.float32, device="cuda")
    outs = [torch.full(s, mark, **f32) for s in ((1, T, 2, 128),) * 3 + ((1, T, 2),) * 2 + (tuple(g.initial_state.shape),)]
    run = lambda cu: torch.ops.avelang_gdn.recurrent_backward(g.q, g.k, g.v, g.g, g.beta, d_o.cuda(), float(inp.scale), g.initial_state, None,
                                                              torch.tensor(cu, dtype=torch.int32, device="cuda"), *outs)
    run(bad)
    assert gdn.read_status() == 2  # AVE_GDN_DEV_BAD_SEQLEN
    for x in outs:
        assert bool((x == mark).all()), "a rejected batch leaves its outputs alone"
    good = [0] + [T * (i + 1) // n for i in range(n)]
    run(good)
    assert gdn.read_status() == 0
    ref = O.recurrent_grads(inp.q, inp.k, inp.v, inp.g, inp.beta, d_o, inp.scale, inp.initial_state, None, torch.tensor(good, dtype=torch.int32))
    dq, dk, dv, dg, dbeta, ds0 = outs
    for name, x, r in zip(("dq", "dk", "dv", "dg", "dbeta", "ds0"), (dq.sum(2, keepdim=True), dk.sum(2, keepdim=True), dv, dg, dbeta, ds0), ref):
        e = O.rel_l2(x.cpu(), r)
        assert e <= 2e-5, f"{name}: rel-L2 {e:.3e}"  # as in the test of the chunk edges
