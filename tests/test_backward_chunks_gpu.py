"""GPU parity of the chunked backward pass at the edges of its 64-token chunks, and of its two output forms."""
import pytest
import torch

from avelang_b200 import synth
from gpu_util import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [[1], [63], [64], [65], [129, 0, 1, 64]])
def test_backward_at_chunk_edges(built_lib, checker, lens):
    from avelang_b200 import gdn
    O, _ = checker
    T = sum(lens)
    inp = synth.make_inputs(1, T, 2, 4, 128, 128, seed=71 + T, n_states=len(lens), gate_scale=0.3)
    inp.beta[:, ::5] = 0.0  # masked tokens
    cu = torch.tensor([0] + lens, dtype=torch.int64).cumsum(0).to(torch.int32)
    gen = torch.Generator().manual_seed(72)
    d_o = torch.randn(inp.v.shape, generator=gen).bfloat16()
    d_final = 0.1 * torch.randn(inp.initial_state.shape, generator=gen)
    g = dev(inp)
    args = (g.q, g.k, g.v, g.g, g.beta, d_o.cuda(), inp.scale, g.initial_state, d_final.cuda(), cu.cuda())
    got = gdn.gated_delta_rule_backward(*args)
    # the operator's form: dq and dk per value head, everything in fp32
    f32 = dict(dtype=torch.float32, device="cuda")
    dq, dk, dv = (torch.empty(1, T, 4, 128, **f32) for _ in range(3))
    dg, dbeta, ds0 = torch.empty(1, T, 4, **f32), torch.empty(1, T, 4, **f32), torch.empty_like(g.initial_state)
    torch.ops.avelang_gdn.recurrent_backward(*args[:6], float(inp.scale), *args[7:], dq, dk, dv, dg, dbeta, ds0)
    assert gdn.read_status() == 0
    ref = O.recurrent_grads(inp.q, inp.k, inp.v, inp.g, inp.beta, d_o, inp.scale, inp.initial_state, d_final, cu)
    for name, x, r in zip(("dq", "dk", "dv", "dg", "dbeta", "ds0"), got, ref):
        e = O.rel_l2(x.float().cpu(), r.to(torch.bfloat16).float() if x.dtype == torch.bfloat16 else r)
        assert e <= (1e-3 if x.dtype == torch.bfloat16 else 2e-5), f"{name}: rel-L2 {e:.3e}"
    summed = lambda x: x.view(1, T, 2, 2, 128).sum(3)
    for name, x, r in zip(("dq", "dk", "dv"), (summed(dq), summed(dk), dv), ref):
        e = O.rel_l2(x.cpu(), r)
        assert e <= 2e-5, f"operator {name}: rel-L2 {e:.3e}"
