"""GPU parity of the backward pass in the numbers of value heads a key head has, and where a CTA of the gradient launch takes several
(chunk, key head) pairs one after the other (it has 148 CTAs, one a multiprocessor)."""
from types import SimpleNamespace

import pytest
import torch

from avelang_b200 import synth
from gpu_util import dev

pytestmark = pytest.mark.gpu
NAMES = ("dq", "dk", "dv", "dg", "dbeta", "ds0")


def _both_forms(gdn, g, d_o, ds, cu):
    """The public call (bf16, summed over the value heads of a key head) and the operator's fp32 form, per value head."""
    args = (g.q, g.k, g.v, g.g, g.beta, d_o, float(g.scale), g.initial_state, ds, cu)
    f32 = lambda like, *s: torch.empty(*s, dtype=torch.float32, device="cuda") if s else torch.empty_like(like, dtype=torch.float32)
    B, T, Hv = g.g.shape
    per_head = [f32(None, B, T, Hv, 128) for _ in range(3)] + [f32(g.g), f32(g.g), f32(g.initial_state)]
    torch.ops.avelang_gdn.recurrent_backward(*args, *per_head)
    return gdn.gated_delta_rule_backward(*args), per_head


def _check(O, got, per_head, ref, ratio):
    for name, x, r in zip(NAMES, got, ref):
        bf16 = x.dtype == torch.bfloat16
        e = O.rel_l2(x.float().cpu(), r.to(torch.bfloat16).float() if bf16 else r)
        assert e <= (1e-3 if bf16 else 2e-5), f"{name}: rel-L2 {e:.3e}"  # as in the test of the chunk edges
    B, T, Hv, d = per_head[0].shape
    for name, x, r in zip(NAMES, per_head, ref):
        x = x.cpu().view(B, T, Hv // ratio, ratio, d).sum(3) if name in ("dq", "dk") else x.cpu()
        e = O.rel_l2(x, r)
        assert e <= 2e-5, f"operator {name}: rel-L2 {e:.3e}"


@pytest.mark.parametrize("ratio", [1, 3, 4])
def test_value_heads_per_key_head(built_lib, checker, ratio):
    from avelang_b200 import gdn
    O, _ = checker
    inp = synth.make_inputs(1, 131, 2, 2 * ratio, 128, 128, seed=111, n_states=2, gate_scale=0.3)
    cu = torch.tensor([0, 66, 131], dtype=torch.int32)
    gen = torch.Generator().manual_seed(112)
    d_o = torch.randn(inp.v.shape, generator=gen).bfloat16()
    ds = 0.1 * torch.randn(inp.initial_state.shape, generator=gen)
    got, per_head = _both_forms(gdn, dev(inp), d_o.cuda(), ds.cuda(), cu.cuda())
    assert gdn.read_status() == 0
    _check(O, got, per_head, O.recurrent_grads(inp.q, inp.k, inp.v, inp.g, inp.beta, d_o, inp.scale, inp.initial_state, ds, cu), ratio)


@pytest.mark.parametrize("ratio", [1, 2])
def test_several_pairs_a_cta(built_lib, checker, ratio):
    """Twelve ragged sequences x 16 key heads: 500 pairs and more, three or four to a CTA.  Every sequence must come out as it does
    alone, where no CTA has a second pair; the first, a middle and the last one are held against the oracle."""
    from avelang_b200 import gdn
    O, _ = checker
    Hk, lens = 16, [130, 64, 1, 200, 65, 127, 190, 128, 63, 129, 256, 70]
    n, Hv = len(lens), Hk * ratio
    cu = torch.tensor([0] + lens, dtype=torch.int64).cumsum(0).to(torch.int32)
    T = int(cu[-1])
    inp = synth.make_inputs(1, T, Hk, Hv, 128, 128, seed=113, n_states=n, gate_scale=0.3)
    assert sum((x + 63) // 64 for x in lens) * Hk > 3 * 148
    gen = torch.Generator().manual_seed(114)
    d_o = torch.randn(inp.v.shape, generator=gen).bfloat16()
    ds = 0.1 * torch.randn(inp.initial_state.shape, generator=gen)
    g = dev(inp)
    got, per_head = _both_forms(gdn, g, d_o.cuda(), ds.cuda(), cu.cuda())
    assert gdn.read_status() == 0
    for i in range(n):
        a, b = int(cu[i]), int(cu[i + 1])
        one = SimpleNamespace(**{k: getattr(g, k)[:, a:b].contiguous() for k in ("q", "k", "v", "g", "beta")}, scale=g.scale,
                              initial_state=g.initial_state[i:i + 1].contiguous())
        forms = _both_forms(gdn, one, d_o[:, a:b].contiguous().cuda(), ds[i:i + 1].cuda(), None)
        for form, whole in zip(forms, (got, per_head)):
            for name, x, y in zip(NAMES, form, whole):
                assert torch.equal(x, y[i:i + 1] if name == "ds0" else y[:, a:b]), f"sequence {i}: {name}"
        if i in (0, 5, n - 1):
            ref = O.recurrent_grads(inp.q[:, a:b], inp.k[:, a:b], inp.v[:, a:b], inp.g[:, a:b], inp.beta[:, a:b], d_o[:, a:b], inp.scale,
                                    inp.initial_state[i:i + 1], ds[i:i + 1])
            _check(O, *forms, ref, ratio)
