"""GPU parity of the d = 64 prefill at the edges of its chunks, with every option, to fp32 accuracy of the states."""
import pytest
import torch

from avelang_b200 import synth
from gpu_util import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [[1], [63], [64], [65], [256], [130, 0, 1, 64, 300]])
@pytest.mark.parametrize("gate_scale", [1.0, 0.02])
@pytest.mark.parametrize("gated", [False, True])
def test_d64_prefill(built_lib, checker, lens, gate_scale, gated):
    from avelang_b200 import gdn
    O, C = checker
    T, n = sum(lens), len(lens)
    inp = synth.make_inputs(1, T, 2, 4, 64, 64, seed=81 + T, with_z=gated, n_states=n + 1, gate_scale=gate_scale, l2norm=False)
    cu = torch.tensor([0] + lens, dtype=torch.int64).cumsum(0).to(torch.int32)
    idx = torch.arange(n, dtype=torch.int32).flip(0).contiguous()
    if n > 1:
        idx[0] = -1  # skipped: zero output, state untouched
    g = dev(inp)
    pool = g.initial_state.clone()
    o, final = gdn.chunk_gated_delta_rule(g.q, g.k, g.v, g.g, g.beta, initial_state=pool, output_final_state=True, use_qk_l2norm_in_kernel=True,
                                          cu_seqlens=cu.cuda(), z=g.z, state_indices=idx.cuda())
    assert gdn.read_status() == 0 and final.data_ptr() == pool.data_ptr()
    unit = lambda x: x.double() * torch.rsqrt(x.double().pow(2).sum(-1, keepdim=True) + 1e-6)
    s0 = inp.initial_state[idx.clamp_min(0).long()]
    o_ref, s_ref = O.naive_recurrent_gated_delta_rule(unit(inp.q), unit(inp.k), inp.v.double(), inp.g.double(), inp.beta.double(), inp.scale,
                                                      s0.double(), cu)
    if gated:
        o_ref = O.gated_rmsnorm(o_ref, inp.z)
    for i in range(n):
        a, b = int(cu[i]), int(cu[i + 1])
        if int(idx[i]) < 0:
            assert not bool(o[0, a:b].any())
            continue
        assert O.rel_l2(final[idx[i].item()].cpu(), s_ref[i]) <= 2e-6
        if b > a:
            assert O.rel_l2(o[0, a:b].float().cpu(), o_ref[0, a:b].to(torch.bfloat16).float()) <= 3e-4
    assert torch.equal(final[n].cpu(), inp.initial_state[n])  # a slot nobody names
