"""A batch without tokens: no kernel runs, the states and their gradients pass through."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("packed", [False, True])
def test_states_pass_through(built_lib, d, packed):
    from avelang_b200 import gdn
    n = 3
    qk, v = (torch.zeros(1 if packed else n, 0, h, d, dtype=torch.bfloat16, device="cuda") for h in (2, 4))
    gb = torch.zeros(*v.shape[:3], device="cuda")
    cu = torch.zeros(n + 1, dtype=torch.int32, device="cuda") if packed else None
    s0 = torch.randn(n, 4, d, d, device="cuda")
    junk = [torch.full_like(s0, float("nan")) for _ in range(4)]  # what a fresh buffer would hold
    del junk
    for fn in (gdn.chunk_gated_delta_rule, gdn.fused_recurrent_gated_delta_rule):
        o, s = fn(qk, qk, v, gb, gb, initial_state=s0, output_final_state=True, cu_seqlens=cu)
        assert o.shape == v.shape and torch.equal(s, s0) and s.data_ptr() != s0.data_ptr()
        _, s = fn(qk, qk, v, gb, gb, output_final_state=True, cu_seqlens=cu)
        assert s.shape == s0.shape and not bool(s.any())
    if d == 128:
        ds = torch.randn_like(s0)
        assert torch.equal(gdn.gated_delta_rule_backward(qk, qk, v, gb, gb, v, None, s0, ds, cu)[5], ds)
        assert not bool(gdn.gated_delta_rule_backward(qk, qk, v, gb, gb, v, None, s0, None, cu)[5].any())
    assert gdn.read_status() == 0
