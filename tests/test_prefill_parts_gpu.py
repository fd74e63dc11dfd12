"""GPU parity of the prefill where its schedule or its grouping of heads changes: nine to sixteen parallel parts, and value heads per key
head that do not come in pairs (pass 1 takes two a CTA)."""
import pytest
import torch

from avelang_b200 import synth
from gpu_util import check_o, check_s, dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hk, Hv, T", [(2, 4, 64 * 128), (2, 4, 64 * 140 + 1), (4, 8, 64 * 130 - 1)])  # 16, 16 and 9 parts
@pytest.mark.parametrize("gate_scale, with_z", [(1.0, True), (0.01, False), (0.001, True)])
def test_more_than_eight_parts(built_lib, checker, Hk, Hv, T, gate_scale, with_z):
    from avelang_b200 import gdn
    O, C = checker
    inp = synth.make_inputs(1, T, Hk, Hv, 128, 128, seed=101, with_z=with_z, n_states=1, gate_scale=gate_scale)
    g = dev(inp)
    o, s = gdn.chunk_gated_delta_rule(g.q, g.k, g.v, g.g, g.beta, initial_state=g.initial_state, output_final_state=True, z=g.z)
    assert gdn.read_status() == 0
    o_ref, s_ref = C.recurrent(inp.q, inp.k, inp.v, inp.g, inp.beta, inp.scale, inp.initial_state)
    if with_z:
        o_ref = O.gated_rmsnorm(o_ref, inp.z)
    for t0 in range(0, T, 256):  # half a part at a time, so that one wrong part cannot hide in the total
        check_o(O, o[:, t0:t0 + 256], o_ref[:, t0:t0 + 256])
    check_s(O, s, s_ref)


@pytest.mark.parametrize("ratio", [1, 3, 5])
@pytest.mark.parametrize("T", [200, 64 * 40 + 3])  # whole chains, and parts
def test_value_heads_per_key_head(built_lib, checker, ratio, T):
    from avelang_b200 import gdn
    O, C = checker
    inp = synth.make_inputs(1, T, 2, 2 * ratio, 128, 128, seed=103, with_z=True, n_states=1, gate_scale=0.05, l2norm=False)
    g = dev(inp)
    o, s = gdn.chunk_gated_delta_rule(g.q, g.k, g.v, g.g, g.beta, initial_state=g.initial_state, output_final_state=True,
                                      use_qk_l2norm_in_kernel=True, z=g.z)
    assert gdn.read_status() == 0
    o_ref, s_ref = C.recurrent(inp.q, inp.k, inp.v, inp.g, inp.beta, inp.scale, inp.initial_state, use_qk_l2norm_in_kernel=True)
    y_ref = O.gated_rmsnorm(o_ref, inp.z)
    for h in range(2 * ratio):
        check_o(O, o[:, :, h], y_ref[:, :, h])
        check_s(O, s[:, h], s_ref[:, h])


# the longest sequence unknown (the parts are sized from the packed total), known, and bounded from above
@pytest.mark.parametrize("bound", [None, 3000, 4100])
@pytest.mark.parametrize("with_z", [False, True])
def test_parts_of_a_packed_batch(built_lib, checker, bound, with_z):
    from avelang_b200 import gdn
    O, C = checker
    lens = (700, 3000, 64, 1, 2500)
    cu = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32)
    inp = synth.make_inputs(1, sum(lens), 2, 4, 128, 128, seed=107, with_z=with_z, n_states=len(lens), gate_scale=0.05)
    g = dev(inp)
    o, s = gdn.chunk_gated_delta_rule(g.q, g.k, g.v, g.g, g.beta, initial_state=g.initial_state, output_final_state=True, cu_seqlens=cu.cuda(), z=g.z,
                                      max_seqlen=bound)
    assert gdn.read_status() == 0
    o_ref, s_ref = C.recurrent(inp.q, inp.k, inp.v, inp.g, inp.beta, inp.scale, inp.initial_state, cu)
    if with_z:
        o_ref = O.gated_rmsnorm(o_ref, inp.z)
    for n in range(len(lens)):
        check_o(O, o[:, cu[n]:cu[n + 1]], o_ref[:, cu[n]:cu[n + 1]])
        check_s(O, s[n], s_ref[n])
