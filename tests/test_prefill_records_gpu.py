"""GPU parity of packed batches on both sides of the rule for the chunk tables (sequences x value heads against 148), with lengths
around the chunk size, empty sequences, and a rejected offset table."""
import pytest
import torch

from avelang_b200 import synth
from gpu_util import check_o, check_s, dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [[1], [0, 64, 0], [63, 1, 64, 65, 1, 0, 127], [300] + [1, 0, 62] * 11 + [2], [5] * 36 + [129], [3, 0, 64, 70] * 10])
def test_packed_records(built_lib, checker, lens):
    from avelang_b200 import gdn
    O, C = checker
    T, n = sum(lens), len(lens)
    inp = synth.make_inputs(1, T, 2, 4, 128, 128, seed=7 + T, n_states=n, gate_scale=0.1)
    cu = torch.tensor([0] + lens, dtype=torch.int64).cumsum(0).to(torch.int32)
    g = dev(inp)
    call = lambda off: gdn.chunk_gated_delta_rule(g.q, g.k, g.v, g.g, g.beta, initial_state=g.initial_state, output_final_state=True, cu_seqlens=off)
    o, s = call(cu.cuda())
    assert gdn.read_status() == 0
    o_ref, s_ref = C.recurrent(inp.q, inp.k, inp.v, inp.g, inp.beta, inp.scale, inp.initial_state, cu)
    check_o(O, o, o_ref)
    check_s(O, s, s_ref)
    if n > 2:
        bad = cu.clone()
        bad[n // 2] = T + 1
        call(bad.cuda())
        assert gdn.read_status() & 2
