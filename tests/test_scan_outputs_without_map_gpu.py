"""A result whose layout no tensor map describes: the scan's whole chunks then leave by 16-byte stores.  One head, so the head stride is never walked, and it
is longer than a map takes (2^40 bytes)."""
import pytest
import torch

from avelang_b200 import synth
from gpu_util import check_o, check_s, dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T, lens", [(64, None), (257, None), (200, [1, 63, 64, 72])])
def test_rows_without_a_map(built_lib, checker, T, lens):
    from avelang_b200 import gdn
    O, C = checker  # noqa: N806
    n = len(lens) if lens else 1
    inp = synth.make_inputs(1, T, 1, 1, 128, 128, seed=T, n_states=n)
    if lens:
        inp.cu_seqlens = torch.tensor([sum(lens[:i]) for i in range(n + 1)], dtype=torch.int32)
    g = dev(inp)
    whole = torch.full((T + 64, 2, 128), 7.0, dtype=torch.bfloat16, device="cuda")  # rows between the result's and behind them hold a mark
    out = whole.as_strided((1, T, 1, 128), (256 * (T + 64), 256, 1 << 40, 1))
    _, s = gdn.chunk_gated_delta_rule(g.q, g.k, g.v, g.g, g.beta, initial_state=g.initial_state, output_final_state=True,
                                      cu_seqlens=g.cu_seqlens if lens else None, out=out)
    assert gdn.read_status() == 0
    o_ref, s_ref = C.recurrent(inp.q, inp.k, inp.v, inp.g, inp.beta, inp.scale, inp.initial_state, inp.cu_seqlens if lens else None)
    check_o(O, whole[:T, :1][None], o_ref)
    check_s(O, s, s_ref)
    assert bool((whole[T:] == 7.0).all()) and bool((whole[:, 1:] == 7.0).all())


def test_rows_of_a_heads_first_result(built_lib, checker):
    """The same results where heads lie further apart than tokens, and batch rows between them."""
    from avelang_b200 import gdn
    O, C = checker  # noqa: N806
    B, T, Hv = 2, 257, 4
    inp = synth.make_inputs(B, T, Hv // 2, Hv, 128, 128, seed=5, n_states=B)
    g = dev(inp)
    whole = torch.full((Hv, B, T + 64, 128), 7.0, dtype=torch.bfloat16, device="cuda")
    out = whole[:, :, :T].permute(1, 2, 0, 3)
    _, s = gdn.chunk_gated_delta_rule(g.q, g.k, g.v, g.g, g.beta, initial_state=g.initial_state, output_final_state=True, out=out)
    o_ref, s_ref = C.recurrent(inp.q, inp.k, inp.v, inp.g, inp.beta, inp.scale, inp.initial_state)
    check_o(O, out, o_ref)
    check_s(O, s, s_ref)
    assert bool((whole[:, :, T:] == 7.0).all())
