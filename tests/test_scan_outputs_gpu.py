"""Where the scan's rows go: whole chunks leave by asynchronous copies of 64 tokens, which may not touch what lies behind a sequence or a batch row."""
import pytest
import torch

from avelang_b200 import synth
from gpu_util import check_o, check_s, dev

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gdn(built_lib):
    from avelang_b200 import gdn
    return gdn


@pytest.mark.parametrize("T,lens,Hv", [(70, None, 4), (128, None, 3), (257, None, 4), (200, [1, 63, 64, 72], 4), (130, [65, 65], 2)])
@pytest.mark.parametrize("gated", [False, True])
def test_rows_behind_a_sequence_stay(gdn, checker, T, lens, Hv, gated):
    """The result is a view into a larger tensor, with rows and heads between its own that hold a mark."""
    O, C = checker
    B = 1 if lens else 2
    inp = synth.make_inputs(B, T, Hv // 2 if Hv % 2 == 0 else Hv, Hv, 128, 128, seed=T + Hv, with_z=gated, n_states=len(lens) if lens else B)
    if lens:
        inp.cu_seqlens = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32)
    g = dev(inp)
    whole = torch.full((B, T + 64, Hv + 1, 128), 7.0, dtype=torch.bfloat16, device="cuda")
    out = whole[:, :T, :Hv]
    _, s = gdn.chunk_gated_delta_rule(g.q, g.k, g.v, g.g, g.beta, initial_state=g.initial_state, output_final_state=True,
                                      cu_seqlens=g.cu_seqlens if lens else None, z=g.z if gated else None, out=out)
    o_ref, s_ref = C.recurrent(inp.q, inp.k, inp.v, inp.g, inp.beta, inp.scale, inp.initial_state, inp.cu_seqlens if lens else None)
    if gated:
        o_ref = O.gated_rmsnorm(o_ref, inp.z)
    check_o(O, out, o_ref)
    check_s(O, s, s_ref)
    assert bool((whole[:, T:] == 7.0).all()) and bool((whole[:, :, Hv:] == 7.0).all())


@pytest.mark.parametrize("lens", [[4096], [2079, 2017], [3000, 40, 1056]])
def test_rows_of_parts_behind_a_sequence_stay(gdn, checker, lens):
    """Four heads in parallel parts: local rows and the transition chains' images, with last chunks of odd length."""
    O, C = checker
    T = sum(lens)
    inp = synth.make_inputs(1, T, 2, 4, 128, 128, seed=T + len(lens), n_states=len(lens), gate_scale=0.01)
    inp.cu_seqlens = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32)
    g = dev(inp)
    whole = torch.full((1, T + 64, 5, 128), 7.0, dtype=torch.bfloat16, device="cuda")
    out = whole[:, :T, :4]
    _, s = gdn.chunk_gated_delta_rule(g.q, g.k, g.v, g.g, g.beta, initial_state=g.initial_state, output_final_state=True, cu_seqlens=g.cu_seqlens,
                                      out=out, max_seqlen=max(lens))
    o_ref, s_ref = C.recurrent(inp.q, inp.k, inp.v, inp.g, inp.beta, inp.scale, inp.initial_state, inp.cu_seqlens)
    check_o(O, out, o_ref)
    check_s(O, s, s_ref)
    assert bool((whole[:, T:] == 7.0).all()) and bool((whole[:, :, 4:] == 7.0).all())


@pytest.mark.parametrize("B,T,Hv", [(1, 1024, 4), (1, 1529, 16), (2, 1990, 8), (1, 2048, 24), (1, 6144, 8)])  # four, two, four, two and eight parts
@pytest.mark.parametrize("gated", [False, True])
def test_short_chains_in_parts(gdn, checker, B, T, Hv, gated):
    O, C = checker
    inp = synth.make_inputs(B, T, Hv // 2, Hv, 128, 128, seed=T, with_z=gated, n_states=B, gate_scale=0.02)
    g = dev(inp)
    o, s = gdn.chunk_gated_delta_rule(g.q, g.k, g.v, g.g, g.beta, initial_state=g.initial_state, output_final_state=True, z=g.z if gated else None)
    o_ref, s_ref = C.recurrent(inp.q, inp.k, inp.v, inp.g, inp.beta, inp.scale, inp.initial_state)
    if gated:
        o_ref = O.gated_rmsnorm(o_ref, inp.z)
    check_o(O, o, o_ref)
    check_s(O, s, s_ref)
