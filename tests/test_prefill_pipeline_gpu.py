"""GPU parity of the prefill at the depths of its two pipelines: pass 1 runs persistent CTAs (two an SM) that work a unit ahead with two
sets of token factors, and the scan keeps three chunks in flight."""
import pytest
import torch

from avelang_b200 import synth
from gpu_util import check_o, check_s, dev

pytestmark = pytest.mark.gpu


def _check(checker, inp, with_z, l2norm, cu=None):
    from avelang_b200 import gdn
    O, C = checker
    g = dev(inp)
    o, s = gdn.chunk_gated_delta_rule(g.q, g.k, g.v, g.g, g.beta, initial_state=g.initial_state, output_final_state=True, z=g.z,
                                      use_qk_l2norm_in_kernel=l2norm, cu_seqlens=None if cu is None else cu.to("cuda"))
    assert gdn.read_status() == 0
    o_ref, s_ref = C.recurrent(inp.q, inp.k, inp.v, inp.g, inp.beta, inp.scale, inp.initial_state, cu, use_qk_l2norm_in_kernel=l2norm)
    if with_z:
        o_ref = O.gated_rmsnorm(o_ref, inp.z)
    for t0 in range(0, o.shape[1], 64):  # chunk by chunk: one that is taken from a stale buffer cannot hide in the total
        check_o(O, o[:, t0:t0 + 64], o_ref[:, t0:t0 + 64])
    check_s(O, s, s_ref)


# one to seven chunks: the ring of three stages unused, full, and around twice; a whole last chunk, one token and all but one
@pytest.mark.parametrize("T", [1, 64, 65, 129, 192, 193, 255, 256, 320, 385, 448])
@pytest.mark.parametrize("l2norm", [False, True])
def test_chunks_in_flight(built_lib, checker, T, l2norm):
    _check(checker, synth.make_inputs(1, T, 2, 4, 128, 128, seed=T, with_z=l2norm, n_states=1, gate_scale=0.1, l2norm=not l2norm), l2norm, l2norm)


# 296 CTAs: one, two, three and five units of pass 1 each, with odd numbers of value heads a unit and a packed batch among them
@pytest.mark.parametrize("Hk, Hv, T, lens", [(16, 16, 64 * 19, None), (8, 24, 64 * 36 + 1, None), (16, 32, 64 * 45, None), (16, 32, 5500, (1, 700, 64, 1, 2500, 2234))])
def test_units_of_one_cta(built_lib, checker, Hk, Hv, T, lens):
    inp = synth.make_inputs(1, T, Hk, Hv, 128, 128, seed=Hv, with_z=False, n_states=len(lens) if lens else 1, gate_scale=0.3)
    cu = None if lens is None else torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32)
    _check(checker, inp, False, False, cu)
