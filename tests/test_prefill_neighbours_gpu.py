"""A packed sequence is not touched by what its neighbours hold: every other sequence, and the tokens behind the last offset, full of NaN or infinity
leave its outputs and its state as they are, bit for bit."""
import pytest
import torch

from avelang_b200 import synth

pytestmark = pytest.mark.gpu


# tails of one token, all but one, a block and one off it; whole chunks; a single chunk and several; parallel parts with a ragged end
@pytest.mark.parametrize("Hk, Hv, lens", [(2, 4, (1, 65, 63, 64, 79, 80, 17, 200, 128, 15)), (16, 32, (203, 190, 5, 300, 64, 33)), (2, 4, (64 * 40 + 13, 64 * 33 + 50))])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("gated", [False, True])
def test_neighbours_do_not_leak(built_lib, Hk, Hv, lens, value, gated):
    from avelang_b200 import gdn
    T, n = sum(lens) + 100, len(lens)
    inp = synth.make_inputs(1, T, Hk, Hv, 128, 128, seed=n, with_z=gated, n_states=n, gate_scale=0.3).to("cuda")
    at = [sum(lens[:i]) for i in range(n + 1)]
    cu = torch.tensor(at, dtype=torch.int32, device="cuda")

    def call(x, s0):
        return gdn.chunk_gated_delta_rule(*x, initial_state=s0, output_final_state=True, cu_seqlens=cu, use_qk_l2norm_in_kernel=gated, z=inp.z)

    x = [inp.q, inp.k, inp.v, inp.g, inp.beta]
    o, s = call(x, inp.initial_state)
    for odd in (0, 1):
        bad, s0 = [t.clone() for t in x], inp.initial_state.clone()
        for i in range(n):
            if i % 2 != odd:
                for t in bad:
                    t[:, at[i]:at[i + 1]] = value
                s0[i] = value
        for t in bad:
            t[:, at[n]:] = value
        o2, s2 = call(bad, s0)
        for i in range(odd, n, 2):
            assert torch.equal(o2[:, at[i]:at[i + 1]], o[:, at[i]:at[i + 1]]), f"outputs of sequence {i}"
            assert torch.equal(s2[i], s[i]), f"state of sequence {i}"
    assert gdn.read_status() == 0
