"""A mixed step in which single-token sequences and prompts name the same slots: the single token comes first and the prompt goes on from its state, as
when the two parts are called one after the other."""
import pytest
import torch

from avelang_b200 import synth

pytestmark = pytest.mark.gpu


# a prompt of one chunk, of several, an empty one, a skipped one, more prompts than a warp, sequences in parts, one prompt a slot for two
@pytest.mark.parametrize("Hk, Hv, n, lens, shared", [
    (2, 4, 1, (3,), {0: 0}), (16, 32, 40, (130, 64, 0, 20), {3: 0, 39: 2, 7: 3}), (2, 4, 70, (65,) * 37, {0: 36, 69: 0, 33: 32}),
    (4, 8, 9, (2500,), {8: 0}), (2, 4, 5, (40, 3000), {1: 1})])
@pytest.mark.parametrize("gated", [False, True])
def test_the_single_token_comes_first(built_lib, Hk, Hv, n, lens, shared, gated):
    from avelang_b200 import gdn
    T, seqs = n + sum(lens), n + len(lens)
    inp = synth.make_inputs(1, T, Hk, Hv, 128, 128, seed=n, with_z=gated, n_states=seqs + 2, gate_scale=0.1).to("cuda")
    cu = torch.tensor([0] + list(range(1, n + 1)) + [n + sum(lens[:i + 1]) for i in range(len(lens))], dtype=torch.int32, device="cuda")
    slots = torch.randperm(seqs + 2, generator=torch.Generator().manual_seed(n))[:seqs].to(torch.int32)
    for row, prompt in shared.items():
        slots[row] = slots[n + prompt]
    if n > 30:
        slots[12] = slots[n + 1] = -1  # two that are skipped share nothing
    slots = slots.to("cuda")
    x, z = [inp.q, inp.k, inp.v, inp.g, inp.beta], inp.z
    l2 = dict(use_qk_l2norm_in_kernel=gated)
    pool_a, pool_m = inp.initial_state.clone(), inp.initial_state.clone()
    out_a, out_m = torch.empty_like(inp.v), torch.empty_like(inp.v)
    for _ in range(2):  # the second step starts from what the first left
        gdn.mixed_prefill_decode_step(*[t[:, :n] for t in x], cu[:n + 1], n, pool_a, slots[:n], z=None if z is None else z[:, :n], out=out_a[:, :n], **l2)
        gdn.chunk_gated_delta_rule(*[t[:, n:] for t in x], initial_state=pool_a, output_final_state=True, cu_seqlens=cu[n:] - n, state_indices=slots[n:],
                                   inplace_state=True, z=None if z is None else z[:, n:], out=out_a[:, n:], **l2)
        gdn.mixed_prefill_decode_step(*x, cu, n, pool_m, slots, z=z, out=out_m, **l2)
    assert gdn.read_status() == 0
    assert torch.equal(out_m, out_a) and torch.equal(pool_m, pool_a)
