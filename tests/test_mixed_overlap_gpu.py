"""The two parts of a mixed step run beside one another on the GPU; the same parts as separate calls, one after the other, give the same
bits.  Three steps in a row on one pool, eagerly and replayed from a graph: a step that began before the last one was complete would
read old states."""
import pytest
import torch

from avelang_b200 import synth

pytestmark = pytest.mark.gpu


# one tile and one prompt; prompts that end long before and long after the decode; two and four tiles a CTA (75 x 32 tiles is the
# first size with four), an odd rest; more chains than SMs; sequences in parts; empty sequences; skipped slots
@pytest.mark.parametrize("Hk, Hv, n, lens, gated", [
    (2, 4, 1, (64,), True), (2, 4, 1, (3,), False), (16, 32, 73, (40, 700), True), (16, 32, 75, (1, 0, 129), True),
    (16, 32, 74, (0, 0), True), (16, 32, 3, (64, 200, 0, 300, 128, 1), False), (4, 8, 21, (5000,), True), (8, 24, 33, (640, 65), True)])
def test_mixed_equals_the_parts(built_lib, Hk, Hv, n, lens, gated):
    from avelang_b200 import gdn
    T, seqs = n + sum(lens), n + len(lens)
    inp = synth.make_inputs(1, T, Hk, Hv, 128, 128, seed=n, with_z=gated, n_states=seqs + 3, gate_scale=0.3).to("cuda")
    cu = torch.tensor([0] + list(range(1, n + 1)) + [n + sum(lens[:i + 1]) for i in range(len(lens))], dtype=torch.int32, device="cuda")
    slots = torch.randperm(seqs + 3, generator=torch.Generator().manual_seed(n))[:seqs].to("cuda", torch.int32)
    if n > 8:
        slots[5] = -1  # skipped: zero output, no state access
    x = [inp.q, inp.k, inp.v, inp.g, inp.beta]
    head, tail = [t[:, :n] for t in x], [t[:, n:] for t in x]
    z = inp.z if gated else None

    def apart(pool, out):
        gdn.mixed_prefill_decode_step(*head, cu[:n + 1], n, pool, slots[:n], z=None if z is None else z[:, :n], out=out[:, :n])
        if T > n:
            gdn.chunk_gated_delta_rule(*tail, initial_state=pool, output_final_state=True, cu_seqlens=cu[n:] - n,
                                       state_indices=slots[n:], inplace_state=True, z=None if z is None else z[:, n:], out=out[:, n:])

    def mixed(pool, out):
        gdn.mixed_prefill_decode_step(*x, cu, n, pool, slots, z=z, out=out)

    pools = [inp.initial_state.clone() for _ in range(3)]
    outs = [torch.empty_like(inp.v) for _ in range(3)]
    for _ in range(3):
        apart(pools[0], outs[0])
        mixed(pools[1], outs[1])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        mixed(pools[2], outs[2])
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert gdn.read_status() == 0
    for p, o in zip(pools[1:], outs[1:]):
        assert torch.equal(p, pools[0]) and torch.equal(o, outs[0])
