"""What a call's kernels wait for, read from a captured call: an edge between two kernels is all that orders them."""
import pytest
import torch

from avelang_b200 import synth

pytestmark = pytest.mark.gpu
KERNELS = ("chunk_table", "chunk_tiles", "chunk_scan", "gated_rmsnorm", "gdn_decode_pool", "gdn_shared_slots", "part_combine", "part_finish")


def _waits(call):
    """kernel -> the kernels it waits for, directly (an event adds no node)"""
    driver = pytest.importorskip("cuda.bindings.driver")
    call()  # creates streams, events and the status word outside the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()

    def ok(result):
        assert result[0] == driver.CUresult.CUDA_SUCCESS, result[0]
        return result[1:]

    def name(node):
        full = ok(driver.cuFuncGetName(ok(driver.cuGraphKernelNodeGetParams(node))[0].func))[0].decode()
        return next(k for k in KERNELS if k in full)

    raw = driver.CUgraph(graph.raw_cuda_graph())
    n = ok(driver.cuGraphGetEdges_v2(raw))[3]
    before, after = ok(driver.cuGraphGetEdges_v2(raw, n))[:2]
    waits = {}
    for x, y in zip(before, after):
        waits.setdefault(name(y), set()).add(name(x))
    return waits


# two parts: the scan has written all that the fix-up needs; three: the combine forms the state that enters the third
@pytest.mark.parametrize("B, heads, T, two", [(1, 32, 64 * 112, True), (2, 16, 64 * 112, True), (1, 28, 64 * 40, False)])
@pytest.mark.parametrize("gated", [False, True])
def test_the_fix_up_of_two_parts_waits_for_the_scan_alone(built_lib, B, heads, T, two, gated):
    from avelang_b200 import gdn
    inp = synth.make_inputs(B, T, heads // 2, heads, 128, 128, seed=T, with_z=gated, n_states=B).to("cuda")
    waits = _waits(lambda: gdn.chunk_gated_delta_rule(inp.q, inp.k, inp.v, inp.g, inp.beta, output_final_state=True, z=inp.z))
    assert waits["part_finish"] == ({"chunk_scan"} if two else {"part_combine"})
    assert waits["part_combine"] == {"chunk_scan"} and waits.get("gated_rmsnorm", set()) <= {"chunk_scan", "gated_rmsnorm"}  # (a launch a batch row)


@pytest.mark.parametrize("lens", [(200, 100), (3000,)])  # whole chains; parts
def test_single_tokens_run_beside_the_scan_and_nothing_waits_through_them(built_lib, lens):
    from avelang_b200 import gdn
    n, seqs = 40, 40 + len(lens)
    inp = synth.make_inputs(1, n + sum(lens), 2, 4, 128, 128, seed=n, with_z=True, n_states=seqs).to("cuda")
    cu = torch.tensor([0] + list(range(1, n + 1)) + [n + sum(lens[:i + 1]) for i in range(len(lens))], dtype=torch.int32, device="cuda")
    slots = torch.arange(seqs, dtype=torch.int32, device="cuda")
    waits = _waits(lambda: gdn.mixed_prefill_decode_step(inp.q, inp.k, inp.v, inp.g, inp.beta, cu, n, inp.initial_state, slots, z=inp.z))
    assert waits["gdn_shared_slots"] == {"chunk_tiles"} and waits["gdn_decode_pool"] == {"gdn_shared_slots"}
    assert waits["chunk_scan"] == {"gdn_shared_slots"} and waits["gated_rmsnorm"] == {"chunk_scan"}  # the norm reads the scan's rows: an edge of its own
    assert not any("gdn_decode_pool" in w for w in waits.values())
