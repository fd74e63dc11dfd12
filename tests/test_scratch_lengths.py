"""Scratch sized for the longest of a caller's prompts serves the shorter ones: a prompt whose best schedule would want more runs with fewer parts."""
import ctypes

import pytest
import torch

from avelang_b200 import _lib, synth
from test_prefill_schedule import _args


def _parts(args, workspace_bytes=None):
    a = args._obj
    a.workspace, a.workspace_bytes = (0x1000, workspace_bytes) if workspace_bytes is not None else (None, 0)
    return _lib.load().ave_gdn_prefill_parts(args)


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("B, heads", [(1, 2), (1, 4), (2, 4), (3, 4), (1, 10), (1, 12), (1, 16), (1, 20), (1, 24), (3, 8), (1, 30), (1, 32), (1, 48)])
def test_scratch_of_the_longest_prompt_is_enough(built_lib, B, heads, gated):
    lib, per_chunk = _lib.load(), 21504 + 32768  # of a chunk-head: its record and its rows in fp32; with parts its images as well
    for longest in range(1, 200):
        have = lib.ave_gdn_prefill_workspace_bytes(_args(B, 64 * longest, heads, gated))
        for chunks in {longest, longest - 1, longest - 2, longest // 2, min(longest, 31)} - {0, -1}:
            args = _args(B, 64 * chunks, heads, gated)
            parts = _parts(args, have)
            need = B * chunks * heads * (per_chunk + 32768) + B * heads * 65536 * (3 * parts - 2) if parts > 1 else B * chunks * heads * (per_chunk if gated else 21504)
            assert need <= have
            if lib.ave_gdn_prefill_workspace_bytes(args) <= have:
                assert parts == _parts(args)


@pytest.mark.gpu
@pytest.mark.parametrize("chunks, heads, B", [(20, 4, 3), (24, 16, 1), (56, 2, 1)])  # more scratch wanted than a chunk further on
@pytest.mark.parametrize("gated", [False, True])
def test_shorter_prompts_in_the_scratch_of_a_longer_one(built_lib, checker, chunks, heads, B, gated):
    from gpu_util import check_o, check_s, dev
    O, C = checker  # noqa: N806
    lib = _lib.load()
    inp = synth.make_inputs(B, 64 * chunks, heads // 2, heads, 128, 128, seed=chunks, with_z=gated, n_states=B, gate_scale=0.02)
    g = dev(inp)
    args = _args(B, 64 * chunks, heads, gated)
    a = args._obj
    o, s, status = torch.empty_like(g.v), torch.empty_like(g.initial_state), torch.zeros(1, dtype=torch.int32, device="cuda")
    for name in ("q", "k", "v", "g", "beta", "z"):
        if getattr(g, name, None) is not None:
            setattr(a, name, getattr(g, name).data_ptr())
    a.o, a.initial_state, a.final_state, a.status = o.data_ptr(), g.initial_state.data_ptr(), s.data_ptr(), status.data_ptr()
    for name in "qkvoz":
        t = {"q": g.q, "k": g.k, "v": g.v, "o": o, "z": g.z}[name]
        if t is not None:
            for i, d in ((0, "b"), (1, "t"), (2, "h")):
                setattr(a, f"{name}_stride_{d}", t.stride(i))
    a.g_stride_b, a.g_stride_t, a.scale, a.norm_eps = g.g.stride(0), g.g.stride(1), inp.scale, 1e-6
    have = lib.ave_gdn_prefill_workspace_bytes(_args(B, 64 * (chunks + 1), heads, gated))
    ws = torch.empty(have, dtype=torch.uint8, device="cuda")
    a.workspace, a.workspace_bytes = ws.data_ptr(), have
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.ave_gdn_chunk_prefill(args, stream) == _lib.OK
    o_ref, s_ref = C.recurrent(inp.q, inp.k, inp.v, inp.g, inp.beta, inp.scale, inp.initial_state)
    if gated:
        o_ref = O.gated_rmsnorm(o_ref, inp.z)
    assert int(status) == 0
    check_o(O, o, o_ref)
    check_s(O, s, s_ref)
    a.workspace_bytes = 1 << 20
    assert lib.ave_gdn_chunk_prefill(args, stream) == _lib.WORKSPACE_TOO_SMALL
