"""The backward pass with less scratch than all key heads need: it takes them in several passes, with the same results."""
import ctypes

import pytest
import torch

from avelang_b200 import _lib, synth
from gpu_util import dev


def _args(g, d_o, ds, cu, outs, flags):
    a = _lib.BwdArgs()
    a.struct_size, a.flags = ctypes.sizeof(_lib.BwdArgs), flags
    a.q, a.k, a.v, a.g, a.beta, a.d_o, a.initial_state, a.d_final_state, a.cu_seqlens = (
        t.data_ptr() for t in (g.q, g.k, g.v, g.g, g.beta, d_o, g.initial_state, ds, cu))
    a.d_q, a.d_k, a.d_v, a.d_g, a.d_beta, a.d_initial_state = (t.data_ptr() for t in outs)
    a.B, a.T, a.Hk, a.dk = g.q.shape
    a.Hv, a.dv, a.n_seqs, a.scale = g.v.shape[2], g.v.shape[3], cu.numel() - 1, g.scale
    for name, t in (("q", g.q), ("k", g.k), ("v", g.v), ("do", d_o)):
        for d, ax in (("b", 0), ("t", 1), ("h", 2)):
            setattr(a, f"{name}_stride_{d}", t.stride(ax))
    a.g_stride_b, a.g_stride_t = g.g.stride(0), g.g.stride(1)
    return a


@pytest.mark.parametrize("B, T, packed, Hk, Hv", [(2, 4096, 0, 16, 32), (1, 131072, 0, 16, 32), (1, 300, 7, 1, 3)])
def test_scratch_size_is_what_the_header_says(built_lib, B, T, packed, Hk, Hv):
    a = _lib.BwdArgs()
    a.struct_size = ctypes.sizeof(_lib.BwdArgs)
    for n in ("q", "k", "v", "g", "beta", "d_o", "d_q", "d_k", "d_v", "d_g", "d_beta"):
        setattr(a, n, 0x1000)  # never read: only sizes enter
    a.B, a.T, a.Hk, a.Hv, a.dk, a.dv, a.n_seqs = B, T, Hk, Hv, 128, 128, packed or B
    a.cu_seqlens = 0x1000 if packed else None
    size = lambda: _lib.load().ave_gdn_backward_workspace_bytes(ctypes.byref(a))
    records = B * T // 64 + a.n_seqs + 1
    assert size() == 246528 * records * Hv
    a.Hk, a.Hv = 1, Hv // Hk
    assert size() == 246528 * records * (Hv // Hk)


@pytest.mark.gpu
@pytest.mark.parametrize("summed", [False, True])
def test_key_heads_in_passes(built_lib, summed):
    lib = _lib.load()
    Hk, r, T = 3, 2, 330
    g = dev(synth.make_inputs(1, T, Hk, Hk * r, 128, 128, seed=95, n_states=3, gate_scale=0.3))
    cu = torch.tensor([0, 70, 71, T], dtype=torch.int32, device="cuda")
    d_o, ds = torch.randn_like(g.v), 0.1 * torch.randn_like(g.initial_state)
    dt, hq = (torch.bfloat16, Hk) if summed else (torch.float32, Hk * r)
    def fresh():
        return [torch.full(s, 7.0, dtype=t, device="cuda") for s, t in
                (((1, T, hq, 128), dt), ((1, T, hq, 128), dt), ((1, T, Hk * r, 128), dt), ((1, T, Hk * r), torch.float32),
                 ((1, T, Hk * r), torch.float32), ((3, Hk * r, 128, 128), torch.float32))]

    def run(scratch_heads, less=0):
        outs = fresh()
        a = _args(g, d_o, ds, cu, outs, _lib.FLAG_BWD_SUMMED if summed else 0)
        a.Hk, a.Hv = scratch_heads, scratch_heads * r
        n = lib.ave_gdn_backward_workspace_bytes(ctypes.byref(a)) - less
        assert n > 0
        a.Hk, a.Hv = Hk, Hk * r
        ws = torch.empty(n, dtype=torch.uint8, device="cuda")
        a.workspace, a.workspace_bytes = ws.data_ptr(), n
        rc = lib.ave_gdn_recurrent_backward(ctypes.byref(a), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        return rc, outs

    rc, want = run(Hk)
    assert rc == _lib.OK
    for heads, less in ((Hk, 1), (2, 0), (2, 1), (1, 0)):  # passes of 2 + 1, 2 + 1, 1 + 1 + 1 and 1 + 1 + 1 key heads
        rc, got = run(heads, less)
        assert rc == _lib.OK and all(torch.equal(x, y) for x, y in zip(got, want))
    rc, got = run(1, 1)
    assert rc == _lib.WORKSPACE_TOO_SMALL and all(bool((x == 7.0).all()) for x in got)


@pytest.mark.gpu
def test_public_call_when_memory_is_short(built_lib):
    from avelang_b200 import gdn
    g = dev(synth.make_inputs(1, 2048, 8, 16, 128, 128, seed=96, gate_scale=0.3))  # 141 MB of scratch in one pass
    d_o = torch.randn_like(g.v)
    run = lambda: gdn.gated_delta_rule_backward(g.q, g.k, g.v, g.g, g.beta, d_o)
    want = run()
    total = torch.cuda.get_device_properties(0).total_memory
    allow = lambda more: torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + more) / total)
    torch.cuda.synchronize()
    try:
        allow(0)
        with pytest.raises(torch.OutOfMemoryError):
            torch.empty(total, dtype=torch.uint8, device="cuda")  # kept scratch goes back
        torch.cuda.empty_cache()
        allow(80 << 20)
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        got = run()
        torch.cuda.synchronize()
        assert torch.cuda.max_memory_allocated() - before <= 80 << 20
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert got[5] is None and all(torch.equal(x, y) for x, y in zip(got[:5], want[:5])) and gdn.read_status() == 0
