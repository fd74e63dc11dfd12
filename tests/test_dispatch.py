"""Every public function reaches its kernels through its operator of torch.ops.avelang_gdn, where dispatch modes (and with them
tensor subclasses, tracing and the profiler) see the call.  Fake CUDA tensors: no GPU needed."""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from torch.utils._python_dispatch import TorchDispatchMode

from avelang_b200 import synth
from gpu_util import dev


class Recorder(TorchDispatchMode):
    """Notes the operators of the library that are called; runs them only where there is a GPU."""

    def __init__(self, run):
        super().__init__()
        self.run, self.seen = run, []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        if func.namespace != "avelang_gdn":
            return func(*args, **(kwargs or {}))
        self.seen.append(func._schema.name.split("::")[1])
        return func(*args, **(kwargs or {})) if self.run else None


def _calls():
    from avelang_b200 import gdn, gemm
    bf = lambda *s: torch.zeros(*s, dtype=torch.bfloat16, device="cuda:0")
    f32 = lambda *s: torch.zeros(*s, device="cuda:0")
    i32 = lambda *s: torch.zeros(*s, dtype=torch.int32, device="cuda:0")
    qkvgb = lambda b, t: (bf(b, t, 2, 128), bf(b, t, 2, 128), bf(b, t, 4, 128), f32(b, t, 4), f32(b, t, 4))
    cols, cn = 2 * 256 + 2 * 512 + 8, 2 * 256 + 512
    return {
        "chunk_prefill": lambda: gdn.chunk_gated_delta_rule(*qkvgb(1, 9), z=bf(1, 9, 4, 128), output_final_state=True),
        "decode_step": lambda: gdn.fused_recurrent_gated_delta_rule(*qkvgb(3, 1), initial_state=f32(5, 4, 128, 128), state_indices=i32(3)),
        "mixed_step": lambda: gdn.mixed_prefill_decode_step(*qkvgb(1, 9), i32(4), 2, f32(5, 4, 128, 128), i32(3)),
        "recurrent_backward": lambda: gdn.gated_delta_rule_backward(*qkvgb(1, 9), bf(1, 9, 4, 128), initial_state=f32(1, 4, 128, 128)),
        "decode_layer_step": lambda: gdn.decode_layer_step(bf(3, cols), bf(cn, 4), bf(5, 3, cn), f32(4), f32(4), f32(5, 4, 128, 128), i32(3), Hk=2, Hv=4),
        "gated_rmsnorm": lambda: gdn.gated_rmsnorm(bf(2, 3, 4, 128), bf(2, 3, 4, 128), f32(128)),
        "conv1d_silu": lambda: gdn.causal_conv1d_silu(bf(1, 9, 64), bf(64, 4), bf(64)),
        "conv1d_update": lambda: gdn.causal_conv1d_update(bf(3, 64), bf(5, 3, 64), bf(64, 4), state_indices=i32(3)),
        "gate_beta": lambda: gdn.gate_beta(bf(2, 3, 4), bf(2, 3, 4), f32(4), f32(4)),
        "gemm_bf16_nt": lambda: gemm.gemm_pipeline_transposed_b(bf(9, 64), bf(16, 64)),
    }


NAMES = ["chunk_prefill", "decode_step", "mixed_step", "recurrent_backward", "decode_layer_step", "gated_rmsnorm", "conv1d_silu",
         "conv1d_update", "gate_beta", "gemm_bf16_nt"]


@pytest.mark.parametrize("name", NAMES)
def test_public_functions_call_their_operator(built_lib, name):
    with FakeTensorMode(), Recorder(run=False) as mode:
        _calls()[name]()
    assert mode.seen == [name]


def test_checks_hold_under_a_mode(built_lib):
    from avelang_b200 import gdn
    with FakeTensorMode():
        bf = lambda *s: torch.zeros(*s, dtype=torch.bfloat16, device="cuda:0")
        with pytest.raises(ValueError, match="kernel width must be 2, 3 or 4"):
            gdn.causal_conv1d_silu(bf(1, 9, 64), bf(64, 5))
        x = bf(1, 9, 64)
        with pytest.raises(ValueError, match="out must not alias x"):
            gdn.causal_conv1d_silu(x, bf(64, 4), out=x)


@pytest.mark.gpu
def test_results_under_a_mode_and_ranges_in_the_profiler(built_lib):
    from avelang_b200 import gdn
    g = dev(synth.make_inputs(1, 130, 2, 4, 128, 128, seed=7, with_z=True))
    run = lambda: gdn.chunk_gated_delta_rule(g.q, g.k, g.v, g.g, g.beta, z=g.z, output_final_state=True)
    want = run()
    with Recorder(run=True) as mode:
        got = run()
    assert mode.seen == ["chunk_prefill"] and torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        run()
    assert "avelang_gdn::chunk_prefill" in [e.name for e in prof.events()]
    q = torch.zeros(1, 130, 2, 136, dtype=torch.bfloat16, device="cuda")[..., 4:132]  # rows not on 16 bytes: refused before any launch
    with pytest.raises(ValueError, match="16-byte"):
        gdn.chunk_gated_delta_rule(q, q, g.v, g.g, g.beta)
    with pytest.raises(ValueError, match="16-byte"):  # an operator called by itself maps errors the same way
        torch.ops.avelang_gdn.chunk_prefill(q, q, g.v, g.g, g.beta, torch.empty_like(g.v), 1.0, None, None, None, None, None, None, 1e-6, False, 0, None)
