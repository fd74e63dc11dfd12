"""GPU parity of the causal convolution where its runs of tokens per CTA change (64, 128, 256), with sequence ends inside and at
the ends of runs, and with weights that are not 16-byte aligned."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [3, 128 * 2368 - 3, 256 * 2368 - 255, 256 * 2368 + 5])
@pytest.mark.parametrize("width", [2, 4])
def test_conv_runs(built_lib, T, width):
    from avelang_b200 import gdn
    gen = torch.Generator().manual_seed(T)
    x = torch.randn(1, T, 8, generator=gen).bfloat16().cuda()
    store = torch.empty(8 * width + 1, dtype=torch.bfloat16, device="cuda")
    w = store[1:].view(8, width)
    w.copy_(torch.randn(8, width, generator=gen) / 2)
    cu = torch.tensor(sorted({0, 1, T // 3, T // 2 // 256 * 256, T - 1, T}), dtype=torch.int32)
    y = gdn.causal_conv1d_silu(x, w, cu_seqlens=cu.cuda())
    xs, ws, ref = x.float(), w.float(), torch.empty_like(x)
    for a, b in zip(cu[:-1].tolist(), cu[1:].tolist()):
        pad = torch.nn.functional.pad(xs[:, a:b], (0, 0, width - 1, 0))
        ref[:, a:b] = torch.nn.functional.silu(sum(pad[:, j:j + b - a] * ws[:, j] for j in range(width)))
    assert torch.equal(gdn.causal_conv1d_silu(x, w.clone(), cu_seqlens=cu.cuda()), y)
    assert float((y.float() - ref.float()).norm() / ref.float().norm()) <= 1e-3
