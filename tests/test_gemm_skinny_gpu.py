"""GPU parity of the GEMM's form for few row tiles (narrow column tiles, K split over a cluster)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1, 12352, 2048), (64, 2048, 4096), (37, 2056, 4104), (128, 136, 8192), (129, 96, 72), (64, 16, 8192),
                                   (256, 2048, 4096), (300, 12352, 2048), (5, 8, 64), (2000, 1544, 520)])
def test_few_row_tiles(built_lib, m, n, k):
    from avelang_b200 import gdn, gemm
    torch.manual_seed(m + n + k)
    A = torch.randn(m, k, device="cuda").bfloat16()
    B = (torch.randn(n, k, device="cuda") * 0.02).bfloat16()
    wide = torch.full((m, n + 24), 7.0, device="cuda").bfloat16()
    out = gemm.gemm_pipeline_transposed_b(A, B, out=wide[:, 8:n + 8])  # 16-byte aligned rows inside a wider matrix
    ref = (A.double() @ B.double().T)
    err = (out.double() - ref).norm() / ref.norm()
    assert err < 2.5e-3, f"rel-L2 {err:.3e}"  # one rounding to bf16
    assert gdn.read_status() == 0
    assert bool((wide[:, :8] == 7).all()) and bool((wide[:, n + 8:] == 7).all())  # nothing outside the result
