"""The fused decode layer step deals (sequence, key head) units to pairs of CTAs, which share the last of an odd number: its states and histories are those of the
separate kernels, bit for bit, for every way the units can fall."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N, Hk, ratio", [(1, 16, 2), (9, 16, 2), (10, 16, 2), (20, 16, 2), (28, 16, 2), (64, 16, 2),  # 1; 1; 1 or 2; 3 or 2; 4 or 3; 7 or 6 units a pair
                                          (1, 1, 1), (150, 1, 1), (5, 3, 3), (60, 3, 3), (37, 8, 4)])
def test_units_of_every_number(built_lib, N, Hk, ratio):
    from avelang_b200 import gdn
    d, W, Hv, slots = 128, 4, Hk * ratio, N + 3
    Cn, cols = 2 * Hk * d + Hv * d, 2 * Hk * d + 2 * Hv * d + 2 * Hv
    gen = torch.Generator(device="cuda").manual_seed(N * 100 + Hk)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    cw, Al, dtb, nw = (rand(Cn, W) / 2).bfloat16(), torch.rand(Hv, generator=gen, device="cuda") * 2.77, 0.1 * rand(Hv), 1.0 + 0.1 * rand(d)
    ix = torch.randperm(slots, generator=gen, device="cuda")[:N].to(torch.int32)
    if N > 4:
        ix[3] = -1
    pool_f, conv_f = 0.02 * rand(slots, Hv, d, d), rand(slots, W - 1, Cn).bfloat16()
    pool_s, conv_s = pool_f.clone(), conv_f.clone()
    for _ in range(2):
        proj = rand(N, (cols + 15) // 8 * 8).bfloat16()[:, :cols]  # (rows are 16-byte aligned)
        o_f = gdn.decode_layer_step(proj, cw, conv_f, Al, dtb, pool_f, ix, Hk=Hk, Hv=Hv, norm_weight=nw)
        qkv = gdn.causal_conv1d_update(proj[:, :Cn], conv_s, cw, state_indices=ix)
        q, k, v = (x.reshape(N, 1, -1, d) for x in qkv.split([Hk * d, Hk * d, Hv * d], 1))
        g, beta = gdn.gate_beta(proj[:, cols - Hv:cols], proj[:, cols - 2 * Hv:cols - Hv], Al, dtb)
        o_s, _ = gdn.fused_recurrent_gated_delta_rule(q, k, v, g.reshape(N, 1, Hv), beta.reshape(N, 1, Hv), initial_state=pool_s, state_indices=ix,
                                                      use_qk_l2norm_in_kernel=True, z=proj[:, Cn:Cn + Hv * d].reshape(N, 1, Hv, d), norm_weight=nw)
        assert gdn.read_status() == 0
        assert torch.equal(conv_f, conv_s) and torch.equal(pool_f, pool_s)
        live = (ix >= 0).nonzero().flatten()
        a, b = o_f[live].float(), o_s.reshape(N, Hv, d)[live].float()
        assert ((a - b).norm() / b.norm()).item() <= 1e-3  # the two may contract the output expression into different FMAs
        assert N <= 4 or torch.count_nonzero(o_f[3]) == 0
