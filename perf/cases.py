"""The work a user of this framework has it do, as cases that can be timed and whose outputs can be compared.

Every case calls the public entry points the way a serving or training program does.  Head counts follow the Qwen3-Next
layer of the repository's configurations (16 key heads, 32 value heads, head dimension 128, hidden size 2048) and its
head-sharded forms; token counts run from one decoded token to the 131072 tokens of the full block.  All inputs are
made on the GPU from the seed: q and k unit vectors (raw normals where the kernel normalises them), gates
g = -exp(A_log) softplus(a + dt_bias) with A_log ~ U(0, ln 16), beta = sigmoid(N(0, 1)), states N(0, 0.02).
"""
import math
import random

import torch

from avelang_b200 import gdn, gemm
from avelang_b200.block import GdnBlockShard

D = 128
HIDDEN = 2048
DEV = "cuda"


def listed():
    return [
        # one user's token: the smallest call there is, all latency and launch cost
        {"name": "decode_one", "kind": "decode", "n": 1, "hk": 16, "hv": 32, "gated": False, "l2norm": False},
        # a half-empty continuous batch of odd size with the fused gated norm and the in-kernel q/k norm
        {"name": "decode_ragged", "kind": "decode", "n": 37, "hk": 16, "hv": 32, "gated": True, "l2norm": True},
        # the continuous-batching step at its full size: 256 sequences over a pool of 512 slots
        {"name": "decode_pool", "kind": "decode", "n": 256, "hk": 16, "hv": 32, "gated": False, "l2norm": False},
        # a whole decode layer of a serving engine: in-projection, fused layer step, out-projection
        {"name": "decode_layer", "kind": "decode_layer", "n": 64},
        # time to first token of a chat message: one short prompt of odd length, every option on, slot pool written
        {"name": "prefill_short", "kind": "prefill", "b": 1, "t": 203, "seqs": 1, "hk": 16, "hv": 32, "d": 128,
         "gated": True, "l2norm": True, "state": True},
        # the headline layer: one 8192-token prompt with the fused gated norm
        {"name": "prefill_layer", "kind": "prefill", "b": 1, "t": 8192, "seqs": 0, "hk": 16, "hv": 32, "d": 128,
         "gated": True, "l2norm": False, "state": False},
        # the heads one of eight GPUs owns, on a long document
        {"name": "prefill_sharded", "kind": "prefill", "b": 1, "t": 32768, "seqs": 0, "hk": 2, "hv": 4, "d": 128,
         "gated": True, "l2norm": True, "state": False},
        # a packed batch of 64 prompts of very unequal length that continue from states
        {"name": "prefill_packed", "kind": "prefill", "b": 1, "t": 262144, "seqs": 64, "hk": 16, "hv": 32, "d": 128,
         "gated": False, "l2norm": False, "state": True},
        # the small model of the CPU reference: head dimension 64
        {"name": "prefill_d64", "kind": "prefill", "b": 1, "t": 256, "seqs": 0, "hk": 4, "hv": 4, "d": 64,
         "gated": False, "l2norm": False, "state": False},
        # one continuous-batching step: running sequences decode one token each while new prompts are prefilled
        {"name": "mixed_step", "kind": "mixed", "n": 61, "seqs": 3, "t": 1500},
        # one training step of the layer: chunked forward and the gradients of every input
        {"name": "train", "kind": "train", "b": 2, "t": 4096, "hk": 16, "hv": 32, "state": True},
        # the whole block of the largest configuration: in-projection, convolution, gates, delta rule, gated norm
        {"name": "block", "kind": "block", "b": 4, "t": 32768},
    ]


def _log_int(rng, lo, hi):
    """An integer spread evenly over the logarithm of [lo, hi]."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _flag(rng):
    return rng.random() < 0.5


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode_layer", "prefill", "prefill", "prefill", "packed", "d64", "mixed", "train", "block"])
    if kind == "decode":
        hk, hv = rng.choice([(2, 4), (4, 8), (8, 16), (16, 32), (16, 32)])
        return {"kind": "decode", "n": _log_int(rng, 1, 256), "hk": hk, "hv": hv, "gated": _flag(rng), "l2norm": _flag(rng)}
    if kind == "decode_layer":
        return {"kind": "decode_layer", "n": _log_int(rng, 1, 256)}
    if kind == "prefill":  # one dense prompt or a few, all heads or one GPU's share of them
        hk, hv = rng.choice([(2, 4), (4, 8), (8, 16), (16, 32), (16, 32)])
        b = rng.choice([1, 1, 1, 2, 3])
        return {"kind": "prefill", "b": b, "t": _log_int(rng, 33, 32768 // b), "seqs": 0, "hk": hk, "hv": hv, "d": 128,
                "gated": _flag(rng), "l2norm": _flag(rng), "state": _flag(rng)}
    if kind == "packed":
        t = _log_int(rng, 512, 262144)
        return {"kind": "prefill", "b": 1, "t": t, "seqs": _log_int(rng, 1, min(64, t // 64)), "hk": 16, "hv": 32, "d": 128,
                "gated": _flag(rng), "l2norm": _flag(rng), "state": True}
    if kind == "d64":
        h = rng.choice([4, 8, 16])
        return {"kind": "prefill", "b": rng.choice([1, 2]), "t": _log_int(rng, 33, 4096), "seqs": 0, "hk": h, "hv": h, "d": 64,
                "gated": _flag(rng), "l2norm": _flag(rng), "state": _flag(rng)}
    if kind == "mixed":
        return {"kind": "mixed", "n": _log_int(rng, 1, 200), "seqs": _log_int(rng, 1, 8), "t": _log_int(rng, 64, 8192)}
    if kind == "train":
        hk, hv = rng.choice([(4, 8), (8, 16), (16, 32)])
        return {"kind": "train", "b": rng.choice([1, 2]), "t": _log_int(rng, 100, 4096), "hk": hk, "hv": hv, "state": _flag(rng)}
    b = rng.choice([1, 2, 4])
    return {"kind": "block", "b": b, "t": _log_int(rng, 65, 32768)}


# ---------------------------------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _normal(gen, *shape, std=1.0, dtype=torch.bfloat16):
    x = torch.randn(*shape, generator=gen, device=DEV, dtype=dtype)
    return x if std == 1.0 else x.mul_(std)


def _unit(gen, *shape):
    """Unit vectors along the last dimension, in bf16; made in pieces so that large inputs need little extra memory."""
    x = torch.randn(*shape, generator=gen, device=DEV, dtype=torch.bfloat16)
    rows = x.view(-1, shape[-1])
    for part in rows.split(1 << 20):
        part.copy_(torch.nn.functional.normalize(part.float(), dim=-1))
    return x


def _gate(gen, b, t, hv):
    a_log = torch.rand(hv, generator=gen, device=DEV) * math.log(16.0)
    dt_bias = 0.1 * torch.randn(hv, generator=gen, device=DEV)
    a = torch.randn(b, t, hv, generator=gen, device=DEV)
    g = -torch.exp(a_log) * torch.nn.functional.softplus(a + dt_bias)
    beta = torch.sigmoid(torch.randn(b, t, hv, generator=gen, device=DEV))
    return g.contiguous(), beta.contiguous()


def _qkv(gen, b, t, hk, hv, d, raw):
    make = _normal if raw else _unit
    return make(gen, b, t, hk, d), make(gen, b, t, hk, d), _normal(gen, b, t, hv, d)


def _lengths(seed, n, total):
    """n sequence lengths, log-uniform over two decades before they are scaled to sum to total."""
    rng = random.Random(int(seed) * 7919 + n)
    w = [math.exp(rng.uniform(0.0, math.log(128.0))) for _ in range(n)]
    lens = [max(1, int(x * total / sum(w))) for x in w]
    lens[lens.index(max(lens))] += total - sum(lens)
    return lens


def _offsets(lens):
    cu = [0]
    for x in lens:
        cu.append(cu[-1] + x)
    return torch.tensor(cu, dtype=torch.int32, device=DEV)


def _slots(gen, n, slots):
    return torch.randperm(slots, generator=gen, device=DEV)[:n].to(torch.int32).contiguous()


def prepare(case, seed):
    gen = _gen(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind == "decode":
        n, hk, hv = case["n"], case["hk"], case["hv"]
        s["q"], s["k"], s["v"] = _qkv(gen, n, 1, hk, hv, D, case["l2norm"])
        s["g"], s["beta"] = _gate(gen, n, 1, hv)
        s["z"] = _normal(gen, n, 1, hv, D) if case["gated"] else None
        s["w"] = torch.ones(D, device=DEV) if case["gated"] else None
        s["pool"] = _normal(gen, 2 * n, hv, D, D, std=0.02, dtype=torch.float32)
        s["idx"] = _slots(gen, n, 2 * n)
    elif kind == "decode_layer":
        n, hk, hv = case["n"], 16, 32
        conv = 2 * hk * D + hv * D
        s["x"] = _normal(gen, n, HIDDEN)
        s["w_in"] = _normal(gen, 2 * hk * D + 2 * hv * D + 2 * hv, HIDDEN, std=0.02)
        s["w_out"] = _normal(gen, HIDDEN, hv * D, std=0.02)
        s["conv_w"] = _normal(gen, conv, 4, std=0.3)
        s["conv_state"] = _normal(gen, 2 * n, 3, conv)
        s["a_log"] = torch.rand(hv, generator=gen, device=DEV) * math.log(16.0)
        s["dt_bias"] = 0.1 * torch.randn(hv, generator=gen, device=DEV)
        s["w"] = torch.ones(D, device=DEV)
        s["pool"] = _normal(gen, 2 * n, hv, D, D, std=0.02, dtype=torch.float32)
        s["idx"] = _slots(gen, n, 2 * n)
    elif kind == "prefill":
        b, t, hk, hv, d = case["b"], case["t"], case["hk"], case["hv"], case["d"]
        s["q"], s["k"], s["v"] = _qkv(gen, b, t, hk, hv, d, case["l2norm"])
        s["g"], s["beta"] = _gate(gen, b, t, hv)
        s["z"] = _normal(gen, b, t, hv, d) if case["gated"] else None
        s["w"] = torch.ones(d, device=DEV) if case["gated"] else None
        seqs = case["seqs"]
        s["cu"], s["longest"] = None, None
        if seqs:
            lens = _lengths(seed, seqs, t)
            s["cu"], s["longest"] = _offsets(lens), max(lens)
        n = seqs or b
        s["state"] = _normal(gen, n, hv, d, d, std=0.02, dtype=torch.float32) if case["state"] else None
    elif kind == "mixed":
        n, seqs, t, hk, hv = case["n"], case["seqs"], case["t"], 16, 32
        lens = [1] * n + _lengths(seed, seqs, t)
        total = n + t
        s["q"], s["k"], s["v"] = _qkv(gen, 1, total, hk, hv, D, True)
        s["g"], s["beta"] = _gate(gen, 1, total, hv)
        s["z"] = _normal(gen, 1, total, hv, D)
        s["w"] = torch.ones(D, device=DEV)
        s["cu"] = _offsets(lens)
        s["pool"] = _normal(gen, 2 * (n + seqs), hv, D, D, std=0.02, dtype=torch.float32)
        s["idx"] = _slots(gen, n + seqs, 2 * (n + seqs))
    elif kind == "train":
        b, t, hk, hv = case["b"], case["t"], case["hk"], case["hv"]
        s["q"], s["k"], s["v"] = _qkv(gen, b, t, hk, hv, D, False)
        s["g"], s["beta"] = _gate(gen, b, t, hv)
        s["state"] = _normal(gen, b, hv, D, D, std=0.02, dtype=torch.float32) if case["state"] else None
        s["d_o"] = _normal(gen, b, t, hv, D)
        s["d_final"] = _normal(gen, b, hv, D, D, std=0.1, dtype=torch.float32)
        for name in ("q", "k", "v", "g", "beta", "state"):
            if s[name] is not None:
                s[name].requires_grad_(True)
    else:
        b, t, hk, hv = case["b"], case["t"], 16, 32
        conv = 2 * hk * D + hv * D
        s["x"] = _normal(gen, b, t, HIDDEN)
        s["block"] = GdnBlockShard(_normal(gen, 2 * hk * D + 2 * hv * D + 2 * hv, HIDDEN, std=0.02), _normal(gen, conv, 4, std=0.3),
                                   torch.rand(hv, generator=gen, device=DEV) * math.log(16.0),
                                   0.1 * torch.randn(hv, generator=gen, device=DEV), torch.ones(D, device=DEV),
                                   Hk=hk, Hv=hv, dk=D, dv=D, device=DEV)
    return s


# ---------------------------------------------------------------------------------------------------------------- one pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "decode":
        o, pool = gdn.fused_recurrent_gated_delta_rule(s["q"], s["k"], s["v"], s["g"], s["beta"], initial_state=s["pool"],
                                                       use_qk_l2norm_in_kernel=case["l2norm"], state_indices=s["idx"], z=s["z"],
                                                       norm_weight=s["w"])
        return {"o": o, "pool": pool}
    if kind == "decode_layer":
        proj = gemm.gemm_pipeline_transposed_b(s["x"], s["w_in"])
        o = gdn.decode_layer_step(proj, s["conv_w"], s["conv_state"], s["a_log"], s["dt_bias"], s["pool"], s["idx"], Hk=16, Hv=32,
                                  norm_weight=s["w"])
        y = gemm.gemm_pipeline_transposed_b(o.view(case["n"], -1), s["w_out"])
        return {"y": y, "pool": s["pool"], "conv_state": s["conv_state"]}
    if kind == "prefill":
        o, final = gdn.chunk_gated_delta_rule(s["q"], s["k"], s["v"], s["g"], s["beta"], initial_state=s["state"],
                                              output_final_state=True, use_qk_l2norm_in_kernel=case["l2norm"], cu_seqlens=s["cu"],
                                              z=s["z"], norm_weight=s["w"], max_seqlen=s["longest"])
        return {"o": o, "final": final}
    if kind == "mixed":
        o = gdn.mixed_prefill_decode_step(s["q"], s["k"], s["v"], s["g"], s["beta"], s["cu"], case["n"], s["pool"], s["idx"],
                                          use_qk_l2norm_in_kernel=True, z=s["z"], norm_weight=s["w"])
        return {"o": o, "pool": s["pool"]}
    if kind == "train":
        o, final = gdn.GatedDeltaRuleFunction.apply(s["q"], s["k"], s["v"], s["g"], s["beta"], D ** -0.5, s["state"])
        wanted = [s[name] for name in ("q", "k", "v", "g", "beta", "state") if s[name] is not None]
        grads = torch.autograd.grad([o, final], wanted, [s["d_o"], s["d_final"]])
        return {"o": o.detach(), "final": final.detach(), "grads": list(grads)}
    return {"o": s["block"].forward(s["x"])}


# ---------------------------------------------------------------------------------------------------------------- work
def _rule_flops(tokens, hk, hv, d):
    """The delta rule in chunks of 64 tokens: K K^T and Q K^T once per key head; W, U, W H, Q H, P V and K^T V per value head."""
    per_token = hk * 2 * (2 * 64 * d) + hv * (2 * (2 * 64 * d) + 2 * 64 * d + 3 * (2 * d * d))
    return float(tokens) * per_token


def _rule_bytes(tokens, hk, hv, d, gated):
    return float(tokens) * (2 * hk * d * 2 + (3 if gated else 2) * hv * d * 2 + 2 * hv * 4)


def work(case):
    kind = case["kind"]
    state = 4.0 * D * D
    if kind == "decode":
        n, hv = case["n"], case["hv"]
        return {"bytes": _rule_bytes(n, case["hk"], hv, D, case["gated"]) + 2 * n * hv * state, "flops": n * hv * 8.0 * D * D}
    if kind == "decode_layer":
        n, hk, hv = case["n"], 16, 32
        rows, conv = 2 * hk * D + 2 * hv * D + 2 * hv, 2 * hk * D + hv * D
        weights = 2.0 * HIDDEN * (rows + hv * D)
        return {"bytes": weights + 2 * n * hv * state + n * (4.0 * HIDDEN + 2 * 3 * 2 * conv) + 8.0 * conv,
                "flops": n * (weights + hv * 8.0 * D * D)}
    if kind == "prefill":
        d, n, hv = case["d"], case["seqs"] or case["b"], case["hv"]
        tokens = case["b"] * case["t"]
        return {"bytes": _rule_bytes(tokens, case["hk"], hv, d, case["gated"]) + (2 if case["state"] else 1) * n * hv * 4.0 * d * d,
                "flops": _rule_flops(tokens, case["hk"], hv, d)}
    if kind == "mixed":
        n, t, hk, hv = case["n"], case["t"], 16, 32
        return {"bytes": _rule_bytes(n + t, hk, hv, D, True) + 2 * (n + case["seqs"]) * hv * state,
                "flops": _rule_flops(t, hk, hv, D) + n * hv * 8.0 * D * D}
    if kind == "train":
        tokens, hk, hv = case["b"] * case["t"], case["hk"], case["hv"]
        states = case["b"] * hv * state * (4 if case["state"] else 2)
        # forward once; backward reads q, k, v, g, beta, do and writes dq, dk, dv, dg, dbeta, with twice the forward's products
        grads = tokens * (4.0 * hk * D * 2 + 3.0 * hv * D * 2 + 4.0 * hv * 4)
        return {"bytes": _rule_bytes(tokens, hk, hv, D, False) + grads + states, "flops": 3 * _rule_flops(tokens, hk, hv, D)}
    tokens, hk, hv = case["b"] * case["t"], 16, 32
    rows = 2 * hk * D + 2 * hv * D + 2 * hv
    return {"bytes": 2.0 * (tokens * HIDDEN + rows * HIDDEN + tokens * hv * D), "flops": 2.0 * tokens * rows * HIDDEN + _rule_flops(tokens, hk, hv, D)}


def tolerance(case):
    # results are bf16 (rounding 2^-9 of the value) beside fp32 states; where bf16 intermediates (projection, convolution)
    # feed the rule, a rounding of theirs that falls the other way shows in the result
    return {"rel": 1e-2} if case["kind"] in ("decode_layer", "block") else {"rel": 4e-3}
