"""What this framework's performance is measured on: the work that a training run and a generation loop
have it do, through the layers, the model and the operator front ends that a program calls.

Sizes are those of the benchmark configurations (125M: hidden 768, 12 / 4 heads of 64; 1.3B: hidden 2048, 16 / 4
heads of 128, FFN 5504; 7B: hidden 4096, 32 / 8 heads of 128, FFN 11008; vocabulary 32000) and their neighbours.
``draw`` gives more cases of the same kinds with other batch sizes, lengths (odd ones among them) and widths.

Kinds:
  attn     GroupedQueryAttention forward + backward (projections, rotary embedding, flash attention)
  mlp      SwiGLU forward + backward
  norm     RMSNorm forward + backward with the residual gradient folded in
  head     tied LM head + cross-entropy, forward + backward
  adamw    gradient statistics and clipped AdamW on one ZeRO unit
  decode   one token of each sequence of a batch through one transformer block with its KV cache
  token    one token through a whole model: logits and the caches it extends
  prefill  full-sequence logits of a whole model
  train    loss and all gradients of a whole model
"""
from __future__ import annotations

import math

import torch
from torch.utils.checkpoint import checkpoint

from create_llm_by_cupy_b200.models.layers import (ChunkedCrossEntropy_Share, GroupedQueryAttention, RMSNorm,
                                                   SwiGLU)
from create_llm_by_cupy_b200.models.model import Cupa_ver4
from create_llm_by_cupy_b200.ops import functional as F

DEV = "cuda"
VOCAB = 32000
EPS = 1e-6
ROPE_BASE = 10000.0
# hidden, query heads, KV heads, FFN width, layers, context of the benchmark's models
MODELS = {
    "125m": dict(H=768, QH=12, KVH=4, I=2048, L=12, ctx=1024),
    "1.3b": dict(H=2048, QH=16, KVH=4, I=5504, L=24, ctx=2048),
    "7b": dict(H=4096, QH=32, KVH=8, I=11008, L=32, ctx=4096),
}
# AdamW: the hyper-parameters of the training entry points
ADAM = dict(lr=3e-4, beta1=0.9, beta2=0.95, eps=1e-6, weight_decay=0.1, step=1000, grad_scale=1.0, max_grad_norm=1.0)


# ------------------------------------------------------------------------------------------- the cases
def _attn(model, B, T, ragged):
    m = MODELS[model]
    return dict(kind="attn", B=B, T=T, H=m["H"], QH=m["QH"], KVH=m["KVH"], ragged=ragged)


def _decode(model, B, pos):
    m = MODELS[model]
    return dict(kind="decode", B=B, pos=pos, H=m["H"], QH=m["QH"], KVH=m["KVH"], I=m["I"], ctx=m["ctx"])


def listed():
    return [
        # the attention half of a 1.3B block in training, micro-batch 4 of 2048 packed tokens
        dict(_attn("1.3b", 4, 2048, False), name="attn_1.3b"),
        # the attention half of a 125M block on padded sequences of different lengths
        dict(_attn("125m", 8, 1024, True), name="attn_125m_ragged"),
        # the MLP half of a 1.3B block in training
        dict(kind="mlp", M=8192, H=2048, I=5504, name="mlp_1.3b"),
        # an MLP whose width is left at the layer's default int(8 H / 3): rows of 2730 and 5460 elements
        dict(kind="mlp", M=2048, H=1024, I=0, name="mlp_default_width"),
        # one of the 49 norms of a 1.3B step
        dict(kind="norm", M=8192, H=2048, name="norm_1.3b"),
        # the loss of a 1.3B step; a few targets are padding
        dict(kind="head", M=8192, H=2048, V=VOCAB, name="head_1.3b"),
        # the update of one 1.3B block (a ZeRO unit of 44.3 M parameters), bf16 gradients, fp32 state
        dict(kind="adamw", n=44306432, f32=False, name="adamw_1.3b_unit"),
        # generation with the 1.3B model, late in its context: the latency of one block per token
        dict(_decode("1.3b", 1, 1800), name="decode_1.3b"),
        # batched generation with a 7B model: eight sequences, long context
        dict(_decode("7b", 8, 3000), name="decode_7b_batch8"),
        # one token of a small model, early in its context: launches and latency
        dict(kind="token", model="125m", pos=100, name="token_125m"),
        # scoring one document of odd length
        dict(kind="prefill", model="125m", B=1, T=777, name="prefill_125m"),
        # a whole 125M training pass: micro-batch 8 of 1024 tokens
        dict(kind="train", model="125m", B=8, T=1024, name="train_125m"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attn", "attn", "mlp", "mlp", "norm", "head", "adamw", "decode", "decode", "decode", "token",
                       "prefill", "train"])
    if kind == "attn":
        model = rng.choice(["125m", "1.3b", "7b"])
        T = _log_int(rng, 64, 4096)
        tokens = {"125m": 16384, "1.3b": 8192, "7b": 4096}[model]
        return _attn(model, max(1, min(rng.choice([1, 2, 3, 4, 8]), tokens // T)), T, rng.random() < 0.5)
    if kind == "mlp":
        H, I = rng.choice([(768, 2048), (768, 0), (1024, 0), (1280, 0), (2048, 5504), (4096, 11008)])
        return dict(kind=kind, M=_log_int(rng, 64, 2048 if I == 0 else (4096 if H == 4096 else 8192)), H=H, I=I)
    if kind == "norm":
        return dict(kind=kind, M=_log_int(rng, 1, 16384), H=rng.choice([512, 768, 1024, 2048, 4096]))
    if kind == "head":
        return dict(kind=kind, M=_log_int(rng, 64, 8192), H=rng.choice([768, 1024, 2048]),
                    V=rng.choice([512, 8192, 32000, 32003, 50257]) if rng.random() < 0.5 else VOCAB)
    if kind == "adamw":
        return dict(kind=kind, n=_log_int(rng, 1000, 70_000_000), f32=rng.random() < 0.3)
    if kind == "decode":
        model = rng.choice(list(MODELS))
        return _decode(model, rng.choice([1, 1, 2, 3, 4, 8, 13, 16]), _log_int(rng, 1, MODELS[model]["ctx"] - 1))
    if kind == "token":
        return dict(kind=kind, model="125m", pos=_log_int(rng, 1, 1023))
    if kind == "prefill":
        return dict(kind=kind, model="125m", B=rng.choice([1, 1, 2, 3]), T=_log_int(rng, 16, 1024))
    return dict(kind=kind, model="125m", B=rng.choice([1, 2, 4, 8]), T=_log_int(rng, 64, 1024))


def _ffn(case):
    return case["I"] or int(case["H"] * 8 / 3)


# ------------------------------------------------------------------------------------------- inputs
class _Gen:
    """Seeded normal / integer tensors on the device."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(seed)

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
        t = torch.randn(*shape, device=DEV, generator=self.g)
        return t.mul_(std).add_(mean).to(dtype)

    def ints(self, lo, hi, *shape):
        return torch.randint(lo, hi, shape, device=DEV, generator=self.g, dtype=torch.int32)


def _block_weights(g, H, QH, KVH, I, L):
    """[W_KQV, W_O, W_gate_val, W_out, gamma1, gamma2] with the scales of the layers' initialisers."""
    KV = H // QH * KVH
    s = 1.0 / math.sqrt(H)
    return [g.normal(H, H + 2 * KV, std=s), g.normal(H, H, std=1.0 / math.sqrt(2.0 * H * L)),
            g.normal(H, 2 * I, std=s), g.normal(I, H, std=1.0 / math.sqrt(2.0 * I * L)),
            g.normal(H, std=0.05, mean=1.0), g.normal(H, std=0.05, mean=1.0)]


def _model_weights(g, name):
    m = MODELS[name]
    w = []
    for _ in range(m["L"]):
        w += _block_weights(g, m["H"], m["QH"], m["KVH"], m["I"], m["L"])
    return w + [g.normal(VOCAB, m["H"], std=0.02), g.normal(m["H"], std=0.05, mean=1.0)]


def _inputs(case, seed):
    g = _Gen(seed)
    k = case["kind"]
    if k == "attn":
        B, T, H, QH, KVH = (case[n] for n in ("B", "T", "H", "QH", "KVH"))
        w = _block_weights(g, H, QH, KVH, 8, 12)[:2]
        d = dict(w=w, x=g.normal(B * T, H), res=g.normal(B * T, H), dout=g.normal(B * T, H, std=0.01), valid=None)
        if case["ragged"]:
            d["valid"] = g.ints(T // 2 + 1, T + 1, B)
        return d
    if k == "mlp":
        M, H, I = case["M"], case["H"], _ffn(case)
        return dict(w=_block_weights(g, H, 1, 1, I, 12)[2:4], x=g.normal(M, H), res=g.normal(M, H),
                    dout=g.normal(M, H, std=0.01))
    if k == "norm":
        M, H = case["M"], case["H"]
        return dict(gamma=g.normal(H, std=0.05, mean=1.0), x=g.normal(M, H), dy=g.normal(M, H, std=0.01),
                    add=g.normal(M, H, std=0.01))
    if k == "head":
        M, H, V = case["M"], case["H"], case["V"]
        t = g.ints(1, V, M)
        t[g.ints(0, 50, M) == 0] = 0                     # padding
        return dict(W=g.normal(V, H, std=0.02), x=g.normal(M, H), t=t)
    if k == "adamw":
        n = case["n"]
        return dict(grad=g.normal(n, std=1e-3, dtype=torch.float32 if case["f32"] else torch.bfloat16),
                    m=g.normal(n, std=3e-4, dtype=torch.float32),
                    v=g.normal(n, std=1e-3, dtype=torch.float32).square_().add_(1e-9),
                    master=g.normal(n, std=0.02, dtype=torch.float32))
    if k == "decode":
        B, H, QH, KVH = (case[n] for n in ("B", "H", "QH", "KVH"))
        D = H // QH
        w = _block_weights(g, H, QH, KVH, case["I"], 24)
        kc = g.normal(B, KVH, case["ctx"], D)
        vc = g.normal(B, KVH, case["ctx"], D)
        kc[:, :, case["pos"]:] = 0
        vc[:, :, case["pos"]:] = 0
        return dict(w=w, x=g.normal(B, H), kc=kc, vc=vc)
    m = MODELS[case["model"]]
    w = _model_weights(g, case["model"])
    if k == "token":
        D = m["H"] // m["QH"]
        caches = []
        for _ in range(2 * m["L"]):
            c = g.normal(1, m["KVH"], m["ctx"], D)
            c[:, :, case["pos"]:] = 0
            caches.append(c)
        return dict(w=w, ids=g.ints(1, VOCAB, 1), kc=caches[::2], vc=caches[1::2])
    d = dict(w=w, ids=g.ints(1, VOCAB, case["B"], case["T"]))
    if k == "train":
        d["t"] = g.ints(1, VOCAB, case["B"], case["T"])
        d["valid"] = torch.full((case["B"],), case["T"], dtype=torch.int32, device=DEV)
    return d


def _model(name, weights):
    m = MODELS[name]
    model = Cupa_ver4(dict(vocab_size=VOCAB, hidden_size=m["H"], layer_num=m["L"], time_size=m["ctx"], q_head=m["QH"],
                           kv_head=m["KVH"], ffn_size=m["I"], padding_id=0, dropout_rate=0, half_float=True,
                           dtype="bf16", tie_embeddings=True, rope_base=ROPE_BASE, seed=0), device=DEV)
    model.link_params(weights)
    return model


def prepare(case, seed):
    """The layer, weights, inputs and caches that a program holds before the call."""
    d = _inputs(case, seed)
    d["case"] = case
    k = case["kind"]
    if k == "attn":
        layer = GroupedQueryAttention(case["H"], case["T"], case["QH"], case["KVH"], 12, device=DEV, rope_base=ROPE_BASE)
        layer.params = d.pop("w")
        d["layer"] = layer
    elif k == "mlp":
        layer = SwiGLU(case["H"], 12, device=DEV, ffn_size=case["I"] or None)
        layer.params = d.pop("w")
        d["layer"] = layer
    elif k == "norm":
        layer = RMSNorm(case["H"], device=DEV)
        layer.params = [d.pop("gamma")]
        d["layer"] = layer
    elif k == "head":
        d["layer"] = ChunkedCrossEntropy_Share(0)
    elif k == "adamw":
        d["param"] = d["master"].to(torch.bfloat16)
        d["stats"] = torch.zeros(2, dtype=torch.float32, device=DEV)
    elif k == "decode":
        gqa = GroupedQueryAttention(case["H"], case["ctx"], case["QH"], case["KVH"], 24, device=DEV, rope_base=ROPE_BASE)
        feed = SwiGLU(case["H"], 24, device=DEV, ffn_size=case["I"])
        n1, n2 = RMSNorm(case["H"], device=DEV), RMSNorm(case["H"], device=DEV)
        w = d.pop("w")
        gqa.params, feed.params, n1.params, n2.params = w[:2], w[2:4], [w[4]], [w[5]]
        d["block"] = (gqa, feed, n1, n2)
        d["lens"] = torch.full((case["B"],), case["pos"] + 1, dtype=torch.int32, device=DEV)
    else:
        d["model"] = _model(case["model"], d.pop("w"))
        if k == "token":
            d["lens"] = torch.full((1,), case["pos"] + 1, dtype=torch.int32, device=DEV)
    return d


def _decode_block(block, h, pos, kc, vc, lens):
    gqa, feed, n1, n2 = block
    h = gqa.decode_step(n1.forward(h, False), pos, kc, vc, lens, residual=h)
    return feed.forward(n2.forward(h, False), residual=h, train_flg=False)


def _buckets(grads):
    """One flat gradient per block, then the embedding's and the final norm's."""
    n = 6 * ((len(grads) - 2) // 6)
    return [torch.cat([g.reshape(-1) for g in grads[i:i + 6]]) for i in range(0, n, 6)] + list(grads[n:])


def run(state):
    """One pass, as a training or generation loop makes it."""
    s, case = state, state["case"]
    k = case["kind"]
    if k == "attn":
        out = s["layer"].forward(s["x"], case["B"], case["T"], s["valid"], residual=s["res"])
        dx = s["layer"].backward(s["dout"])
        F.wgrad_join(dx.device)
        return [out, dx, *s["layer"].grads]
    if k == "mlp":
        out = s["layer"].forward(s["x"], residual=s["res"])
        dx = s["layer"].backward(s["dout"])
        F.wgrad_join(dx.device)
        return [out, dx, *s["layer"].grads]
    if k == "norm":
        out = s["layer"].forward(s["x"])
        dx = s["layer"].backward(s["dy"], add=s["add"])
        return [out, dx, *s["layer"].grads]
    if k == "head":
        loss = s["layer"].forward(s["x"], s["t"], s["W"])
        dx = s["layer"].backward(s["W"])
        return [loss, dx, s["layer"].dW]
    if k == "adamw":
        s["stats"].zero_()
        F.grad_stats(s["grad"], s["stats"])
        F.adamw_step(s["grad"], s["m"], s["v"], s["master"], s["param"], stats=s["stats"], **ADAM)
        return [s["stats"], s["m"], s["v"], s["master"], s["param"]]
    if k == "decode":
        h = _decode_block(s["block"], s["x"], case["pos"], s["kc"], s["vc"], s["lens"])
        return [h, s["kc"], s["vc"]]
    m = s["model"]
    if k == "token":
        h = F.embedding_fwd(m.Af_Em_para[0], s["ids"], -1)
        for b in range(m.layernum):
            h = _decode_block(m.block_modules(b), h, case["pos"], s["kc"][b], s["vc"][b], s["lens"])
        logits = F.gemm(m.norm_.forward(h, False), m.Af_Em_para[0], trans_b=True, out_dtype=torch.float32)
        return [logits, *s["kc"], *s["vc"]]
    if k == "prefill":
        return m.logits(s["ids"])
    loss = m.forward(s["ids"], s["t"], s["valid"])
    m.backward(1.0)
    return [loss, *_buckets(m.grads)]


# ------------------------------------------------------------------------------------------- what a pass needs
def _causal_flops(B, T, QH, D):
    """Scores and weighted values of the causal half, one forward."""
    return 4.0 * B * QH * D * T * (T + 1) / 2


def _block_params(m):
    return m["H"] * (2 * m["H"] + 2 * m["H"] // m["QH"] * m["KVH"]) + 3 * m["H"] * m["I"] + 2 * m["H"]


def work(case):
    k = case["kind"]
    if k == "attn":
        B, T, H, QH, KVH = (case[n] for n in ("B", "T", "H", "QH", "KVH"))
        M, D = B * T, H // QH
        wn = H * (H + 2 * KVH * D) + H * H
        return {"bytes": 2.0 * (2 * wn + 5 * M * H), "flops": 6.0 * M * wn + 3.5 * _causal_flops(B, T, QH, D)}
    if k == "mlp":
        M, H, I = case["M"], case["H"], _ffn(case)
        return {"bytes": 2.0 * (6 * H * I + 5 * M * H), "flops": 18.0 * M * H * I}
    if k == "norm":
        M, H = case["M"], case["H"]
        return {"bytes": 2.0 * (5 * M * H + 2 * H), "flops": 14.0 * M * H}
    if k == "head":
        M, H, V = case["M"], case["H"], case["V"]
        return {"bytes": 2.0 * (2 * V * H + 2 * M * H) + 4 * M, "flops": 6.0 * M * H * V}
    if k == "adamw":
        n = case["n"]
        return {"bytes": n * (26.0 + (4 if case["f32"] else 2)), "flops": 18.0 * n}
    if k == "decode":
        m, B = dict(case), case["B"]
        D = case["H"] // case["QH"]
        kv = 2.0 * B * case["KVH"] * D * (case["pos"] + 1)
        return {"bytes": 2.0 * (_block_params(m) + kv + 2 * B * case["H"]),
                "flops": 2.0 * B * _block_params(m) + 4.0 * B * case["H"] * (case["pos"] + 1)}
    m = MODELS[case["model"]]
    H, QH, D, L = m["H"], m["QH"], m["H"] // m["QH"], m["L"]
    n = L * _block_params(m) + VOCAB * H + H
    if k == "token":
        kv = 2.0 * L * m["KVH"] * D * (case["pos"] + 1)
        return {"bytes": 2.0 * (n + kv) + 4.0 * VOCAB, "flops": 2.0 * n + 4.0 * L * H * (case["pos"] + 1)}
    M = case["B"] * case["T"]
    att = L * _causal_flops(case["B"], case["T"], QH, D)
    if k == "prefill":
        return {"bytes": 2.0 * n + 4.0 * M * VOCAB, "flops": 2.0 * M * n + att}
    return {"bytes": 4.0 * n + 8.0 * M, "flops": 6.0 * M * n + 3.5 * att}


def tolerance(case):
    """About four times the distance from the 64-bit result: bf16 outputs alone are 1.7e-3 off by their rounding,
    an output behind several bf16 tensors 2e-3 to 5e-3, one behind twelve blocks 1e-2 to 2e-2."""
    return {"rel": {"adamw": 7e-3, "norm": 7e-3, "decode": 1e-2, "attn": 2e-2, "mlp": 1.5e-2, "head": 1.5e-2}.get(case["kind"], 3e-2)}


# ------------------------------------------------------------------------------------------- 64-bit results
def _rms64(x, gamma):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * gamma


def _rot64(x, pos):
    """Rotary embedding of [..., positions, heads, D] at ``pos``, half-split pairs (j, j + D / 2)."""
    D = x.shape[-1]
    freq = ROPE_BASE ** (-2.0 * torch.arange(D // 2, dtype=torch.float64, device=x.device) / D)
    ang = pos.double()[:, None] * freq
    c, s = torch.cos(ang)[:, None, :], torch.sin(ang)[:, None, :]
    a, b = x[..., :D // 2], x[..., D // 2:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _attn64(x, B, T, QH, KVH, w_kqv, w_o, valid):
    H = x.shape[-1]
    D = H // QH
    kqv = (x @ w_kqv).view(B, T, -1)
    pos = torch.arange(T, device=x.device)
    k = _rot64(kqv[..., :KVH * D].reshape(B, T, KVH, D), pos)
    q = _rot64(kqv[..., KVH * D:KVH * D + H].reshape(B, T, QH, D), pos)
    v = kqv[..., KVH * D + H:].reshape(B, T, KVH, D)
    R = QH // KVH
    q = q.permute(0, 2, 1, 3).reshape(B, KVH, R * T, D)
    s = q @ k.permute(0, 2, 3, 1) / math.sqrt(D)
    ok = pos[None, :] <= pos[:, None]
    ok = ok[None].expand(B, T, T)
    if valid is not None:
        ok = ok & (pos[None, None, :] < valid[:, None, None])
    s = s.view(B, KVH, R, T, T).masked_fill(~ok[:, None, None], float("-inf")).view(B, KVH, R * T, T)
    o = torch.softmax(s, -1) @ v.permute(0, 2, 1, 3)
    return o.view(B, QH, T, D).permute(0, 2, 1, 3).reshape(B * T, H) @ w_o


def _mlp64(x, w_gv, w_out):
    gate, val = (x @ w_gv).chunk(2, -1)
    return (torch.nn.functional.silu(gate) * val) @ w_out


def _block64(h, B, T, QH, KVH, valid, w):
    h = h + _attn64(_rms64(h, w[4]), B, T, QH, KVH, w[0], w[1], valid)
    return h + _mlp64(_rms64(h, w[5]), w[2], w[3])


def _hidden64(case, w, ids, valid):
    """Final normed hidden states [B * T, H] of a whole model."""
    m = MODELS[case["model"]]
    B, T = ids.shape
    h = w[-2][ids.reshape(-1).long()]
    for b in range(m["L"]):
        h = checkpoint(_block64, h, B, T, m["QH"], m["KVH"], valid, w[6 * b:6 * b + 6], use_reentrant=False)
    return _rms64(h, w[-1])


def _loss64(logits, t):
    return torch.nn.functional.cross_entropy(logits, t.reshape(-1).long(), ignore_index=0)


def _step64(h, pos, QH, KVH, kc, vc, w):
    """One token of each sequence through a block; ``kc`` / ``vc`` (64-bit) are extended at ``pos``."""
    B, H = h.shape
    D = H // QH
    kqv = _rms64(h, w[4]) @ w[0]
    at = torch.full((1,), pos, device=h.device)
    k = _rot64(kqv[:, :KVH * D].reshape(B, 1, KVH, D), at)[:, 0]
    q = _rot64(kqv[:, KVH * D:KVH * D + H].reshape(B, 1, QH, D), at)[:, 0]
    kc[:, :, pos], vc[:, :, pos] = k, kqv[:, KVH * D + H:].reshape(B, KVH, D)
    s = q.view(B, KVH, QH // KVH, D) @ kc[:, :, :pos + 1].transpose(2, 3) / math.sqrt(D)
    o = torch.softmax(s, -1) @ vc[:, :, :pos + 1]
    h = h + o.reshape(B, H) @ w[1]
    return h + _mlp64(_rms64(h, w[5]), w[2], w[3])


def exact(case, seed):
    d = _inputs(case, seed)
    k = case["kind"]

    def leaf(t):
        return t.double().requires_grad_(True)

    if k in ("attn", "mlp"):
        x, w0, w1 = leaf(d["x"]), leaf(d["w"][0]), leaf(d["w"][1])
        if k == "attn":
            y = _attn64(x, case["B"], case["T"], case["QH"], case["KVH"], w0, w1, d["valid"])
        else:
            y = _mlp64(x, w0, w1)
        grads = torch.autograd.grad(y, (x, w0, w1), d["dout"].double())
        return [y.detach() + d["res"].double(), *grads]
    if k == "norm":
        x, gamma = leaf(d["x"]), leaf(d["gamma"])
        y = _rms64(x, gamma)
        dx, dg = torch.autograd.grad(y, (x, gamma), d["dy"].double())
        return [y.detach(), dx + d["add"].double(), dg]
    if k == "head":
        x, W = leaf(d["x"]), leaf(d["W"])
        loss = _loss64(x @ W.t(), d["t"])
        return [loss.detach(), *torch.autograd.grad(loss, (x, W))]
    if k == "adamw":
        a = ADAM
        g = d["grad"].double()
        ss = g.square().sum()
        g = g * min(1.0, a["max_grad_norm"] / (math.sqrt(float(ss)) + 1e-6))
        m = d["m"].double() * a["beta1"] + g * (1 - a["beta1"])
        v = d["v"].double() * a["beta2"] + g.square() * (1 - a["beta2"])
        upd = (m / (1 - a["beta1"] ** a["step"])) / ((v / (1 - a["beta2"] ** a["step"])).sqrt() + a["eps"])
        p = d["master"].double() * (1 - a["lr"] * a["weight_decay"]) - a["lr"] * upd
        return [torch.stack([ss, torch.zeros_like(ss)]), m, v, p, p]
    with torch.no_grad():
        if k == "decode":
            kc, vc = d["kc"].double(), d["vc"].double()
            h = _step64(d["x"].double(), case["pos"], case["QH"], case["KVH"], kc, vc, [w.double() for w in d["w"]])
            return [h, kc, vc]
        if k == "token":
            m = MODELS[case["model"]]
            w = [t.double() for t in d["w"]]
            kc, vc = [c.double() for c in d["kc"]], [c.double() for c in d["vc"]]
            h = w[-2][d["ids"].long()]
            for b in range(m["L"]):
                h = _step64(h, case["pos"], m["QH"], m["KVH"], kc[b], vc[b], w[6 * b:6 * b + 6])
            return [_rms64(h, w[-1]) @ w[-2].t(), *kc, *vc]
        if k == "prefill":
            w = [t.double() for t in d["w"]]
            return (_hidden64(case, w, d["ids"], None) @ w[-2].t()).view(case["B"], case["T"], VOCAB)
    w = [leaf(t) for t in d["w"]]
    loss = _loss64(_hidden64(case, w, d["ids"], d["valid"]) @ w[-2].t(), d["t"])
    return [loss.detach(), *_buckets(torch.autograd.grad(loss, w))]
