"""The work that programs on this framework spend their GPU time on, as cases that can be timed and compared.

Each case is one call (or one forward + backward pass) through a public entry point: normalisations, causal
grouped-query attention in training, prefill and decoding, the SwiGLU MLP, the mixture-of-experts layer, the output
head with its loss, and two whole calls of the dense decoder.  Shapes are those of the models that the benchmarks use
(hidden 896 / 14 query and 2 KV heads of 64 / FFN 4864 / vocabulary 151936; 12 / 2 and 16 / 4 heads of 128; experts of
2048 x 768, 128 of them, top 8) and of the kernel sweep.

`exact` restates each case in plain torch at 64 bits.
"""
import math
import os

import torch

# torch's own memory statistics, which a timing program may ask for, exist only with torch's own allocator
os.environ.setdefault("GENESIS_B200_POOL", "0")

import genesis_b200 as genesis  # noqa: E402
import genesis_b200.nn.functional as F  # noqa: E402
from genesis_b200.device import default_device, set_default_device  # noqa: E402
from genesis_b200.models.transformers import QwenForCausalLM, TransformerConfig  # noqa: E402
from genesis_b200.models.transformers.dense import FeedForward  # noqa: E402
from genesis_b200.models.transformers.moe import MoELayer  # noqa: E402

DEV = "cuda"
TYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
AMP = {"bf16": genesis.bfloat16, "fp16": genesis.float16}
VOCAB = 151936
LR = 3e-4


def listed():
    return [
        # the norm of one token-by-token decoding step of a small batch: the smallest call, all latency
        dict(name="norm_decode", kind="norm", rows=8, cols=896, dtype="bf16", train=False),
        # residual addition + RMSNorm of a wide model's training step, both directions
        dict(name="norm_train", kind="norm", rows=8192, cols=4096, dtype="bf16", train=True),
        # one decoding step against a key/value cache: a single query row per sequence
        dict(name="attn_decode", kind="attn", B=8, S=1, Sk=4096, Hq=32, Hkv=4, D=128, dtype="bf16", train=False),
        # prefill of one prompt of ordinary, odd length
        dict(name="attn_prefill", kind="attn", B=1, S=1003, Sk=1003, Hq=14, Hkv=2, D=64, dtype="bf16", train=False),
        # prefill of one long document
        dict(name="attn_long", kind="attn", B=1, S=16384, Sk=16384, Hq=16, Hkv=4, D=128, dtype="bf16", train=False),
        # the attention of the 0.5B-shaped model's training step
        dict(name="attn_train_d64", kind="attn", B=8, S=2048, Sk=2048, Hq=14, Hkv=2, D=64, dtype="bf16", train=True),
        # the attention of the 1.5B-shaped model's fp16 training step
        dict(name="attn_train_d128", kind="attn", B=4, S=4096, Sk=4096, Hq=12, Hkv=2, D=128, dtype="fp16", train=True),
        # the SwiGLU MLP of the 0.5B-shaped model's training step
        dict(name="mlp_train", kind="mlp", tokens=16384, hidden=896, inner=4864, dtype="bf16"),
        # one mixture-of-experts layer in training: routing, grouped expert GEMMs, combination
        dict(name="moe_train", kind="moe", B=2, S=2048, hidden=2048, inner=768, experts=128, top=8, dtype="bf16"),
        # output projection and cross-entropy over the large vocabulary, both directions
        dict(name="head_train", kind="head", tokens=2048, hidden=896, vocab=VOCAB, dtype="bf16"),
        # a whole call: logits of a short, ragged batch of prompts from the 24-layer model
        dict(name="model_prefill", kind="prefill", B=2, S=333, layers=24, dtype="bf16"),
        # a whole call: a training step (forward, backward, AdamW) of the same widths, two layers deep
        dict(name="model_train", kind="train", B=4, S=2048, layers=2, dtype="bf16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["norm", "attn", "attn", "attn", "decode", "mlp", "moe", "head", "prefill", "train"])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    if kind == "norm":
        rows, cols = _log_int(rng, 1, 16384), rng.choice([64, 256, 896, 1000, 1536, 2048, 2051, 4096, 8192, 16384])
        return dict(kind="norm", rows=max(1, min(rows, (1 << 26) // cols)), cols=cols,
                    dtype=rng.choice(["bf16", "fp16", "fp32"]), train=rng.random() < 0.6)
    if kind == "attn":
        Hq, Hkv, D = rng.choice([(14, 2, 64), (12, 2, 128), (16, 4, 128), (32, 4, 128), (4, 4, 64), (4, 4, 128), (6, 3, 64)])
        S = _log_int(rng, 16, 8192)
        B = max(1, min(_log_int(rng, 1, 16), int(4 * 4096 * 4096 * 12 / (S * S * Hq))))
        return dict(kind="attn", B=B, S=S, Sk=S + rng.choice([0, 0, 0, rng.randint(1, 300)]), Hq=Hq, Hkv=Hkv, D=D,
                    dtype=dtype, train=rng.random() < 0.6)
    if kind == "decode":
        Hq, Hkv, D = rng.choice([(14, 2, 64), (12, 2, 128), (16, 4, 128), (32, 4, 128), (4, 4, 64)])
        return dict(kind="attn", B=_log_int(rng, 1, 64), S=rng.choice([1, 1, 1, 2, 5]), Sk=_log_int(rng, 17, 8192), Hq=Hq,
                    Hkv=Hkv, D=D, dtype=dtype, train=False)
    if kind == "mlp":
        hidden, inner = rng.choice([(256, 512), (896, 4864), (1536, 8960)])
        tokens = _log_int(rng, 1, 16384 if hidden < 1536 else 5000)
        return dict(kind="mlp", tokens=tokens, hidden=hidden, inner=inner, dtype=dtype)
    if kind == "moe":
        hidden, inner, experts, top = rng.choice([(2048, 768, 128, 8), (1024, 512, 32, 4), (256, 128, 8, 2)])
        return dict(kind="moe", B=2, S=_log_int(rng, 8, 2048), hidden=hidden, inner=inner, experts=experts, top=top,
                    dtype="bf16")
    if kind == "head":
        hidden, vocab = rng.choice([(896, VOCAB), (896, 32000), (1536, 32000)])
        return dict(kind="head", tokens=_log_int(rng, 16, 2048), hidden=hidden, vocab=vocab, dtype=dtype)
    if kind == "prefill":
        return dict(kind="prefill", B=rng.randint(1, 3), S=_log_int(rng, 4, 400), layers=rng.choice([2, 8, 24]), dtype="bf16")
    return dict(kind="train", B=rng.randint(1, 4), S=_log_int(rng, 256, 2048), layers=rng.choice([1, 2]), dtype="bf16")


# ------------------------------------------------------------------------------------------------
# inputs: made from the seed alone
# ------------------------------------------------------------------------------------------------
class _Maker:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)

    def normal(self, *shape, std=1.0, dtype=torch.float32, mean=0.0):
        x = torch.randn(*shape, device=DEV, dtype=torch.float32, generator=self.g)
        return (x.mul_(std).add_(mean) if (std, mean) != (1.0, 0.0) else x).to(dtype)

    def tokens(self, high, *shape):
        return torch.randint(0, high, shape, device=DEV, generator=self.g)


def _inputs(case, seed):
    """Plain torch tensors of a case, in the order that the framework and the restatement both use them."""
    m, dt = _Maker(seed), TYPES[case["dtype"]]
    k = case["kind"]
    if k == "norm":
        r, c = case["rows"], case["cols"]
        return dict(x=m.normal(r, c, dtype=dt), res=m.normal(r, c, dtype=dt), w=m.normal(c, std=0.1, mean=1.0),
                    gy=m.normal(r, c, dtype=dt))
    if k == "attn":
        B, S, Sk, Hq, Hkv, D = (case[n] for n in ("B", "S", "Sk", "Hq", "Hkv", "D"))
        return dict(q=m.normal(B, S, Hq, D, dtype=dt), k=m.normal(B, Sk, Hkv, D, dtype=dt),
                    v=m.normal(B, Sk, Hkv, D, dtype=dt), do=m.normal(B, S, Hq, D, dtype=dt))
    if k == "mlp":
        T, H, I = case["tokens"], case["hidden"], case["inner"]
        return dict(x=m.normal(T, H, dtype=dt), gate=m.normal(I, H, std=0.02), up=m.normal(I, H, std=0.02),
                    down=m.normal(H, I, std=0.02), gy=m.normal(T, H, dtype=dt))
    if k == "moe":
        B, S, H, I, E = (case[n] for n in ("B", "S", "hidden", "inner", "experts"))
        return dict(x=m.normal(B, S, H, dtype=dt), router=m.normal(E, H, std=0.02), gu=m.normal(E, 2 * I, H, std=0.02),
                    down=m.normal(E, H, I, std=0.02), gy=m.normal(B, S, H, dtype=dt))
    if k == "head":
        return dict(x=m.normal(case["tokens"], case["hidden"], dtype=dt),
                    w=m.normal(case["vocab"], case["hidden"], std=0.02), t=m.tokens(case["vocab"], case["tokens"]))
    cfg = _config(case)
    H, I, d = cfg.hidden_size, cfg.intermediate_size, cfg.head_dim
    nq, nkv = cfg.num_attention_heads * d, cfg.num_key_value_heads * d
    w = {"model.embed_tokens.weight": m.normal(VOCAB, H, std=0.02)}
    for i in range(case["layers"]):
        p = "model.layers.%d." % i
        for name, rows in (("q", nq), ("k", nkv), ("v", nkv)):
            w[p + "self_attn.%s_proj.weight" % name] = m.normal(rows, H, std=0.02)
            w[p + "self_attn.%s_proj.bias" % name] = m.normal(rows, std=0.02)
        w[p + "self_attn.o_proj.weight"] = m.normal(H, nq, std=0.02)
        w[p + "mlp.gate_proj.weight"] = m.normal(I, H, std=0.02)
        w[p + "mlp.up_proj.weight"] = m.normal(I, H, std=0.02)
        w[p + "mlp.down_proj.weight"] = m.normal(H, I, std=0.02)
        w[p + "input_layernorm.weight"] = m.normal(H, std=0.1, mean=1.0)
        w[p + "post_attention_layernorm.weight"] = m.normal(H, std=0.1, mean=1.0)
    w["model.norm.weight"] = m.normal(H, std=0.1, mean=1.0)
    return dict(weights=w, tokens=m.tokens(VOCAB, case["B"], case["S"] + 1))


def _config(case):
    return TransformerConfig(vocab_size=VOCAB, hidden_size=896, intermediate_size=4864, num_hidden_layers=case["layers"],
                             num_attention_heads=14, num_key_value_heads=2, head_dim=64, max_position_embeddings=2048,
                             rope_theta=1e6, norm_eps=1e-6, tie_word_embeddings=True)


def _module(make):
    """A module on the GPU: parameters are drawn there, and tables that are made on the host move there."""
    before = default_device()
    set_default_device(DEV)
    try:
        return make().cuda()
    finally:
        set_default_device(before)


def _leaf(t):
    return genesis.Tensor(t, requires_grad=True)


def prepare(case, seed):
    k, d = case["kind"], _inputs(case, seed)
    s = dict(case=case, kind=k)
    if k == "norm":
        s.update(x=_leaf(d["x"]), res=_leaf(d["res"]), w=_leaf(d["w"]), gy=genesis.Tensor(d["gy"]))
    elif k == "attn":
        s.update({n: _leaf(d[n]) for n in "qkv"}, do=genesis.Tensor(d["do"]))
    elif k == "mlp":
        cfg = TransformerConfig(vocab_size=64, hidden_size=case["hidden"], intermediate_size=case["inner"],
                                num_hidden_layers=1, num_attention_heads=case["hidden"] // 64)
        mod = _module(lambda: FeedForward(cfg))
        for p, n in ((mod.gate_proj, "gate"), (mod.up_proj, "up"), (mod.down_proj, "down")):
            p.weight.copy_(genesis.Tensor(d[n]))
        s.update(mod=mod, x=_leaf(d["x"]), gy=genesis.Tensor(d["gy"]))
    elif k == "moe":
        mod = _module(lambda: MoELayer(case["hidden"], case["experts"], case["top"], case["inner"], aux_loss_alpha=0.0))
        mod.gate.weight.copy_(genesis.Tensor(d["router"]))
        mod.experts.w_gate_up.copy_(genesis.Tensor(d["gu"]))
        mod.experts.w_down.copy_(genesis.Tensor(d["down"]))
        s.update(mod=mod, x=_leaf(d["x"]), gy=genesis.Tensor(d["gy"]))
    elif k == "head":
        s.update(x=_leaf(d["x"]), w=_leaf(d["w"]), t=genesis.Tensor(d["t"]))
    else:
        model = _module(lambda: QwenForCausalLM(_config(case)))
        for n, p in model.named_parameters():
            if n in d["weights"]:
                p.copy_(genesis.Tensor(d["weights"][n]))
        s.update(model=model, idx=genesis.Tensor(d["tokens"][:, :-1].contiguous()))
        if k == "train":
            s.update(labels=genesis.Tensor(d["tokens"][:, 1:].reshape(-1).contiguous()))
            s["opt"] = genesis.optim.AdamW(model.parameters(), lr=LR)
        else:
            model.eval()
    return s


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------
def _out(*tensors):
    return [t._t for t in tensors]


def run(s):
    k, case = s["kind"], s["case"]
    if k == "norm":
        if not case["train"]:
            with genesis.no_grad():
                return _out(F.rms_norm(s["x"], s["w"]))
        for n in ("x", "res", "w"):
            s[n].grad = None
        # a pre-norm block: the sum goes on as the residual stream, its norm into a branch that joins it again
        total, y = F.add_rms_norm(s["x"], s["res"], s["w"])
        out = total + y
        out.backward(s["gy"])
        return _out(out, s["x"].grad, s["res"].grad, s["w"].grad)
    if k == "attn":
        if not case["train"]:
            with genesis.no_grad():
                return _out(F.flash_attention(s["q"], s["k"], s["v"], causal=True))
        for n in "qkv":
            s[n].grad = None
        o = F.flash_attention(s["q"], s["k"], s["v"], causal=True)
        o.backward(s["do"])
        return _out(o, s["q"].grad, s["k"].grad, s["v"].grad)
    if k in ("mlp", "moe"):
        params = list(s["mod"].parameters())
        for p in [s["x"]] + params:
            p.grad = None
        with genesis.amp.autocast(dtype=AMP[case["dtype"]]):
            y = s["mod"](s["x"])
        y.backward(s["gy"])
        return _out(y, s["x"].grad, *[p.grad for p in params])
    if k == "head":
        s["x"].grad = s["w"].grad = None
        with genesis.amp.autocast(dtype=AMP[case["dtype"]]):
            loss = F.cross_entropy(F.linear(s["x"], s["w"]), s["t"], _inplace_backward=True)
        loss.backward()
        return _out(loss, s["x"].grad, s["w"].grad)
    if k == "prefill":
        with genesis.no_grad(), genesis.amp.autocast(dtype=AMP[case["dtype"]]):
            return _out(s["model"](s["idx"]))
    with genesis.amp.autocast(dtype=AMP[case["dtype"]]):
        loss = s["model"](s["idx"], labels=s["labels"], return_logits=False)
    s["opt"].zero_grad()
    loss.backward()
    s["opt"].step()
    # all updated weights, and the gradients of all but the embedding table (the first): a few of its rows, those of the
    # batch's tokens, are so much larger than the rest that no one scale fits it
    params = list(s["model"].parameters())
    return _out(loss, *[p.grad for p in params[1:]], *params)


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------
def _pairs(S, Sk):
    """(query, key) pairs of a causal mask aligned to the end of the keys."""
    return S * (Sk - S) + S * (S + 1) // 2


def work(case):
    k, e = case["kind"], 4 if case["dtype"] == "fp32" else 2
    if k == "norm":
        n = case["rows"] * case["cols"]
        return dict(bytes=(8 if case["train"] else 2) * n * e + 8 * case["cols"], flops=(20 if case["train"] else 4) * n)
    if k == "attn":
        B, S, Sk, Hq, Hkv, D = (case[n] for n in ("B", "S", "Sk", "Hq", "Hkv", "D"))
        q, kv = B * S * Hq * D * e, B * Sk * Hkv * D * e
        f = 4 * B * Hq * D * _pairs(S, Sk)
        if not case["train"]:
            return dict(bytes=2 * q + 2 * kv, flops=f)
        return dict(bytes=4 * q + 4 * kv, flops=3.5 * f)
    if k == "mlp":
        T, H, I = case["tokens"], case["hidden"], case["inner"]
        return dict(bytes=4 * T * H * e + 2 * 3 * H * I * 4, flops=18 * T * H * I)
    if k == "moe":
        T, H, I, E, top = case["B"] * case["S"], case["hidden"], case["inner"], case["experts"], case["top"]
        return dict(bytes=4 * T * H * e + 2 * (3 * H * I * E + E * H) * 4, flops=18 * T * top * H * I + 6 * T * E * H)
    if k == "head":
        T, H, V = case["tokens"], case["hidden"], case["vocab"]
        return dict(bytes=2 * T * H * e + 2 * H * V * 4, flops=6 * T * H * V)
    B, S, L, H, I = case["B"], case["S"], case["layers"], 896, 4864
    per = H * (896 + 256) + 896 * H + 3 * H * I
    f = 2 * B * S * (L * per + H * VOCAB) + 4 * L * B * 14 * 64 * _pairs(S, S)
    n = L * per + H * VOCAB
    if k == "prefill":
        return dict(bytes=n * 4 + B * S * VOCAB * e, flops=f)
    return dict(bytes=28 * n, flops=3 * f + 2 * L * B * 14 * 64 * _pairs(S, S))


def tolerance(case):
    return _TOLERANCE[case["dtype"]] if case["kind"] in ("norm", "attn", "mlp", "head") else dict(rel=2e-2, max=0.5)


# 16-bit results of 32-bit sums: half a unit in the last place is 2^-9 (bf16) or 2^-12 (fp16) of the value, and
# gradients pass through two or three such roundings; fp32 sums in another order
_TOLERANCE = {"bf16": dict(rel=1e-2, max=0.2), "fp16": dict(rel=2e-3, max=0.05), "fp32": dict(rel=1e-5, max=1e-3)}


# ------------------------------------------------------------------------------------------------
# the same in plain torch at 64 bits
# ------------------------------------------------------------------------------------------------
def _attention(q, k, v):
    """Causal attention of one head group: q [g, S, D], k and v [Sk, D]."""
    S, Sk = q.shape[1], k.shape[0]
    s = q @ k.T / math.sqrt(q.shape[-1])
    hidden = torch.ones(S, Sk, dtype=torch.bool, device=q.device).triu_(Sk - S + 1)
    return torch.softmax(s.masked_fill_(hidden, -math.inf), -1) @ v


def _rms_norm(x, w, eps=1e-6):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _swiglu(g, u):
    return torch.nn.functional.silu(g) * u


def _exact_attention(case, d):
    B, S, Hq, D = d["q"].shape
    Hkv = d["k"].shape[2]
    g = Hq // Hkv
    train = case["train"]
    o = torch.empty(B, S, Hq, D, dtype=torch.float64, device=DEV)
    dq, dk, dv = (torch.empty(d[n].shape, dtype=torch.float64, device=DEV) for n in "qkv") if train else (None,) * 3
    step = g if S * d["k"].shape[1] <= 4096 * 4096 else 1
    for b in range(B):
        for h in range(Hkv):
            k, v = (d[n][b, :, h].double().requires_grad_(train) for n in "kv")
            for a in range(h * g, (h + 1) * g, step):
                q = d["q"][b, :, a:a + step].transpose(0, 1).double().requires_grad_(train)
                with torch.set_grad_enabled(train):
                    y = _attention(q, k, v)
                o[b, :, a:a + step] = y.detach().transpose(0, 1)
                if train:
                    y.backward(d["do"][b, :, a:a + step].transpose(0, 1).double())
                    dq[b, :, a:a + step] = q.grad.transpose(0, 1)
            if train:
                dk[b, :, h], dv[b, :, h] = k.grad, v.grad
    return [o, dq, dk, dv] if train else [o]


def _exact_moe(case, d):
    B, S, H = d["x"].shape
    E, top, I = case["experts"], case["top"], case["inner"]
    x = d["x"].reshape(-1, H).double().requires_grad_()
    router, gu, down = (d[n].double().requires_grad_() for n in ("router", "gu", "down"))
    # the selection is discrete: it is made from logits in the compute type, as autocast makes them, ties to the lower
    # index; the weights of the selected experts are those of the unrounded logits
    logits = x @ router.T
    dt = TYPES[case["dtype"]]
    seen = (d["x"].reshape(-1, H).double() @ d["router"].to(dt).double().T).to(dt).float()
    idx = torch.sort(seen, dim=-1, descending=True, stable=True)[1][:, :top]
    w = torch.softmax(logits.gather(1, idx), -1)
    y = torch.zeros_like(x)
    for e in range(E):
        t, slot = (idx == e).nonzero(as_tuple=True)
        if len(t):
            h = x[t] @ gu[e].T
            y = y.index_add(0, t, _swiglu(h[:, :I], h[:, I:]) @ down[e].T * w[t, slot, None])
    y.backward(d["gy"].reshape(-1, H).double())
    return [y.detach().reshape(B, S, H), x.grad.reshape(B, S, H), router.grad, gu.grad, down.grad]


def _exact_model(case, d):
    cfg, train = _config(case), case["kind"] == "train"
    with torch.set_grad_enabled(train):
        w = {n: t.double().requires_grad_(train) for n, t in d["weights"].items()}
        idx = d["tokens"][:, :-1]
        B, S = idx.shape
        D, half = cfg.head_dim, cfg.head_dim // 2
        freq = 1.0 / cfg.rope_theta ** (torch.arange(0, D, 2, dtype=torch.float64, device=DEV) / D)
        angle = torch.outer(torch.arange(S, dtype=torch.float64, device=DEV), freq)
        cos, sin = (torch.cat([f(angle)] * 2, -1)[:, None] for f in (torch.cos, torch.sin))

        def rope(t):
            return t * cos + torch.cat([-t[..., half:], t[..., :half]], -1) * sin

        x = w["model.embed_tokens.weight"][idx]
        for i in range(case["layers"]):
            p = "model.layers.%d." % i
            n = _rms_norm(x, w[p + "input_layernorm.weight"])
            q, k, v = ((n @ w[p + "self_attn.%s_proj.weight" % a].T + w[p + "self_attn.%s_proj.bias" % a]).reshape(B, S, -1, D)
                       for a in "qkv")
            q, k = rope(q), rope(k)
            g = q.shape[2] // k.shape[2]
            o = torch.stack([torch.cat([_attention(q[b, :, h * g:(h + 1) * g].transpose(0, 1), k[b, :, h], v[b, :, h])
                                        for h in range(k.shape[2])]) for b in range(B)])
            x = x + o.transpose(1, 2).reshape(B, S, -1) @ w[p + "self_attn.o_proj.weight"].T
            n = _rms_norm(x, w[p + "post_attention_layernorm.weight"])
            x = x + _swiglu(n @ w[p + "mlp.gate_proj.weight"].T, n @ w[p + "mlp.up_proj.weight"].T) @ w[p + "mlp.down_proj.weight"].T
        x = _rms_norm(x, w["model.norm.weight"])
        if not train:
            return [x @ w["model.embed_tokens.weight"].T]
        # the head in blocks of rows, so that its 64-bit logits are never held at once
        labels, total = d["tokens"][:, 1:].reshape(-1), 0.0
        h, x = x.reshape(B * S, -1), x.detach().reshape(B * S, -1).requires_grad_()
        for a in range(0, B * S, 512):
            part = torch.nn.functional.cross_entropy(x[a:a + 512] @ w["model.embed_tokens.weight"].T, labels[a:a + 512],
                                                     reduction="sum") / (B * S)
            part.backward()
            total += part.detach()
        h.backward(x.grad)
    names = list(d["weights"])
    grads = [w[n].grad for n in names]
    # the first AdamW step: both moments are bias-corrected back to the gradient itself
    after = [w[n].detach() * (1 - LR * 0.01) - LR * w[n].grad / (w[n].grad.abs() + 1e-8) for n in names]
    order = [names.index(n) for n in _parameter_names(case)]
    return [total] + [grads[i] for i in order[1:]] + [after[i] for i in order]


def _parameter_names(case):
    """Parameter names in the order in which the model lists them."""
    names = ["model.embed_tokens.weight"]
    for i in range(case["layers"]):
        p = "model.layers.%d." % i
        names += [p + "self_attn.%s_proj.%s" % (a, b) for a in "qkv" for b in ("weight", "bias")]
        names += [p + n for n in ("self_attn.o_proj.weight", "mlp.gate_proj.weight", "mlp.up_proj.weight",
                                  "mlp.down_proj.weight", "input_layernorm.weight", "post_attention_layernorm.weight")]
    return names + ["model.norm.weight"]


def exact(case, seed):
    k, d = case["kind"], _inputs(case, seed)
    if k == "norm":
        x, res, w = (d[n].double().requires_grad_() for n in ("x", "res", "w"))
        if not case["train"]:
            return [_rms_norm(x, w).detach()]
        # the stream that goes on is of the type of its inputs, and the norm is that of the stream
        total = x + res
        total = total + (total.to(d["x"].dtype).double() - total).detach()
        out = total + _rms_norm(total, w)
        out.backward(d["gy"].double())
        return [out.detach(), x.grad, res.grad, w.grad]
    if k == "attn":
        return _exact_attention(case, d)
    if k == "mlp":
        x, gate, up, down = (d[n].double().requires_grad_() for n in ("x", "gate", "up", "down"))
        y = _swiglu(x @ gate.T, x @ up.T) @ down.T
        y.backward(d["gy"].double())
        return [y.detach(), x.grad, gate.grad, up.grad, down.grad]
    if k == "moe":
        return _exact_moe(case, d)
    if k == "head":
        x, w = d["x"].double().requires_grad_(), d["w"].double().requires_grad_()
        loss = torch.nn.functional.cross_entropy(x @ w.T, d["t"])
        loss.backward()
        return [loss.detach(), x.grad, w.grad]
    return _exact_model(case, d)
