"""Performance cases of the framework: its sequence operators, projections and whole-model calls through the public
entry points, at the sizes of the shipped configurations (hidden 4096, 32 heads of 128, filter lengths 3 / 7 / 128, modal
order 16, SwiGLU inner 11264, 8192 tokens) and at smaller, ragged ones.

A case is a plain dict.  `kind` selects the path:

  li        Hyena-LI modal convolution on featurised projections              ops.hyena_li_modal
  mr        Hyena-MR gated FIR of up to 128 taps                              ops.hyena_mr_inner
  se        featuriser convolution (3 taps) followed by Hyena-SE (7 taps)     ops.causal_conv1d, ops.hyena_se_inner
  attn      causal self-attention with rotary embedding, packed projection    ops.attention_packed
  mlp       pre-norm gated MLP of a block, bf16 or fp8 projections            ops.mlp_gated
  head      final norm, logits projection and per-token cross-entropy         ops.rmsnorm, ops.linear, ops.cross_entropy
  model     forward + backward of a small multi-hybrid model                  models.build_model
  generate  prompt prefill, then one decode step per given token              inference.cached.CachedDecoder

`train` selects forward + backward (outputs and all gradients) or the forward alone, as inference runs it.
"""
from __future__ import annotations

import math
import os

import torch
import torch.nn.functional as F

from savanna_b200 import ops

BF = torch.bfloat16
DEV = "cuda"
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
EPS = 1e-6


def listed():
    return [
        # the long-filter layer of the 7B model in training: one 8192-token sequence per GPU
        dict(name="li_train_8k", kind="li", B=1, L=8192, D=4096, order=16, train=True),
        # the same layer over a batch of prompts of an odd length, forward only (prefill of a narrower model)
        dict(name="li_prefill_ragged", kind="li", B=2, L=1237, D=1024, order=16, train=False),
        # the medium-filter layer of the 7B model in training
        dict(name="mr_train_8k", kind="mr", B=1, L=8192, D=4096, G=256, K=128, train=True),
        # the same operator fine-tuning a small model on short sequences of an odd length
        dict(name="mr_train_ragged", kind="mr", B=3, L=777, D=512, G=32, K=128, train=True),
        # featuriser + short-filter layer of the 7B model in training
        dict(name="se_train_8k", kind="se", B=1, L=8192, D=4096, G=256, K=7, train=True),
        # attention layer of the 7B model in training
        dict(name="attn_train_8k", kind="attn", B=1, L=8192, H=32, train=True),
        # attention over a batch of prompts of an odd length, forward only
        dict(name="attn_prefill_ragged", kind="attn", B=2, L=1333, H=16, train=False),
        # gated MLP of the 7B model in training, fp8 projections (the default recipe of the benchmark)
        dict(name="mlp_train_fp8_8k", kind="mlp", B=1, L=8192, D=4096, Fi=11264, fp8=True, train=True),
        # gated MLP of a small model in bf16, odd token count
        dict(name="mlp_train_bf16_ragged", kind="mlp", B=3, L=333, D=1024, Fi=2816, fp8=False, train=True),
        # byte-vocabulary head of the 7B model in training
        dict(name="head_train_8k", kind="head", B=1, L=8192, D=4096, V=512, train=True),
        # one micro-batch of the tiny four-operator model (launch-bound training: tests, sweeps, small fine-tunes)
        dict(name="model_train_tiny", kind="model", B=2, L=1024, D=256, H=2, train=True),
        # a short generation on a small four-operator model: prompt of an odd length, 16 decode steps
        dict(name="generate_small", kind="generate", B=2, L=517, D=1024, H=8, steps=16, train=False),
    ]


def _logint(rng, lo, hi, mult=1):
    """Integer spread evenly over the logarithm of [lo, hi], a multiple of `mult`."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(mult, int(round(v / mult)) * mult)


def draw(rng):
    kind = rng.choice(["li", "mr", "se", "attn", "mlp", "head", "model", "generate"])
    train = rng.random() < 0.6
    if kind in ("li", "mr", "se"):
        D = _logint(rng, 256, 4096, 256)
        L = _logint(rng, 64, 8192)
        B = max(1, min(rng.randint(1, 4), 8192 * 4096 // (L * D)))
        if kind == "li":
            return dict(kind=kind, B=B, L=L, D=D, order=rng.choice([8, 16, 16]), train=train)
        G = D // rng.choice([16, 16, 16, 64])
        return dict(kind=kind, B=B, L=L, D=D, G=G, K=(rng.choice([31, 64, 128, 128]) if kind == "mr" else rng.choice([4, 7])),
                    train=train)
    if kind == "attn":
        L = _logint(rng, 64, 8192)
        H = rng.choice([2, 8, 16, 32])
        B = max(1, min(rng.randint(1, 4), 8192 // L))
        return dict(kind=kind, B=B, L=L, H=H, train=train)
    if kind == "mlp":
        D = _logint(rng, 256, 4096, 128)
        Fi = 128 * max(1, round(D * 2.75 / 128))
        L = _logint(rng, 64, 8192)
        fp8 = rng.random() < 0.5
        if fp8:
            L = max(64, L // 16 * 16)
        return dict(kind=kind, B=1, L=L, D=D, Fi=Fi, fp8=fp8, train=train)
    if kind == "head":
        return dict(kind=kind, B=1, L=_logint(rng, 64, 8192), D=_logint(rng, 256, 4096, 128), V=512, train=train)
    H = rng.choice([2, 4, 8])
    if kind == "model":
        return dict(kind=kind, B=rng.randint(1, 2), L=_logint(rng, 128, 2048, 64), D=128 * H, H=H, train=True)
    return dict(kind=kind, B=rng.randint(1, 4), L=_logint(rng, 33, 1500), D=128 * H, H=H, steps=rng.randint(4, 16), train=False)


# ------------------------------------------------------------------------------------------------ inputs


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _randn(g, *shape, std=1.0, dtype=BF):
    return (torch.randn(*shape, generator=g, device=DEV) * std).to(dtype)


def _mr_decay(G, K):
    # decay rates spread over the channel groups, as the explicit Hyena-MR filter has them ("weak" preset and stronger)
    alpha = torch.logspace(-2, 2, G, device=DEV)[:, None]
    return torch.exp(-alpha * torch.linspace(0, 1, K, device=DEV)[None])


def _model_cfg(case):
    from savanna_b200.config import GlobalConfig
    D, H = case["D"], case["H"]
    cfg = GlobalConfig.from_ymls([os.path.join(ROOT, "configs", "baseline", "tiny_sh2_gpu.yml")],
                                 {"global_num_gpus": 1, "hidden_size": D, "num_attention_heads": H, "num_groups_hyena": D,
                                  "num_groups_hyena_medium": D // 16, "num_groups_hyena_short": D // 16,
                                  "seq_length": 2048, "max_position_embeddings": 2048})
    cfg.build_tokenizer()
    return cfg


def _build_model(case, seed):
    from savanna_b200.models import build_model
    torch.manual_seed(1000 + int(seed))
    model = build_model(_model_cfg(case), device=DEV)
    g = _gen(seed + 5)
    with torch.no_grad():
        for n, p in model.named_parameters():
            # weights of a model in use: filters, biases and gains away from their initial constants
            if n.endswith("filter.h"):
                p.copy_(torch.randn(p.shape, generator=g, device=DEV) / math.sqrt(p.shape[-1]))
            elif n.endswith("bias"):
                p.copy_(torch.randn(p.shape, generator=g, device=DEV) * 0.1)
            elif p.dim() == 1:
                p.copy_(1.0 + 0.1 * torch.randn(p.shape, generator=g, device=DEV))
    return model


def prepare(case, seed):
    g = _gen(seed)
    k = case["kind"]
    st = {"case": case}
    if k in ("li", "mr", "se"):
        B, L, D = case["B"], case["L"], case["D"]
        if k == "li":
            O = case["order"]
            st["args"] = [_randn(g, B, L, 3 * D, std=0.7),
                          (torch.rand(D, O, generator=g, device=DEV) * 0.09 + 0.01).log(),
                          0.1 * _randn(g, D, O, dtype=torch.float32) / math.sqrt(O),
                          -torch.ones(D, O, device=DEV),
                          _randn(g, D, dtype=torch.float32)]
        elif k == "mr":
            G, K = case["G"], case["K"]
            st["args"] = [_randn(g, B, L, 3 * D),
                          _randn(g, G, K, std=1.0 / math.sqrt(K), dtype=torch.float32) * _mr_decay(G, K),
                          _randn(g, D, dtype=torch.float32)]
        else:
            st["args"] = [_randn(g, B, L, 3 * D), _randn(g, 3 * D, 3, std=0.5), _randn(g, case["G"], case["K"], std=0.4)]
        if case["train"]:
            st["gout"] = _randn(g, B, L, D)
    elif k == "attn":
        B, L, H = case["B"], case["L"], case["H"]
        st["args"] = [_randn(g, B, L, H, 3 * 128)]
        inv = 1.0 / (10000.0 ** (torch.arange(0, 128, 2, device=DEV, dtype=torch.float32) / 128))
        ang = torch.outer(torch.arange(L, device=DEV, dtype=torch.float32), inv)
        ang = torch.cat([ang, ang], dim=-1)
        st["cos"], st["sin"] = ang.cos(), ang.sin()
        if case["train"]:
            st["gout"] = _randn(g, B, L, H, 128)
    elif k == "mlp":
        B, L, D, Fi = case["B"], case["L"], case["D"], case["Fi"]
        std = math.sqrt(2.0 / (5.0 * D))
        st["args"] = [_randn(g, B, L, D), (1.0 + 0.1 * _randn(g, D, dtype=torch.float32)).to(BF),
                      _randn(g, 2 * Fi, D, std=std), _randn(g, D, Fi, std=1.0 / math.sqrt(Fi))]
        if case["train"]:
            st["gout"] = _randn(g, B, L, D)
    elif k == "head":
        B, L, D, V = case["B"], case["L"], case["D"], case["V"]
        st["args"] = [_randn(g, B, L, D), (1.0 + 0.1 * _randn(g, D, dtype=torch.float32)).to(BF),
                      _randn(g, V, D, std=1.0 / math.sqrt(D))]
        st["labels"] = torch.randint(0, V, (B, L), generator=g, device=DEV)
        if case["train"]:
            st["gout"] = torch.full((B, L), 1.0 / (B * L), device=DEV)
    else:
        st["model"] = _build_model(case, seed)
        n = case["L"] + (1 if k == "model" else case["steps"])
        # a nucleotide alphabet in byte codes, as the synthetic data of the benchmark has it
        acgt = torch.tensor([65, 67, 71, 84], device=DEV)
        st["tokens"] = acgt[torch.randint(0, 4, (case["B"], n), generator=g, device=DEV)]
        if k == "generate":
            st["model"].eval()
    if "args" in st and case["train"]:
        st["args"] = [torch.nn.Parameter(a) for a in st["args"]]
    if k == "mlp" and case["fp8"]:
        # a running program has its amax histories and quantised weights
        for _ in range(2):
            run(st)
    return st


# ------------------------------------------------------------------------------------------------ one pass


def _operator(st, a):
    case = st["case"]
    k = case["kind"]
    if k == "li":
        return ops.hyena_li_modal(*a)
    if k == "mr":
        return ops.hyena_mr_inner(*a)
    if k == "se":
        return ops.hyena_se_inner(ops.causal_conv1d(a[0], a[1]), a[2])
    if k == "attn":
        return ops.attention_packed(a[0], st["cos"], st["sin"], True)
    if k == "mlp":
        return ops.mlp_gated(a[0], a[1], EPS, "te", a[2], a[3], None, "silu", fp8=case["fp8"])
    st["logits"] = ops.linear(ops.rmsnorm(a[0], a[1], EPS, "te"), a[2])
    return ops.cross_entropy(st["logits"], st["labels"])


def run(st):
    case = st["case"]
    k = case["kind"]
    if k == "generate":
        from savanna_b200.inference.cached import CachedDecoder
        dec = CachedDecoder(st["model"])
        toks, L = st["tokens"], case["L"]
        out = [dec.prefill(toks[:, :L])]
        for i in range(case["steps"]):
            out.append(dec.step(toks[:, L + i]))
        return out
    if k == "model":
        model = st["model"]
        for p in model.parameters():
            p.grad = None
        logits = model(st["tokens"][:, :-1])
        loss = ops.cross_entropy(logits, st["tokens"][:, 1:].contiguous()).mean()
        loss.backward()
        return [loss.detach(), logits.detach()] + [p.grad for p in model.parameters() if p.grad is not None]
    a = st["args"]
    if not case["train"]:
        with torch.no_grad():
            out = _operator(st, a)
        return [out, st["logits"]] if k == "head" else out
    for t in a:
        t.grad = None
    out = _operator(st, a)
    out.backward(st["gout"])
    head = [st["logits"].detach()] if k == "head" else []
    return [out.detach()] + head + [t.grad for t in a]


# ------------------------------------------------------------------------------------------------ cost


def work(case):
    """Bytes: every input and output of the pass once.  Flops: the products of the path (2 per multiply-add); causal
    attention counts the half of the score matrix that it needs, the backward of a product counts two products."""
    k, tr = case["kind"], case["train"]
    B, L = case["B"], case["L"]
    T = B * L
    if k in ("li", "mr", "se"):
        D = case["D"]
        n = T * D
        # features 3 in, 1 out; backward: features and the output's gradient in, the features' gradient out
        by = 8 * n if not tr else 8 * n + 14 * n
        if k == "li":
            O = case["order"]
            # state update and read-out per (time, channel, mode); the backward needs state, sensitivity and adjoint
            fl = 4.0 * n * O * (1 if not tr else 4)
            by += D * O * 12
        elif k == "mr":
            fl = 2.0 * n * case["K"] * (1 if not tr else 4)
        else:
            # the featuriser reads and writes 3 D channels as well, in both directions
            by += 6 * n if not tr else 6 * n + 6 * n
            fl = 2.0 * n * (9 + case["K"]) * (1 if not tr else 3)
        return {"bytes": float(by), "flops": float(fl)}
    if k == "attn":
        n = T * case["H"] * 128
        fl = 4.0 * B * case["H"] * L * L * 128 / 2
        return {"bytes": float(8 * n if not tr else 8 * n + 8 * n + 8 * n), "flops": fl if not tr else 3.5 * fl}
    if k == "mlp":
        D, Fi = case["D"], case["Fi"]
        fl = 2.0 * T * 3 * D * Fi
        by = 4.0 * T * D + 2.0 * 3 * D * Fi
        return {"bytes": by if not tr else 2 * by, "flops": fl if not tr else 3 * fl}
    if k == "head":
        D, V = case["D"], case["V"]
        fl = 2.0 * T * D * V
        by = 2.0 * (T * D + D * V + T * V) + 12.0 * T
        return {"bytes": by if not tr else 2 * by, "flops": fl if not tr else 3 * fl}
    D = case["D"]
    Fi = 16 * math.ceil((8 * D / 3) / 16)
    wts = 4 * (4 * D * D + 3 * D * Fi) + 512 * D
    if k == "model":
        return {"bytes": 2.0 * wts * 2, "flops": 3 * 2.0 * T * wts}
    n = case["steps"]
    return {"bytes": 2.0 * wts * (1 + n), "flops": 2.0 * B * (L + n) * wts}


def tolerance(case):
    """bf16 results: one rounding of the result is 2^-9 of a value at most and 1.7e-3 relative in the 2-norm; paths that
    keep bf16 operands of a tensor-core product inside (attention probabilities, filter taps, gated products) show about
    twice that.  fp8 operands: a value next to a rounding boundary moves by one step of its format."""
    k = case["kind"]
    if k == "mlp" and case["fp8"]:
        return {"rel": 2e-2}
    if k == "model":
        return {"rel": 4e-2}
    if k == "generate":
        return {"rel": 4e-2}
    return {"rel": 1e-2}


# ------------------------------------------------------------------------------------------------ the same in 64 bits


def _d(t):
    return t.detach().double()


def _rms64(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS) * w


def _fir64(u, h):
    """Causal convolution of u [B, L, C] with h [C, n] (h[:, s] multiplies u[t - s]) by a zero-padded real FFT."""
    L, n = u.shape[1], u.shape[1] + h.shape[1]
    y = torch.fft.irfft(torch.fft.rfft(u.transpose(1, 2), n=n) * torch.fft.rfft(h, n=n), n=n)[..., :L]
    return y.transpose(1, 2)


def _modal64(gamma, R, p, L):
    t = torch.arange(L, device=gamma.device, dtype=torch.float64)
    ll = -torch.exp(p) * torch.exp(gamma)
    h = torch.zeros(gamma.shape[0], L, device=gamma.device, dtype=torch.float64)
    for o in range(gamma.shape[1]):
        h = h + R[:, o, None] * torch.exp(ll[:, o, None] * t)
    return h


def _gated64(feat, conv):
    """z = x1 * conv(x2 * v) on interleaved features."""
    u = feat[..., 1::3] * feat[..., 2::3]
    return feat[..., 0::3] * conv(u)


def _rope64(x, cos, sin):
    h = x.shape[-1] // 2
    rot = torch.cat([-x[..., h:], x[..., :h]], dim=-1)
    return x * cos[:, None] + rot * sin[:, None]


def _attn64(qkv, cos, sin):
    """Causal attention on the packed [B, L, H, 3 hd] projection, one head of one batch row at a time."""
    hd = qkv.shape[-1] // 3
    q, k, v = _rope64(qkv[..., :hd], cos, sin), _rope64(qkv[..., hd:2 * hd], cos, sin), qkv[..., 2 * hd:]
    L = qkv.shape[1]
    mask = torch.ones(L, L, dtype=torch.bool, device=qkv.device).triu(1)
    rows = []
    for b in range(qkv.shape[0]):
        heads = []
        for i in range(qkv.shape[2]):
            s = (q[b, :, i] @ k[b, :, i].T) / math.sqrt(hd)
            heads.append(s.masked_fill(mask, float("-inf")).softmax(-1) @ v[b, :, i])
        rows.append(torch.stack(heads, dim=1))
    return torch.stack(rows)


def _model64(model, P, tokens):
    """Logits of the four-operator model (short / medium / long Hyena, attention) in 64 bits from its parameters P."""
    cfg = model.cfg
    H, hd = cfg.num_attention_heads, cfg.hidden_size // cfg.num_attention_heads
    x = P["sequential.0.word_embeddings.weight"][tokens]
    L = tokens.shape[1]
    for i, op in enumerate(cfg.operator_config):
        pre = f"sequential.{i + 2}."
        proj = _rms64(x, P[pre + "input_layernorm.weight"]) @ P[pre + "mixer.dense_projection.weight"].T
        if op.startswith("hyena"):
            w = P[pre + "mixer.hyena_proj_conv.short_conv_weight"].reshape(proj.shape[-1], -1)
            feat = _fir64(proj, w.flip(-1))
            D = feat.shape[-1] // 3
            if op == "hyena_se":
                w = P[pre + "mixer.mixer.short_conv.short_conv_weight"]
                h = w.reshape(w.shape[0], -1).flip(-1)
                bias = torch.zeros(D, device=x.device, dtype=x.dtype)
            else:
                bias = P[pre + "mixer.mixer.conv_bias"]
                fp = pre + "mixer.mixer.filter."
                if op == "hyena_mr":
                    n = min(cfg.hyena_mr_len, L)
                    h = P[fp + "h"][:, :n] * model.state_dict()[fp + "decay"].double()[:, :n]
                else:
                    h = _modal64(P[fp + "gamma"], P[fp + "R"], P[fp + "p"], L)
            h = h.repeat_interleave(D // h.shape[0], dim=0)
            z = _gated64(feat, lambda u: _fir64(u, h) + bias * u)
        else:
            inv = 1.0 / (10000.0 ** (torch.arange(0, hd, 2, device=x.device, dtype=torch.float64) / hd))
            ang = torch.outer(torch.arange(L, device=x.device, dtype=torch.float64), inv)
            ang = torch.cat([ang, ang], dim=-1)
            z = _attn64(proj.view(x.shape[0], L, H, 3 * hd), ang.cos(), ang.sin()).reshape(x.shape)
        a = x + z @ P[pre + "mixer.dense.weight"].T + P[pre + "mixer.dense.bias"]
        m = _rms64(a, P[pre + "pre_mlp_layernorm.weight"]) @ P[pre + "mlp.w12"].T
        f = m.shape[-1] // 2
        x = a + (F.silu(m[..., :f]) * m[..., f:]) @ P[pre + "mlp.w3.weight"].T
        b3 = P.get(pre + "mlp.w3.bias")
        if b3 is not None:
            x = x + b3
    n = len(cfg.operator_config)
    x = _rms64(x, P[f"sequential.{n + 3}.norm.weight"])
    return x @ P["sequential.0.word_embeddings.weight"].T


def exact(case, seed):
    k = case["kind"]
    st = prepare(case, seed)
    if k in ("model", "generate"):
        model = st["model"]
        P = {n: _d(p).requires_grad_(k == "model") for n, p in model.named_parameters()}
        if k == "generate":
            L, n = case["L"], case["steps"]
            with torch.no_grad():
                logits = _model64(model, P, st["tokens"])
            return [logits[:, L - 1 + i] for i in range(n + 1)]
        logits = _model64(model, P, st["tokens"][:, :-1])
        labels = st["tokens"][:, 1:]
        loss = F.cross_entropy(logits.reshape(-1, logits.shape[-1]), labels.reshape(-1))
        loss.backward()
        return [loss.detach(), logits.detach()] + [P[n].grad for n, _ in model.named_parameters() if P[n].grad is not None]
    a = [_d(t).requires_grad_(case["train"]) for t in st["args"]]
    logits = None
    if k == "li":
        h = _modal64(a[1], a[2], a[3], case["L"])
        out = _gated64(a[0], lambda u: _fir64(u, h) + a[4] * u)
    elif k == "mr":
        h = a[1].repeat_interleave(case["D"] // case["G"], dim=0)
        out = _gated64(a[0], lambda u: _fir64(u, h) + a[2] * u)
    elif k == "se":
        h = a[2].flip(-1).repeat_interleave(case["D"] // case["G"], dim=0)
        out = _gated64(_fir64(a[0], a[1].flip(-1)), lambda u: _fir64(u, h))
    elif k == "attn":
        if case["L"] > 4096 and case["train"]:
            return _attn64_train(st, case)
        out = _attn64(a[0], _d(st["cos"]), _d(st["sin"]))
    elif k == "mlp":
        m = _rms64(a[0], a[1]) @ a[2].T
        out = a[0] + (F.silu(m[..., : case["Fi"]]) * m[..., case["Fi"]:]) @ a[3].T
    else:
        logits = _rms64(a[0], a[1]) @ a[2].T
        out = F.cross_entropy(logits.reshape(-1, case["V"]), st["labels"].reshape(-1), reduction="none").view(st["labels"].shape)
    if not case["train"]:
        return [out, logits] if k == "head" else out
    out.backward(st["gout"].double())
    return [out.detach()] + ([logits.detach()] if k == "head" else []) + [t.grad for t in a]


def _attn64_train(st, case):
    """Output and gradient of a long attention case, one head at a time so that one score matrix is alive."""
    qkv, go = _d(st["args"][0]), st["gout"].double()
    cos, sin = _d(st["cos"]), _d(st["sin"])
    out, grad = torch.empty_like(go), torch.empty_like(qkv)
    for b in range(qkv.shape[0]):
        for i in range(qkv.shape[2]):
            x = qkv[b:b + 1, :, i:i + 1].clone().requires_grad_()
            o = _attn64(x, cos, sin)
            o.backward(go[b:b + 1, :, i:i + 1])
            out[b:b + 1, :, i:i + 1], grad[b:b + 1, :, i:i + 1] = o.detach(), x.grad
    return [out, grad]
