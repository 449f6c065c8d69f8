"""Generation with cached state: one token per step in constant time, instead of re-running the model on the growing context.

Every operator of a StripedHyena 2 block has a small recurrent form:

    featuriser conv (k_f taps)        the last k_f - 1 rows of the in-projection output
    Hyena-SE / Hyena-MR (K taps)      the last K - 1 rows of u = x2 v           (a FIR filter needs nothing older)
    Hyena-LI (modal filter, order O)  the O modal states per channel, s <- lam s + u, y = R . s + bias u
    attention                         the keys (rotary embedding applied) and values of all previous tokens

`CachedDecoder.prefill(tokens)` runs the model's ordinary parallel forward over the prompt once and collects those states
from the layers' inputs (forward pre-hooks; the Hyena-LI state comes from the scan kernel's `return_state`);
`CachedDecoder.step(token)` then advances all layers by one position.  Role of the reference's cached inference path
(savanna/text_generation_utils.py:173-365 `stream_tokens` with `InferenceParams`, :672-774 the interactive driver; its
recurrent Hyena inference lives in the separate vortex project).  Decode steps are matrix-vector work on one token: on CUDA
one native call per step runs five kernels per layer (csrc/decode.cu, see `_FusedStep` for what it covers); everything else
uses plain PyTorch operations on the model's own parameters.  Supported: one device (no tensor / context / pipeline
parallelism), pre-norm blocks with the gated MLP, rotary or no position embedding, implicit-modal Hyena-LI filters; any
other configuration raises and the caller falls back to `stream_tokens` (recompute).
"""
from __future__ import annotations

import ctypes
import math
from typing import Dict, List, Optional

import torch
import torch.nn.functional as F

from ..models.filters import ExplicitSingleDecayFilter, ImplicitModalFilter
from ..models.hyena import HyenaOperator, ShortHyenaOperator
from ..models.mixer import SelfAttention
from ..models.mlp import ParallelGLU
from ..ops import reference as ref
from ..parallel import state


def _rms(x, norm):
    return ref.rmsnorm(x, norm.gain, norm.eps, norm.form) if hasattr(norm, "gain") else norm(x)


def _act(name: str):
    return {"silu": F.silu, "gelu": F.gelu, "relu": F.relu, "identity": lambda t: t}[name]


class _DecLayer(ctypes.Structure):
    """Mirrors sb::dec::Layer (csrc/decode.cu)."""
    _fields_ = ([(n, ctypes.c_int) for n in ("kind", "H", "F", "kf", "K", "G", "O", "heads", "rd", "act", "pregate", "postgate",
                                             "form1", "form2", "norm2", "cap", "f32", "conv_g", "tap_ld", "newest_first")]
                + [(n, ctypes.c_float) for n in ("eps1", "eps2", "pos_scale")]
                + [(n, ctypes.c_void_p) for n in ("norm1_w", "w_in", "w_out", "b_out", "norm2_w", "w12", "w3", "b3", "conv_w", "taps",
                                                  "decay", "bias", "gamma", "p", "R", "inv_freq", "proj_ring", "u_ring", "state",
                                                  "kc", "vc")])


_F32 = {n: 1 << i for i, n in enumerate(("conv_w", "taps", "decay", "bias", "gamma", "p", "R"))}     # bits of _DecLayer.f32


def _ring(tail: torch.Tensor, pos: int) -> torch.Tensor:
    """[B, n, C] rows of times pos - n .. pos - 1, oldest first -> the same rows with time t in slot t mod n."""
    n = tail.shape[1]
    return torch.roll(tail, pos % n, dims=1).contiguous() if n else tail.contiguous()


class _FusedStep:
    """The decode step of csrc/decode.cu: the layers' weights by address, their state in the layout of its kernels.  Built at
    the end of a prefill and after the state was handed out (`CachedDecoder.states`); `build` returns None when something is not
    covered (CPU tensors, other dtypes than bf16, other norms than RMSNorm, head sizes other than 128, more than 8 sequences, an
    inner size above `sb_decode_max_width`: 102400 for one sequence, 12800 for eight; unaligned or non-contiguous weights), and the
    decoder then steps operator by operator."""

    @staticmethod
    def build(dec: "CachedDecoder", batch: int):
        from .. import ops
        from ..models.norms import RMSNorm
        model, cfg = dec.model, dec.cfg
        w = model.embedding.word_embeddings.weight
        if not ops._k(w) or cfg.params_dtype != torch.bfloat16:
            return None
        from ..ops import cuda_ops
        lib = cuda_ops.require()
        if not getattr(lib, "_sb_decode_ready", False):
            P, I, F_ = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
            lib.sb_decode_max_width.restype = lib.sb_decode_layer_bytes.restype = lib.sb_decode_step.restype = I
            lib.sb_decode_max_width.argtypes = [I]
            lib.sb_decode_layer_bytes.argtypes = []
            lib.sb_decode_step.argtypes = [P, I, P, P, P, P, P, I, I, I, P, F_, I, P, I, P, P]
            lib._sb_decode_ready = True
        if lib.sb_decode_layer_bytes() != ctypes.sizeof(_DecLayer):
            raise RuntimeError("decode layer descriptor does not match the native library (rebuild savanna_b200.csrc)")
        D, wmax = cfg.hidden_size, lib.sb_decode_max_width(batch)
        if len(dec._states) != len(dec.blocks):
            return None

        def weight(t, *shape):
            return (t is not None and t.dtype == torch.bfloat16 and t.is_cuda and t.is_contiguous() and t.data_ptr() % 16 == 0
                    and tuple(t.shape) == shape)

        def norm(m):
            return isinstance(m, RMSNorm) and weight(m.gain, D)

        def source(t, *shape):                  # a filter parameter, read as it is stored
            return t.dtype in (torch.bfloat16, torch.float32) and t.is_cuda and t.is_contiguous() and tuple(t.shape) == shape

        def held(t, *shape):                    # a piece of state, whoever filled the dictionary
            return t is not None and t.device == w.device and tuple(t.shape) == (batch,) + shape

        def filters(mixer, st):
            conv, op, H = mixer.hyena_proj_conv, mixer.mixer, mixer.inner_size
            if not source(conv.taps(), conv.num_groups, conv.kernel_size) or conv.num_groups * conv.group_dim != 3 * H \
                    or not held(st.get("proj_tail"), conv.kernel_size - 1, 3 * H) or st["proj_tail"].dtype != torch.bfloat16:
                return False
            if isinstance(op, ShortHyenaOperator):
                return (source(op.short_conv.taps(), op.num_groups, op.kernel_size) and op.num_groups * op.group_dim == H
                        and held(st.get("u_tail"), op.kernel_size - 1, H))
            if not source(op.conv_bias, H) or op.num_groups * op.group_dim != H:
                return False
            if op.is_mr:
                f, G, K = op.filter, op.num_groups, op.hyena_mr_len
                if not held(st.get("u_tail"), K - 1, H):
                    return False
                if type(f) is not ExplicitSingleDecayFilter:
                    return tuple(f(K).shape) == (G, K)
                return f.h.dim() == 2 and f.h.shape[1] >= K and all(source(t, G, f.h.shape[1]) for t in (f.h, f.decay))
            O = op.filter.gamma.shape[1]
            return held(st.get("s"), H, O) and all(source(t, op.num_groups, O) for t in (op.filter.gamma, op.filter.p, op.filter.R))

        for blk, st in zip(dec.blocks, dec._states):
            mixer, mlp = blk.mixer, blk.mlp
            H, Fi = mixer.inner_size, mlp.ffn_local
            if (D % 8 or H % 8 or Fi % 8 or max(D, H, Fi) > wmax or mlp.act not in cuda_ops._ACT or not norm(blk.input_layernorm)
                    or (blk.pre_mlp_norm and not norm(blk.pre_mlp_layernorm)) or not weight(mixer.dense_projection.weight, 3 * H, D)
                    or not weight(mixer.dense.weight, D, H) or not weight(mlp.w12, 2 * Fi, D) or not weight(mlp.w3.weight, D, Fi)
                    or any(b is not None and not weight(b, D) for b in (mixer.dense.bias, mlp.w3.bias))):
                return None
            if isinstance(mixer.mixer, SelfAttention):
                heads = mixer.mixer.heads
                if mixer.mixer.hd != 128 or heads * 128 != H or not all(
                        held(st.get(n), dec.pos, heads, 128) and st[n].dtype == torch.bfloat16 for n in ("k", "v")):
                    return None
            elif not filters(mixer, st):
                return None
        return _FusedStep(dec, lib, batch)

    def __init__(self, dec: "CachedDecoder", lib, batch: int):
        from ..models.norms import RMSNorm
        from ..ops import cuda_ops
        model, cfg = dec.model, dec.cfg
        self.lib, self.model, self.batch, self.D = lib, model, batch, cfg.hidden_size
        dev = model.embedding.word_embeddings.weight.device
        n = len(dec.blocks)
        self.layers = (_DecLayer * n)()
        self.keep = []                          # buffers the descriptors point into
        self.weights = []                       # (descriptor, field, parameter): followed when a parameter's storage moves
        self.filters = []                       # (descriptor, module, taps): filters without a form of their own in the kernel
        self.attn = []                          # (layer index, key cache, value cache)
        self.rings = []                         # (layer index, name of the state, buffer) of the Hyena layers
        self.pos = dec.pos

        def own(t):
            self.keep.append(t)
            return t.data_ptr()

        def ring(i, name, t):
            self.rings.append((i, name, t))
            return t.data_ptr()

        def weight(L, **fields):
            for name, p in fields.items():
                if p is not None:
                    self.weights.append((L, name, p))
                    L.f32 |= _F32.get(name, 0) if p.dtype == torch.float32 else 0

        wide = 0
        for i, (blk, st) in enumerate(zip(dec.blocks, dec._states)):
            L, mixer, inner, mlp = self.layers[i], blk.mixer, blk.mixer.mixer, blk.mlp
            L.H, L.F, L.act = mixer.inner_size, mlp.ffn_local, cuda_ops._ACT[mlp.act]
            L.eps1, L.form1 = blk.input_layernorm.eps, int(blk.input_layernorm.form != "te")
            L.norm2 = int(bool(blk.pre_mlp_norm))
            if L.norm2:
                m = blk.pre_mlp_layernorm
                L.eps2, L.form2 = m.eps, int(m.form != "te")
                weight(L, norm2_w=m.gain)
            weight(L, norm1_w=blk.input_layernorm.gain, w_in=mixer.dense_projection.weight, w_out=mixer.dense.weight,
                   b_out=mixer.dense.bias, w12=mlp.w12, w3=mlp.w3.weight, b3=mlp.w3.bias)
            wide = max(wide, L.H, L.F)
            if isinstance(inner, SelfAttention):
                L.kind, L.heads, L.rd, L.pos_scale = 3, inner.heads, 0, 1.0
                if inner._rotary:
                    r = inner._rotary[0]
                    L.rd, L.pos_scale = r.dim, r.scaling_factor
                    L.inv_freq = own(1.0 / (r.base ** (torch.arange(0, r.dim, 2, device=dev, dtype=torch.float32) / r.dim)))
                self.attn.append([i, st["k"], st["v"]])
            else:
                conv = mixer.hyena_proj_conv
                L.kf, L.conv_g = conv.kernel_size, conv.num_groups
                weight(L, conv_w=conv.short_conv_weight)
                L.proj_ring = ring(i, "proj_tail", _ring(st["proj_tail"].to(torch.bfloat16), dec.pos))
                L.pregate = L.postgate = 1
                L.G = inner.num_groups
                if isinstance(inner, ShortHyenaOperator):
                    L.kind, L.pregate, L.postgate = 0, int(bool(inner.pregate)), int(bool(inner.postgate))
                    L.K = L.tap_ld = inner.kernel_size
                    weight(L, taps=inner.short_conv.short_conv_weight)
                    L.u_ring = ring(i, "u_tail", _ring(st["u_tail"].float(), dec.pos))
                elif inner.is_mr:
                    L.kind, L.newest_first, L.K = 1, 1, st["u_tail"].shape[1] + 1
                    weight(L, bias=inner.conv_bias)
                    if type(inner.filter) is ExplicitSingleDecayFilter:
                        L.tap_ld = inner.filter.h.shape[1]
                        weight(L, taps=inner.filter.h, decay=inner.filter.decay)
                    else:
                        L.tap_ld, L.f32 = L.K, L.f32 | _F32["taps"]
                        self.filters.append([L, inner.filter, None])
                    L.u_ring = ring(i, "u_tail", _ring(st["u_tail"].float(), dec.pos))
                else:
                    L.kind, L.O = 2, inner.filter.gamma.shape[1]
                    weight(L, bias=inner.conv_bias, gamma=inner.filter.gamma, p=inner.filter.p, R=inner.filter.R)
                    L.state = ring(i, "s", st["s"].float().contiguous().clone())
        self._reserve(dec.pos + 1)
        bf = dict(dtype=torch.bfloat16, device=dev)
        self.proj, self.z, self.ab = torch.empty(batch, 3 * wide, **bf), torch.empty(batch, wide, **bf), torch.empty(batch, 2 * wide, **bf)
        self.a = torch.empty(batch, self.D, **bf)
        fn = model.final_norm.norm if hasattr(model.final_norm, "norm") else None
        head = model.embedding.word_embeddings.weight
        self.head = None
        if (not cfg.no_weight_tying and model.mup_output_mult == 1.0 and isinstance(fn, RMSNorm) and fn.gain.dtype == torch.bfloat16
                and head.dtype == torch.bfloat16 and head.is_contiguous() and head.data_ptr() % 16 == 0):
            self.head, self.norm = head, fn
        dec._states = [dict() for _ in dec.blocks]          # this object holds the state from here on

    def _reserve(self, n: int) -> None:
        """Room for n tokens in every key / value cache (doubled when it runs out)."""
        for e in self.attn:
            i, k, v = e
            L = self.layers[i]
            if L.cap >= n:
                continue
            cap = max(2 * L.cap, n + 63)
            for j, (name, old) in enumerate((("kc", k), ("vc", v))):
                new = torch.empty((old.shape[0], cap) + tuple(old.shape[2:]), dtype=torch.bfloat16, device=old.device)
                new[:, : self.pos] = old[:, : self.pos]
                setattr(L, name, new.data_ptr())
                e[1 + j] = new
            L.cap = cap

    def export(self) -> List[Dict]:
        """The state as the operator-by-operator step keeps it, in tensors that later steps leave alone (they only append to
        the key / value caches)."""
        out: List[Dict] = [dict() for _ in self.layers]
        for i, name, t in self.rings:
            n = t.shape[1]
            out[i][name] = t.clone() if name == "s" or n == 0 else torch.roll(t, -(self.pos % n), dims=1)
        for i, k, v in self.attn:
            out[i]["k"], out[i]["v"] = k[:, : self.pos], v[:, : self.pos]
        return out

    def __call__(self, token: torch.Tensor) -> torch.Tensor:
        from ..ops.cuda_ops import _check, _count, _stream
        if token.shape[0] != self.batch:
            raise ValueError(f"decode step for {token.shape[0]} sequences, prefilled with {self.batch}")
        self._reserve(self.pos + 1)
        for L, name, p in self.weights:
            ptr = p.data_ptr()
            if getattr(L, name) != ptr:
                setattr(L, name, ptr)
        for e in self.filters:
            e[2] = e[1](e[0].K).float().contiguous()
            e[0].taps = e[2].data_ptr()
        x = self.model.embedding(token[:, None], None)[:, 0].contiguous()
        V = self.head.shape[0] if self.head is not None else 0
        out = torch.empty(self.batch, V, dtype=torch.float32, device=x.device) if V else None
        _check(self.lib.sb_decode_step(ctypes.addressof(self.layers), len(self.layers), x.data_ptr(), self.proj.data_ptr(),
                                       self.z.data_ptr(), self.a.data_ptr(), self.ab.data_ptr(), self.batch, self.D, self.pos,
                                       self.norm.gain.data_ptr() if V else None, self.norm.eps if V else 0.0,
                                       int(self.norm.form != "te") if V else 0, self.head.data_ptr() if V else None, V,
                                       out.data_ptr() if V else None, _stream()), "decode_step")
        _count(5 * len(self.layers) + (1 if V else 0))
        self.pos += 1
        return out if V else self.model.logits(x[:, None])[:, 0].float()


class CachedDecoder:
    def __init__(self, model):
        cfg = model.cfg
        if state.get_model_parallel_world_size() > 1 or state.get_context_parallel_world_size() > 1 or \
                getattr(model, "is_pipeline_stage", False):
            raise NotImplementedError("cached generation runs on one device")
        if not cfg.prenorm or cfg.postnorm or cfg.outer_mlp_norm or cfg.gpt_j_residual:
            raise NotImplementedError("cached generation supports pre-norm blocks")
        if cfg.pos_emb not in ("rotary", "rotary_linear_scaled", "rotary_ntk_scaled", "rotary2", "none", None):
            raise NotImplementedError(f"cached generation does not support pos_emb={cfg.pos_emb!r}")
        self.model, self.cfg = model, cfg
        self.blocks = model.blocks()
        for b in self.blocks:
            if not isinstance(b.mlp, ParallelGLU):
                raise NotImplementedError("cached generation supports the gated MLP")
            if getattr(b.mixer, "tie_projections", False) or getattr(b.mixer, "proj_groups", 1) > 1:
                raise NotImplementedError("cached generation expects the full-width (3 x hidden) in-projection")
            m = b.mixer.mixer
            if isinstance(m, HyenaOperator) and not m.is_mr and not isinstance(m.filter, ImplicitModalFilter):
                raise NotImplementedError("cached generation needs the implicit modal filter for Hyena-LI")
            if getattr(m, "sparse", False):
                raise NotImplementedError("cached generation does not cover the block-sparse attention operators")
            if isinstance(m, HyenaOperator) and (m.bidirectional or m.slow_heads):
                raise NotImplementedError("cached generation does not cover two-sided filters or outer-product heads")
        self._states: List[Dict] = []
        self.pos = 0
        self._fused: Optional[_FusedStep] = None
        self._resume = False                     # the native step takes the state up again at the next token

    @property
    def states(self) -> List[Dict]:
        """The state of every layer at position `pos`, a dictionary of tensors each.  A step replaces the entries and changes no
        tensor, so a continuation is branched by copying the dictionaries (or the decoder) and resumed by assigning them
        together with `pos`.  Taking the list out of a decoder that steps natively copies the state once: read it again after
        further steps."""
        self._hand_back()
        return self._states

    @states.setter
    def states(self, value: List[Dict]) -> None:
        self._states, self._fused, self._resume = value, None, True

    def _hand_back(self) -> None:
        if self._fused is not None:
            self._states, self._fused, self._resume = self._fused.export(), None, True

    def __getstate__(self):                      # copies: the native step's buffers stay with this decoder
        d = dict(self.__dict__)
        if self._fused is not None:
            d["_states"], d["_fused"], d["_resume"] = self._fused.export(), None, True
        return d

    # ------------------------------------------------------------------ prefill
    @torch.no_grad()
    def prefill(self, tokens: torch.Tensor) -> torch.Tensor:
        """tokens [B, T] -> logits of the last position [B, V]; leaves every layer's state at position T."""
        from .. import ops
        model = self.model
        B, T = tokens.shape
        self._fused, self._resume = None, False
        self._states = [dict() for _ in self.blocks]
        hooks = []

        def tail(x, n):
            """Last n rows of x [B, T, C], zero-padded on the left when the prompt is shorter."""
            if n <= 0:
                return x[:, :0]
            if x.shape[1] >= n:
                return x[:, -n:].clone()
            return F.pad(x, (0, 0, n - x.shape[1], 0))

        for st, blk in zip(self._states, self.blocks):
            mixer = blk.mixer
            inner = mixer.mixer
            if isinstance(inner, SelfAttention):
                def grab_kv(mod, args, st=st):
                    qkv, positions = args[0], args[1]
                    Bq, L, _ = qkv.shape
                    qkv = qkv.view(Bq, L, mod.heads, 3 * mod.hd)
                    k, v = qkv[..., mod.hd: 2 * mod.hd], qkv[..., 2 * mod.hd:]
                    if mod._rotary:
                        cos, sin = mod._rotary[0](positions)
                        k = ref.apply_rope(k.float(), cos, sin).to(qkv.dtype)
                    st["k"], st["v"] = k.clone(), v.clone()
                hooks.append(inner.register_forward_pre_hook(grab_kv))
            else:
                kf = mixer.short_conv_L

                def grab_proj(mod, args, st=st, kf=kf):
                    st["proj_tail"] = tail(args[0], kf - 1)
                hooks.append(mixer.hyena_proj_conv.register_forward_pre_hook(grab_proj))

                def grab_feat(mod, args, st=st):
                    feat = args[0]
                    u = feat[..., 1::3] * feat[..., 2::3]
                    if isinstance(mod, ShortHyenaOperator):
                        st["u_tail"] = tail(u if mod.pregate else feat[..., 2::3], mod.kernel_size - 1)
                    elif mod.is_mr:
                        st["u_tail"] = tail(u, min(mod.hyena_mr_len, 1 << 30) - 1)
                    else:
                        g, R, p = mod._modal()
                        _, s = ops.hyena_li_modal(feat, g, R, p, mod.conv_bias, None, True)
                        st["s"] = s.float()
                hooks.append(inner.register_forward_pre_hook(grab_feat))
        was_training = model.training
        switch = any(m.training for m in model.modules())          # a model in eval mode is left alone
        if switch:
            model.eval()
        try:
            logits = model(tokens)[:, -1].float()
        finally:
            for h in hooks:
                h.remove()
            if switch:
                model.train(was_training)
        self.pos = T
        self._fused = _FusedStep.build(self, B)
        return logits

    # ------------------------------------------------------------------ one decode step
    def _hyena_step(self, blk, st, proj):
        """proj [B, 3D] (in-projection of the new token) -> z [B, D]."""
        mixer, inner = blk.mixer, blk.mixer.mixer
        conv = mixer.hyena_proj_conv
        w = conv.taps().float()
        if conv.group_dim > 1:
            w = w.repeat_interleave(conv.group_dim, dim=0)
        window = torch.cat([st["proj_tail"].float(), proj[:, None].float()], dim=1)          # [B, kf, 3D], oldest first
        feat = torch.einsum("bkc,ck->bc", window, w)
        st["proj_tail"] = window[:, 1:].to(proj.dtype)
        feat = feat.to(proj.dtype).float()                 # the parallel path rounds the featuriser output to the model dtype
        x1, x2, v = feat[:, 0::3], feat[:, 1::3], feat[:, 2::3]
        u = x2 * v
        if isinstance(inner, ShortHyenaOperator):
            un = u if inner.pregate else v
            w = inner.short_conv.taps().float().repeat_interleave(inner.group_dim, dim=0)    # [D, K] correlation order
            window = torch.cat([st["u_tail"].float(), un[:, None]], dim=1)
            y = torch.einsum("bkc,ck->bc", window, w)
            st["u_tail"] = window[:, 1:]
            return (x1 * y) if inner.postgate else y
        if inner.is_mr:
            K = st["u_tail"].shape[1] + 1
            h = inner.filter(K).float().repeat_interleave(inner.group_dim, dim=0)            # [D, K] convolution order
            window = torch.cat([st["u_tail"].float(), u[:, None]], dim=1)
            y = torch.einsum("bkc,ck->bc", window, h.flip(-1)) + inner.conv_bias.float() * u
            st["u_tail"] = window[:, 1:]
            return x1 * y
        g, R, p = inner._modal()
        lam = torch.exp(-torch.exp(p.float()) * torch.exp(g.float()))                         # [D, O]
        s = lam * st["s"] + u[..., None]
        st["s"] = s
        y = (R.float() * s).sum(-1) + inner.conv_bias.float() * u
        return x1 * y

    def _attention_step(self, blk, st, proj):
        inner = blk.mixer.mixer
        B = proj.shape[0]
        qkv = proj.view(B, 1, inner.heads, 3 * inner.hd)
        q, k, v = qkv[..., : inner.hd], qkv[..., inner.hd: 2 * inner.hd], qkv[..., 2 * inner.hd:]
        if inner._rotary:
            pos = torch.tensor([self.pos], device=proj.device)
            cos, sin = ref.rope_tables(pos, inner._rotary[0].dim, inner._rotary[0].base, inner._rotary[0].scaling_factor)
            q = ref.apply_rope(q.float(), cos, sin).to(proj.dtype)
            k = ref.apply_rope(k.float(), cos, sin).to(proj.dtype)
        st["k"] = torch.cat([st["k"], k], dim=1)
        st["v"] = torch.cat([st["v"], v], dim=1)
        scores = torch.einsum("bqhd,bkhd->bhqk", q.float(), st["k"].float()) / math.sqrt(inner.hd)
        o = torch.einsum("bhqk,bkhd->bqhd", scores.softmax(-1), st["v"].float())
        return o.reshape(B, inner.heads * inner.hd)

    @torch.no_grad()
    def step(self, token: torch.Tensor) -> torch.Tensor:
        """token [B] -> logits of the next position [B, V]; advances every layer's state by one token."""
        model, cfg = self.model, self.cfg
        if self._fused is not None and self._fused.pos != self.pos:
            self._hand_back()                    # the caller moved to another position
        if self._resume:
            self._resume, self._fused = False, _FusedStep.build(self, token.shape[0])
        if self._fused is not None:
            was_training = model.training
            switch = any(m.training for m in model.embedding.modules())       # the only module that runs here
            if switch:
                model.eval()
            try:
                logits = self._fused(token)
            finally:
                if switch:
                    model.train(was_training)
            self.pos += 1
            return logits
        dtype = cfg.params_dtype
        pos = torch.tensor([self.pos], device=token.device)
        was_training = model.training
        model.eval()
        try:
            x = model.embedding(token[:, None], pos)[:, 0]                                   # [B, D]
        finally:
            model.train(was_training)
        for blk, st in zip(self.blocks, self._states):
            mixer = blk.mixer
            u = _rms(x.float(), blk.input_layernorm).to(dtype)
            proj = F.linear(u, mixer.dense_projection.weight)
            if isinstance(mixer.mixer, SelfAttention):
                z = self._attention_step(blk, st, proj)
            else:
                z = self._hyena_step(blk, st, proj)
            a = F.linear(z.to(dtype), mixer.dense.weight, mixer.dense.bias).float() + x.float()
            a = a.to(dtype)
            h = _rms(a.float(), blk.pre_mlp_layernorm).to(dtype) if blk.pre_mlp_norm else a
            mlp = blk.mlp
            ab = F.linear(h, mlp.w12)
            g, b = ab.float().chunk(2, dim=-1)
            hid = (_act(mlp.act)(g) * b).to(dtype)
            y = F.linear(hid, mlp.w3.weight, mlp.w3.bias).float() + a.float()
            x = y.to(dtype)
        self.pos += 1
        return model.logits(x[:, None])[:, 0].float()


@torch.no_grad()
def stream_tokens_cached(model, context_tokens: List[List[int]], eos_token_id: Optional[int] = None, maximum_tokens: int = 64,
                         temperature: float = 0.0, top_k: int = 0, top_p: float = 0.0, generator=None):
    """Cached counterpart of `generation.stream_tokens` for prompts of equal length: one prefill, then one `step` per
    generated token.  Yields (tokens [B, T], logits of the step, finished mask)."""
    from .generation import sample_tokens
    lens = {len(c) for c in context_tokens}
    if len(lens) != 1:
        raise ValueError("cached generation takes prompts of equal length (pad or group them by length)")
    device = next(model.parameters()).device
    toks = torch.tensor(context_tokens, dtype=torch.long, device=device)
    dec = CachedDecoder(model)
    logits = dec.prefill(toks)
    done = torch.zeros(toks.shape[0], dtype=torch.bool, device=device)
    for _ in range(maximum_tokens):
        nxt = sample_tokens(logits, temperature, top_k, top_p, generator)
        if eos_token_id is not None:
            nxt = torch.where(done, torch.full_like(nxt, eos_token_id), nxt)
            done |= nxt == eos_token_id
        toks = torch.cat([toks, nxt[:, None]], dim=1)
        yield toks, logits, done
        if bool(done.all()):
            break
        logits = dec.step(nxt)
