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
other configuration raises NotImplementedError and the caller falls back to `stream_tokens` (recompute).  So does a sequence
longer than `rotary_emb_max_unscaled_seq_len` under `rotary_ntk_scaled`: from there on the rotary base of all positions changes
with every token, and with it every key and everything computed from them.
"""
from __future__ import annotations

import ctypes
import math
import operator
from typing import Dict, List, Optional

import torch
import torch.nn.functional as F

from ..models.filters import ExplicitSingleDecayFilter, ImplicitModalFilter
from ..models.hyena import HyenaOperator, ShortHyenaOperator
from ..models.mixer import SelfAttention
from ..models.mlp import ParallelGLU
from ..models.norms import RMSNorm
from .. import ops
from ..ops import cuda_ops
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


class _Watch:
    """Reads attributes and remembers where each was found, so that `same` can tell later, without reading the layers again,
    whether any of them has been replaced."""

    def __init__(self):
        self.seen = []                           # (dictionary or list, key, value)
        self.computed = False                    # something came out of a property: it can be another one at any time

    def __call__(self, obj, name):
        d = obj.__dict__
        for c in (d, d.get("_modules"), d.get("_parameters"), d.get("_buffers")):
            if c is not None and name in c:
                self.seen.append((c, name, c[name]))
                return c[name]
        self.computed = True
        return getattr(obj, name)

    def same(self) -> bool:
        if self.computed:
            return False
        try:
            for c, k, v in self.seen:
                if c[k] is not v:
                    return False
        except (KeyError, IndexError):
            return False
        return True


def _short_taps(conv, at):
    """(weight, the shape it must have) of a depthwise convolution: [groups, k] or [groups, 1, k], the same in memory."""
    w, g, k = at(conv, "short_conv_weight"), conv.num_groups, conv.kernel_size
    return w, ((g, 1, k) if w.dim() == 3 else (g, k))


def _layer_form(blk, D, at):
    """(what a layer computes, its weights) for csrc/decode.cu, or None where the kernels do not cover it; read through `at`, a
    `_Watch`.  The form is a dictionary of descriptor fields; a weight is (field, tensor, shape it must have, whether it is a
    filter parameter, read as it is stored)."""
    mixer, mlp, n1 = at(blk, "mixer"), at(blk, "mlp"), at(blk, "input_layernorm")
    n2 = at(blk, "pre_mlp_layernorm") if at(blk, "pre_mlp_norm") else None
    if not isinstance(mlp, ParallelGLU) or not isinstance(n1, RMSNorm) or not (n2 is None or isinstance(n2, RMSNorm)) \
            or at(mlp, "act") not in cuda_ops._ACT:
        return None
    op, H, Fi = at(mixer, "mixer"), at(mixer, "inner_size"), at(mlp, "ffn_local")
    dense, w3 = at(mixer, "dense"), at(mlp, "w3")
    form: Dict = {"H": H, "F": Fi, "act": cuda_ops._ACT[mlp.act], "norm2": int(n2 is not None)}
    ws = [("w_in", at(at(mixer, "dense_projection"), "weight"), (3 * H, D), False), ("w_out", at(dense, "weight"), (D, H), False),
          ("w12", at(mlp, "w12"), (2 * Fi, D), False), ("w3", at(w3, "weight"), (D, Fi), False),
          ("b_out", at(dense, "bias"), (D,), False), ("b3", at(w3, "bias"), (D,), False)]
    for n, i in ((n1, "1"), (n2, "2")):
        if n is not None:
            te = at(n, "form") == "te"
            form["eps" + i], form["form" + i] = at(n, "eps"), int(not te)
            ws.append((f"norm{i}_w", at(n, "weight" if te else "scale"), (D,), False))
    if isinstance(op, SelfAttention):
        if at(op, "hd") != 128 or at(op, "heads") * 128 != H:
            return None
        form.update(kind=3, heads=op.heads, rd=0, pos_scale=1.0, base=0.0)
        if at(op, "_rotary"):
            r = op._rotary[0]
            at.seen.append((op._rotary, 0, r))
            form.update(rd=at(r, "dim"), pos_scale=at(r, "scaling_factor"), base=at(r, "base"))
        return form, ws
    conv, G = at(mixer, "hyena_proj_conv"), at(op, "num_groups")
    if at(conv, "num_groups") * at(conv, "group_dim") != 3 * H or G * at(op, "group_dim") != H:
        return None
    form.update(kf=at(conv, "kernel_size"), conv_g=conv.num_groups, G=G, pregate=1, postgate=1)
    ws.append(("conv_w", *_short_taps(conv, at), True))
    if isinstance(op, ShortHyenaOperator):
        K, c = at(op, "kernel_size"), at(op, "short_conv")
        form.update(kind=0, K=K, tap_ld=K, pregate=int(bool(at(op, "pregate"))), postgate=int(bool(at(op, "postgate"))))
        if at(c, "num_groups") != G or at(c, "kernel_size") != K:
            return None
        ws.append(("taps", *_short_taps(c, at), True))
        return form, ws
    f = at(op, "filter")
    ws.append(("bias", at(op, "conv_bias"), (H,), True))
    if at(op, "is_mr"):
        K = at(op, "hyena_mr_len")
        if type(f) is ExplicitSingleDecayFilter:
            h = at(f, "h")
            if h.shape[1] < K:
                return None
            form["tap_ld"] = h.shape[1]
            ws += [("taps", h, (G, h.shape[1]), True), ("decay", at(f, "decay"), (G, h.shape[1]), True)]
        else:                                    # no form of its own in the kernel: the module evaluates it in every step
            form["tap_ld"] = K
            ws.append(("taps", f, (G, K), True))
        form.update(kind=1, K=K, newest_first=1)
        return form, ws
    O = at(f, "gamma").shape[1]
    form.update(kind=2, O=O)
    return form, ws + [(n, at(f, n), (G, O), True) for n in ("gamma", "p", "R")]


def _usable(t, shape, filt, device) -> bool:
    """What the kernels assume of a weight: bf16 rows read 16 bytes at a time, or filter parameters read one by one."""
    if t.shape != shape or t.device != device or not t.is_contiguous():
        return False
    return t.dtype in (torch.bfloat16, torch.float32) if filt else t.dtype == torch.bfloat16 and t.data_ptr() % 16 == 0


_PTR, _NUMEL, _CONTIGUOUS = torch.Tensor.data_ptr, torch.Tensor.numel, torch.Tensor.is_contiguous
_DTYPE = operator.attrgetter("dtype")


class _FusedStep:
    """The decode step of csrc/decode.cu: the layers' weights by address, their state in the layout of its kernels.  Built at
    the end of a prefill and after the state was handed out (`CachedDecoder.states`); `build` returns None when something is not
    covered (CPU tensors, other dtypes than bf16, other norms than RMSNorm, head sizes other than 128, more than 8 sequences, an
    inner size above `sb_decode_max_width`: 102400 for one sequence, 12800 for eight; unaligned or non-contiguous weights), and the
    decoder then steps operator by operator.

    A step looks at the modules as they are then: `follow` refuses when a weight has changed its type, shape, device or alignment
    into something that the kernels do not read, or a layer computes something else than it did.  It reads the layers again only
    when an attribute or tensor that it read before is another one now, or lies elsewhere (four layers: 13 us of host time for
    the comparison where the reading takes 130, of the 135 in which a step is issued)."""

    @staticmethod
    def build(dec: "CachedDecoder", batch: int):
        if not ops._k(dec.model.embedding.word_embeddings.weight):
            return None
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
        self = _FusedStep(dec, lib, batch)
        return self if self.follow() and self._adopt(dec) else None

    def __init__(self, dec: "CachedDecoder", lib, batch: int):
        self.model, self.cfg, self.blocks = dec.model, dec.cfg, dec.blocks       # not `dec`, which holds this object
        self.lib, self.batch, self.D, self.wmax = lib, batch, dec.cfg.hidden_size, lib.sb_decode_max_width(batch)
        self.device = dec.model.embedding.word_embeddings.weight.device
        self.layers = (_DecLayer * len(dec.blocks))()
        self.forms: List[Dict] = []             # what each layer computes
        self.watch = None                       # what `follow` read: attributes ...
        self.tensors: List[torch.Tensor] = []   # ... and tensors, with their addresses, types and sizes in `seen`
        self.seen, self.storage = None, []
        self.modules = []                       # (descriptor, filter module): evaluated in every step
        self.temps: List[torch.Tensor] = []     # the evaluated filters
        self.freqs: List[torch.Tensor] = []     # rotary frequencies
        self.attn = []                          # (layer index, key cache, value cache)
        self.rings = []                         # (layer index, name of the state, buffer) of the Hyena layers
        self.pos = dec.pos

    def follow(self) -> bool:
        """Points the descriptors at the weights as they are now; False when the kernels must not read them."""
        if self.watch is None or not self._unchanged():
            if not self._read():
                self.watch = None
                return False
        self.temps = [f(L.K).float().contiguous() for L, f in self.modules]
        for (L, _), t in zip(self.modules, self.temps):
            if t.shape != (L.G, L.K) or t.device != self.device:
                return False
            L.taps = t.data_ptr()
        return True

    def _signature(self):
        ts = self.tensors
        return list(map(_PTR, ts)), list(map(_DTYPE, ts)), list(map(_NUMEL, ts)), list(map(_CONTIGUOUS, ts))

    def _unchanged(self) -> bool:
        return self.watch.same() and self._signature() == self.seen

    def _read(self) -> bool:
        at = _Watch()
        model, cfg = self.model, self.cfg
        seq = at(model, "sequential")
        emb = at(at(seq, "0"), "word_embeddings")
        head = at(emb, "weight")
        at.seen.append((ops.__dict__, "_BACKEND", ops._BACKEND))
        at(cfg, "precision")
        if cfg.params_dtype != torch.bfloat16 or not ops._k(head):
            return False
        self.tensors, self.modules = [], []
        for i, (L, blk) in enumerate(zip(self.layers, self.blocks)):
            lw = _layer_form(blk, self.D, at)
            if lw is None:
                return False
            if i == len(self.forms):             # the first time
                if any(n % 8 or n > self.wmax for n in (self.D, lw[0]["H"], lw[0]["F"])):
                    return False
                self.forms.append(lw[0])
                for name, v in lw[0].items():
                    if name != "base":
                        setattr(L, name, v)
            elif lw[0] != self.forms[i]:
                return False
            f32 = 0
            for name, t, shape, filt in lw[1]:
                if isinstance(t, torch.nn.Module):
                    self.modules.append((L, t))
                    f32 |= _F32[name]
                elif t is None:                  # no bias
                    setattr(L, name, None)
                elif _usable(t, shape, filt, self.device):
                    self.tensors.append(t)
                    if filt and t.dtype == torch.float32:
                        f32 |= _F32[name]
                    setattr(L, name, t.data_ptr())
                else:
                    return False
            L.f32 = f32
        # the logits, where the kernels can form them: (final norm, head weight)
        self.head = None
        tail = at(seq, str(model.num_layers + 3))
        fn = at(tail, "norm") if hasattr(tail, "norm") else None
        if not at(cfg, "no_weight_tying") and at(model, "mup_output_mult") == 1.0 and isinstance(fn, RMSNorm):
            gain = at(fn, "weight" if at(fn, "form") == "te" else "scale")
            self.tensors += [gain, head]
            if _usable(gain, (self.D,), False, self.device) and _usable(head, (head.shape[0], self.D), False, self.device):
                self.head = (gain, at(fn, "eps"), int(fn.form != "te"), head)
        self.watch, self.seen = at, self._signature()
        self.storage = [t.detach() for t in self.tensors]      # held, so that an address seen again is the same memory
        return True

    def _adopt(self, dec: "CachedDecoder") -> bool:
        """Takes over the decoder's state, whoever filled its dictionaries, if its tensors are what the kernels expect."""
        bf = torch.bfloat16
        if len(dec._states) != len(self.forms):
            return False

        def held(st, name, *shape, dtype=None):
            t = st.get(name)
            return (t is not None and t.device == self.device and tuple(t.shape) == (self.batch,) + shape
                    and (dtype is None or t.dtype == dtype))

        for f, st in zip(self.forms, dec._states):
            if f["kind"] == 3:
                ok = all(held(st, n, self.pos, f["heads"], 128, dtype=bf) for n in ("k", "v"))
            else:
                ok = (held(st, "proj_tail", f["kf"] - 1, 3 * f["H"], dtype=bf)
                      and (held(st, "s", f["H"], f["O"]) if f["kind"] == 2 else held(st, "u_tail", f["K"] - 1, f["H"])))
            if not ok:
                return False

        def ring(i, name, t):
            self.rings.append((i, name, t))
            return t.data_ptr()

        for i, (L, f, st) in enumerate(zip(self.layers, self.forms, dec._states)):
            if f["kind"] == 3:
                if f["rd"]:
                    inv = 1.0 / (f["base"] ** (torch.arange(0, f["rd"], 2, device=self.device, dtype=torch.float32) / f["rd"]))
                    self.freqs.append(inv)
                    L.inv_freq = inv.data_ptr()
                self.attn.append([i, st["k"], st["v"]])
                continue
            L.proj_ring = ring(i, "proj_tail", _ring(st["proj_tail"], self.pos))
            if f["kind"] == 2:
                L.state = ring(i, "s", st["s"].float().contiguous().clone())
            else:
                L.u_ring = ring(i, "u_tail", _ring(st["u_tail"].float(), self.pos))
        self._reserve(self.pos + 1)
        wide = max([self.D] + [max(f["H"], f["F"]) for f in self.forms])
        # the in-projection, the operator's output, the stream after the mixer, the gate's two halves
        self.scratch = [torch.empty(self.batch, n, dtype=bf, device=self.device) for n in (3 * wide, wide, self.D, 2 * wide)]
        self.scratch_ptrs = [t.data_ptr() for t in self.scratch]
        self.descr = ctypes.addressof(self.layers)
        dec._states = [dict() for _ in dec.blocks]          # this object holds the state from here on
        return True

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

    def __call__(self, token: torch.Tensor) -> Optional[torch.Tensor]:
        """Logits of the next position, or None (and nothing changed) when the embedding left what the kernels read."""
        if token.shape[0] != self.batch:
            raise ValueError(f"decode step for {token.shape[0]} sequences, prefilled with {self.batch}")
        model = self.model
        x = model.embedding(token[:, None], None)
        if x.dtype != torch.bfloat16 or x.shape != (self.batch, 1, self.D) or x.device != self.device:
            return None
        x = x.contiguous()
        ptr = x.data_ptr()
        if ptr % 16:
            return None
        self._reserve(self.pos + 1)
        norm, eps, form, head, V, out, logits = None, 0.0, 0, None, 0, None, None
        if self.head is not None:
            gain, eps, form, w = self.head
            norm, head, V = gain.data_ptr(), w.data_ptr(), w.shape[0]
            out = torch.empty(self.batch, V, dtype=torch.float32, device=self.device)
            logits = out.data_ptr()
        cuda_ops._check(self.lib.sb_decode_step(self.descr, len(self.layers), ptr, *self.scratch_ptrs, self.batch, self.D, self.pos,
                                                norm, eps, form, head, V, logits, cuda_ops._stream()), "decode_step")
        cuda_ops._count(5 * len(self.layers) + (1 if V else 0))
        self.pos += 1
        return out if V else model.logits(x)[:, 0].float()


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
        # the longest sequence whose keys stay what they are as it grows
        self.limit = min((r.max_unscaled_len for b in self.blocks if isinstance(b.mixer.mixer, SelfAttention)
                          for r in b.mixer.mixer._rotary if r.kind == "rotary_ntk_scaled"), default=None)
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

    def check_length(self, n: int) -> None:
        if self.limit is not None and n > self.limit:
            raise NotImplementedError(f"cached generation of {n} tokens: rotary_ntk_scaled changes its base beyond {self.limit}")

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
        model = self.model
        B, T = tokens.shape
        self.check_length(T)
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
                        # three fp32 operations and one rounding, as the operator-by-operator step rotates: the rotary kernel contracts
                        # product and sum, and keys near a rounding boundary would land on its other side
                        k = ref.apply_rope(k.float(), cos, sin).to(qkv.dtype)
                    else:
                        k = k.clone()
                    st["k"], st["v"] = k, v.clone()
                hooks.append(inner.register_forward_pre_hook(grab_kv))
            else:
                kf = mixer.short_conv_L

                def grab_proj(mod, args, st=st, kf=kf):
                    st["proj_tail"] = tail(args[0], kf - 1)
                hooks.append(mixer.hyena_proj_conv.register_forward_pre_hook(grab_proj))

                if isinstance(inner, HyenaOperator) and not inner.is_mr:
                    # the layer's own scan leaves its state behind: no second pass over the prompt
                    inner.state_sink = lambda s, st=st: st.__setitem__("s", s.float())
                    continue

                def grab_feat(mod, args, st=st):
                    short = isinstance(mod, ShortHyenaOperator)
                    n = (mod.kernel_size if short else min(mod.hyena_mr_len, 1 << 30)) - 1
                    feat = args[0][:, -n:] if n > 0 else args[0][:, :0]          # only these rows are kept
                    v = feat[..., 2::3]
                    st["u_tail"] = tail(v if short and not mod.pregate else feat[..., 1::3] * v, n)
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
            for blk in self.blocks:
                if isinstance(blk.mixer.mixer, HyenaOperator):
                    blk.mixer.mixer.state_sink = None
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
        self.check_length(self.pos + 1)
        if self._fused is not None and (self._fused.pos != self.pos or not self._fused.follow()):
            self._hand_back()                    # the caller moved to another position, or changed the model
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
            if logits is not None:
                self.pos += 1
                return logits
            self._hand_back()
            self._resume = False                 # not at every token again
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


def stream_tokens_cached(model, context_tokens: List[List[int]], eos_token_id: Optional[int] = None, maximum_tokens: int = 64,
                         temperature: float = 0.0, top_k: int = 0, top_p: float = 0.0, generator=None):
    """Cached counterpart of `generation.stream_tokens` for prompts of equal length: one prefill, then one `step` per
    generated token.  Yields (tokens [B, T], logits of the step, finished mask).  Raises before the first token when the model, or
    a sequence of the full length, has no cached form."""
    lens = {len(c) for c in context_tokens}
    if len(lens) != 1:
        raise ValueError("cached generation takes prompts of equal length (pad or group them by length)")
    dec = CachedDecoder(model)
    dec.check_length(lens.pop() + maximum_tokens)
    return _stream(dec, context_tokens, eos_token_id, maximum_tokens, temperature, top_k, top_p, generator)


@torch.no_grad()
def _stream(dec, context_tokens, eos_token_id, maximum_tokens, temperature, top_k, top_p, generator):
    from .generation import sample_tokens
    device = next(dec.model.parameters()).device
    toks = torch.tensor(context_tokens, dtype=torch.long, device=device)
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
