"""The native decode step (csrc/decode.cu) against the operator-by-operator step of the same decoder: the layers' forms,
parameters that change between steps, state that is copied and put back."""
import copy
import os

import pytest
import torch

from savanna_b200.config import GlobalConfig
from savanna_b200.inference import cached
from savanna_b200.inference.cached import CachedDecoder
from savanna_b200.models import build_model
from savanna_b200.models.hyena import ShortHyenaOperator
from savanna_b200.models.mixer import SelfAttention
from savanna_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"
TINY = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "configs", "baseline", "tiny_sh2_gpu.yml")


def _model(**over):
    cfg = GlobalConfig.from_ymls([TINY], {"global_num_gpus": 1, **over})
    cfg.build_tokenizer()
    torch.manual_seed(0)
    model = build_model(cfg, device=DEV)
    with torch.no_grad():                                  # make the state-dependent terms matter
        for n, p in model.named_parameters():
            if n.endswith("filter.h"):
                p.mul_(3e4)
    return model.eval()


def _slow(model, toks, monkeypatch):
    """A decoder prefilled with `toks` that steps operator by operator."""
    dec = CachedDecoder(model)
    with monkeypatch.context() as m:
        m.setattr(cached._FusedStep, "build", staticmethod(lambda *_: None))
        dec.prefill(toks)
    return dec


def _toks(model, B, n):
    return torch.randint(0, 256, (B, n), device=DEV, generator=torch.Generator(DEV).manual_seed(n))


def _agree(fast, slow, toks):
    """Both round activations to bf16, at different places: each step's logits within 2.2 % (2-norm), as derived in
    test_gpu_tile_edges.py."""
    for t in toks.unbind(1):
        a, b = fast.step(t), slow.step(t)
        assert (a - b).norm() <= 2.2e-2 * b.norm(), ((a - b).norm() / b.norm()).item()


_FORMS = {
    "gelu": {"mlp_activation": "gelu"}, "relu": {"mlp_activation": "relu"}, "identity": {"mlp_activation": "identity"},
    "classic_norm": {"rmsnorm_form": "classic", "rms_norm_epsilon": 1e-2}, "no_second_norm": {"pre_mlp_norm": False},
    "no_pregate": {"hyena_se_pregate": False}, "no_postgate": {"hyena_se_postgate": False},
    "partial_rotary": {"rotary_pct": 0.25}, "linear_rotary": {"pos_emb": "rotary_linear_scaled", "rotary_emb_scaling_factor": 4.0},
    "no_rotary": {"pos_emb": "none"}, "untied_head": {"no_weight_tying": True},
    "scaled_head": {"use_mup": True, "mup_width_scale": 2, "mup_output_temp": 0.5, "mup_embedding_mult": 3.0},
    "order_5": {"hyena_filter_order": 5}, "order_40": {"hyena_filter_order": 40}, "grouped_long_filter": {"num_groups_hyena": 64},
    "short_taps": {"hyena_se_len": 4, "short-conv-L": 2, "hyena_mr_len": 17}, "one_tap": {"hyena_se_len": 1, "hyena_mr_len": 1},
}


@pytest.mark.parametrize("B,T", [(1, 7), (3, 150)])
@pytest.mark.parametrize("form", _FORMS)
def test_forms(form, B, T, monkeypatch):
    """Every branch of the kernels: gates, norms, position embeddings, filter lengths and orders, heads that the step leaves to the
    model."""
    model = _model(**_FORMS[form])
    toks = _toks(model, B, T + 12)
    fast, slow = CachedDecoder(model), _slow(model, toks[:, :T], monkeypatch)
    fast.prefill(toks[:, :T])
    assert fast._fused is not None and (fast._fused.head is None) == (form in ("untied_head", "scaled_head"))
    _agree(fast, slow, toks[:, T:])


@pytest.mark.parametrize("form", ["", "partial_rotary", "linear_rotary", "no_rotary"])
@pytest.mark.parametrize("B,T", [(1, 1), (2, 517)])
def test_prefilled_keys(form, B, T):
    """The keys that a prefill leaves are those of the fp32 statement, rounded once, bit for bit."""
    model = _model(**_FORMS.get(form, {}))
    dec, seen = CachedDecoder(model), {}
    mods = {i: b.mixer.mixer for i, b in enumerate(dec.blocks) if isinstance(b.mixer.mixer, SelfAttention)}
    hooks = [m.register_forward_pre_hook(lambda m, a, i=i: seen.update({i: (a[0].clone(), a[1].clone())})) for i, m in mods.items()]
    dec.prefill(_toks(model, B, T))
    for h in hooks:
        h.remove()
    assert mods and seen.keys() == mods.keys()
    for i, m in mods.items():
        q = seen[i][0].view(B, T, m.heads, 3 * m.hd)
        k = q[..., m.hd:2 * m.hd].float()
        if m._rotary:
            k = ref.apply_rope(k, *m._rotary[0](seen[i][1]))
        assert torch.equal(dec.states[i]["k"][:, :T], k.to(q.dtype)) and torch.equal(dec.states[i]["v"][:, :T], q[..., 2 * m.hd:])


@pytest.mark.parametrize("B,ffn,native", [(8, 12800, True), (8, 12816, False), (4, 12816, True), (9, 512, False)])
def test_limits(B, ffn, native, monkeypatch):
    """The widest gate whose inputs fit in shared memory, one step wider, and more sequences than a launch takes."""
    model = _model(ffn_hidden_size=ffn)
    toks = _toks(model, B, 12)
    fast, slow = CachedDecoder(model), _slow(model, toks[:, :9], monkeypatch)
    fast.prefill(toks[:, :9])
    assert (fast._fused is not None) == native
    _agree(fast, slow, toks[:, 9:])


@pytest.mark.parametrize("x2", [float("inf"), float("nan")])
def test_unused_stream_stays_out(x2, monkeypatch):
    """Without its pre-gate the short filter does not read the second stream: what is not finite there reaches nothing."""
    model = _model(hyena_se_pregate=False)
    toks = _toks(model, 2, 30)
    conv = next(b.mixer.hyena_proj_conv for b in model.blocks() if isinstance(b.mixer.mixer, ShortHyenaOperator))
    assert conv.group_dim == 1
    with torch.no_grad():
        conv.short_conv_weight[1::3] = x2
    fast, slow = CachedDecoder(model), _slow(model, toks[:, :20], monkeypatch)
    assert fast.prefill(toks[:, :20]).isfinite().all() and fast._fused is not None
    _agree(fast, slow, toks[:, 20:])
    assert fast._fused is not None


def _is_filter(n):
    return any(k in n for k in ("short_conv", ".filter.", "conv_bias"))


@pytest.mark.parametrize("moved", [False, True], ids=["in_place", "moved"])
@pytest.mark.parametrize("which", ["filters", "projections"])
@pytest.mark.parametrize("over", [{}, {"hyena_medium_filter_cls": "implicit_modal"}], ids=["explicit", "modal_mr"])
def test_parameters_changed_between_steps(which, over, moved, monkeypatch):
    """A step reads every parameter as it is then, filters as well as projections."""
    model = _model(**over)
    toks = _toks(model, 2, 30)
    fast, slow = CachedDecoder(model), _slow(model, toks[:, :20], monkeypatch)
    fast.prefill(toks[:, :20])
    assert fast._fused is not None
    _agree(fast, slow, toks[:, 20:23])
    before = slow.step(toks[:, 23])
    fast.step(toks[:, 23])
    g = torch.Generator(DEV).manual_seed(3)
    with torch.no_grad():
        for n, p in model.named_parameters():
            if _is_filter(n) == (which == "filters") and "norm" not in n and "word_emb" not in n:
                s = float(p.float().std()) or 0.1
                new = p.data + (torch.randn(p.shape, device=DEV, generator=g) * s).to(p.dtype)
                if moved:
                    p.data = new
                else:
                    p.data.copy_(new)
    _agree(fast, slow, toks[:, 24:])
    assert (slow.step(toks[:, 0]) - before).norm() > 0.1 * before.norm()          # the change reached the logits


@pytest.mark.parametrize("bf16", ["", "short_conv", "short_conv filter conv_bias", ".R .h", "conv_bias gamma"],
                         ids=lambda s: s.replace(" ", "+") or "none")
def test_types_of_stored_filters(bf16, monkeypatch):
    """Filter parameters named here are bf16, the others fp32: each mixture has its kernel."""
    model = _model()
    for n, p in model.named_parameters():
        if _is_filter(n):
            p.data = p.data.bfloat16() if any(k in n for k in bf16.split()) else p.data.float()
    toks = _toks(model, 1, 30)
    fast, slow = CachedDecoder(model), _slow(model, toks[:, :25], monkeypatch)
    fast.prefill(toks[:, :25])
    assert fast._fused is not None
    _agree(fast, slow, toks[:, 25:])


@pytest.mark.parametrize("T", [1, 3, 20, 129, 260])
def test_branched_continuations(T, monkeypatch):
    """Two continuations of one prompt, branched by copying the state's dictionaries, the decoder, or a batch of rows."""
    model = _model()
    toks = _toks(model, 2, T + 20)
    fast, slow = CachedDecoder(model), _slow(model, toks[:, :T], monkeypatch)
    fast.prefill(toks[:, :T])
    _agree(fast, slow, toks[:, T:T + 3])
    saved = {d: ([dict(s) for s in d.states], d.pos) for d in (fast, slow)}
    for a, b in zip(saved[fast][0], saved[slow][0]):
        assert a.keys() == b.keys() and all(a[k].shape == b[k].shape for k in a)
    twin, twin_slow = copy.deepcopy(fast), copy.deepcopy(slow)
    first = fast.step(toks[:, T + 3])
    assert fast._fused is not None                                   # the native step took the state up again
    slow.step(toks[:, T + 3])
    _agree(fast, slow, toks[:, T + 4:T + 8])
    for d in (fast, slow):                                           # back to the branch
        d.states, d.pos = [dict(s) for s in saved[d][0]], saved[d][1]
    assert torch.equal(fast.step(toks[:, T + 3]), first)             # bit for bit: nothing of the first branch is left
    slow.step(toks[:, T + 3])
    _agree(fast, slow, toks[:, T + 8:T + 12])
    assert twin._fused is None and torch.equal(twin.step(toks[:, T + 3]), first) and twin._fused is not None
    twin_slow.step(toks[:, T + 3])
    live = copy.deepcopy(twin)                                       # of a decoder in the middle of native steps
    assert twin._fused is not None
    _agree(twin, twin_slow, toks[:, T + 12:T + 16])
    live.step(toks[:, T + 12])
    for d in (fast, slow):                                           # another batch: rows picked by the caller
        d.states, d.pos = [{k: v[[1, 0, 1]] for k, v in s.items()} for s in saved[d][0]], saved[d][1]
    _agree(fast, slow, toks[[1, 0, 1], T + 3:T + 7])
    assert fast._fused is not None and fast._fused.batch == 3


def _get(model, name):
    mod, _, leaf = name.rpartition(".")
    return model.get_submodule(mod), leaf


@pytest.mark.parametrize("name", ["sequential.2.mixer.dense_projection.weight", "sequential.3.mixer.mixer.filter.h",
                                  "sequential.4.mixer.mixer.filter.R", "sequential.4.mlp.w12", "sequential.5.input_layernorm.weight",
                                  "sequential.7.norm.weight", "sequential.0.word_embeddings.weight"])
def test_replaced_parameter_is_followed(name, monkeypatch):
    model = _model()
    toks = _toks(model, 2, 30)
    fast, slow = CachedDecoder(model), _slow(model, toks[:, :20], monkeypatch)
    fast.prefill(toks[:, :20])
    _agree(fast, slow, toks[:, 20:22])
    mod, leaf = _get(model, name)
    old = getattr(mod, leaf)
    setattr(mod, leaf, torch.nn.Parameter(old.detach() * (10 if _is_filter(name) else 1.5) + 0.25 * old.detach().roll(1, 0)))
    _agree(fast, slow, toks[:, 22:26])
    assert fast._fused is not None


def test_replaced_module_and_settings_are_followed(monkeypatch):
    model = _model()
    toks = _toks(model, 2, 40)
    fast, slow = CachedDecoder(model), _slow(model, toks[:, :20], monkeypatch)
    fast.prefill(toks[:, :20])
    other = _model(seed=5)
    blocks = model.blocks()
    blocks[1].mlp = other.blocks()[2].mlp
    _agree(fast, slow, toks[:, 20:24])
    blocks[2].mlp.act = "gelu"
    blocks[0].input_layernorm.eps = 1e-2
    _agree(fast, slow, toks[:, 24:28])
    blocks[0].mixer.mixer.pregate = False                  # the FIR's past is then of another signal, in both steps alike
    _agree(fast, slow, toks[:, 28:32])
    assert fast._fused is not None


def test_unusable_weights_are_refused(monkeypatch):
    """A weight that the kernels cannot read sends the step down the operator-by-operator path, which computes with it or raises
    as it always has; the state survives either."""
    model = _model()
    toks = _toks(model, 2, 40)
    fast, slow = CachedDecoder(model), _slow(model, toks[:, :20], monkeypatch)
    fast.prefill(toks[:, :20])
    _agree(fast, slow, toks[:, 20:22])
    p = model.blocks()[1].mixer.dense_projection.weight
    keep = p.data
    shifted = torch.empty(p.numel() + 1, device=DEV, dtype=p.dtype)[1:].view(p.shape)          # two bytes off a 16-byte boundary
    shifted.copy_(keep)
    p.data = shifted
    _agree(fast, slow, toks[:, 22:24])
    assert fast._fused is None
    p.data = keep.t().contiguous().t()                     # not contiguous
    _agree(fast, slow, toks[:, 24:26])
    p.data = keep
    fast.states = fast.states                              # takes the native step up again
    _agree(fast, slow, toks[:, 26:28])
    assert fast._fused is not None
    model.float()
    for dec in (fast, slow):
        with pytest.raises(RuntimeError):
            dec.step(toks[:, 28])
    model.to(torch.bfloat16)                               # every parameter, the filters too
    fast.states = fast.states
    _agree(fast, slow, toks[:, 28:30])
    assert fast._fused is not None
    model.cpu()
    for dec in (fast, slow):
        with pytest.raises(RuntimeError):
            dec.step(toks[:, 30].cpu())
    assert fast._fused is None


def test_weight_behind_a_property(monkeypatch):
    """A projection whose weight is computed when it is read, as adapters do it: read again in every step."""
    class Adapted(torch.nn.Module):
        def __init__(self, base):
            super().__init__()
            self.base, self.factor = base, 1.0
            self.bias = base.bias

        @property
        def weight(self):
            return self.base.weight * self.factor

        def forward(self, x, *a):
            return self.base(x * self.factor, *a)

        def forward_normed(self, x, norm):
            y, b, r = self.base.forward_normed(x, norm)
            return y * self.factor, b, r
    model = _model()
    mixer = model.blocks()[1].mixer
    mixer.dense_projection = Adapted(mixer.dense_projection)
    toks = _toks(model, 2, 30)
    fast, slow = CachedDecoder(model), _slow(model, toks[:, :20], monkeypatch)
    fast.prefill(toks[:, :20])
    assert fast._fused is not None
    _agree(fast, slow, toks[:, 20:23])
    mixer.dense_projection.factor = 3.0
    _agree(fast, slow, toks[:, 23:27])
    assert fast._fused is not None


def test_embedding_of_another_type(monkeypatch):
    """What the embedding returns is looked at too: fp32 activations go operator by operator."""
    model = _model()
    toks = _toks(model, 2, 30)
    fast, slow = CachedDecoder(model), _slow(model, toks[:, :20], monkeypatch)
    fast.prefill(toks[:, :20])
    h = model.embedding.register_forward_hook(lambda m, a, out: out.float())
    for i in (20, 21):
        a, b = fast.step(toks[:, i]), slow.step(toks[:, i])
        assert torch.equal(a, b) or (a - b).norm() <= 2.2e-2 * b.norm()
        assert fast._fused is None and not fast._resume
    h.remove()
    fast.states = fast.states
    _agree(fast, slow, toks[:, 22:26])
    assert fast._fused is not None
