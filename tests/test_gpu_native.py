"""The C++ autograd functions (csrc/autograd_native.cpp): the nodes that join several operators against the operators one by one, which
inputs get gradients, tracing, saved-tensor hooks, and what autograd refuses."""
import itertools
import os
import subprocess
import sys

import pytest
import torch

from savanna_b200 import ops

pytestmark = pytest.mark.gpu
DEV, BF = "cuda", torch.bfloat16


def _rand(*shape, std=1.0):
    return (torch.randn(*shape, device=DEV) * std).to(BF)


def _grads(fn, tensors, needs, gout):
    leaves = [None if t is None else t.clone().requires_grad_(n) for t, n in zip(tensors, needs)]
    out = fn(*leaves)
    out.backward(gout)
    return [out.detach()] + [None if t is None else t.grad for t in leaves]


@pytest.mark.parametrize("T,D,F,bias", [(1, 64, 8, False), (37, 256, 704, True), (999, 1024, 2816, False)])
@pytest.mark.parametrize("act", ["silu", "gelu"])
def test_mlp_is_its_parts(T, D, F, bias, act):
    torch.manual_seed(T)
    ts = [_rand(1, T, D), _rand(D), _rand(2 * F, D, std=D ** -0.5), _rand(D, F, std=F ** -0.5), _rand(D) if bias else None]
    g = _rand(1, T, D)

    def parts(x, wn, w12, w3, b3):
        y, res = ops.rmsnorm_residual(x, wn, 1e-6)
        return ops.linear(ops.glu_act_packed(ops.linear(y, w12), act), w3, b3, residual=res)

    def whole(x, wn, w12, w3, b3):
        return ops.mlp_gated(x, wn, 1e-6, "te", w12, w3, b3, act)

    for needs in ([True] * 5, [False, False, True, False, False], [False, True, False, False, False], [False, False, False, True, bias]):
        for a, b in zip(_grads(whole, ts, needs, g), _grads(parts, ts, needs, g)):
            assert (a is None) == (b is None)
            # the same kernels on the same values; only the bias gradient is summed with atomics: fp32 sums, rounded once to bf16
            assert a is None or torch.equal(a, b) or (a.float() - b.float()).norm() <= 2 ** -9 * b.float().norm()


@pytest.mark.parametrize("bias", [False, True])
def test_norm_and_projection_are_their_parts(bias):
    torch.manual_seed(3)
    ts = [_rand(2, 77, 512), _rand(512), _rand(1536, 512, std=0.05), _rand(1536) if bias else None]
    for needs in itertools.product([False, True], repeat=3):
        if not any(needs):
            continue
        got = []
        for one in (True, False):
            leaves = [None if t is None else t.clone().requires_grad_(n) for t, n in zip(ts, needs + (needs[2] and bias,))]
            x, wn, w, b = leaves
            if one:
                y, res = ops.norm_linear(x, wn, 1e-6, "te", w, b)
            else:
                u, res = ops.rmsnorm_residual(x, wn, 1e-6)
                y = ops.linear(u, w, b)
            (y.float().square().mean() + (res * 0.5).float().square().sum()).backward()
            got.append([y.detach(), res.detach()] + [None if t is None else t.grad for t in leaves])
        for a, b in zip(*got):
            assert (a is None) == (b is None)
            assert a is None or torch.equal(a, b) or (a.float() - b.float()).norm() <= 2 ** -9 * b.float().norm()


def _joined(kind):
    T, D, F = 4096, 512, 4096
    x, wn = _rand(1, T, D), _rand(D)
    if kind == "mlp":
        ws = [_rand(2 * F, D, std=D ** -0.5), _rand(D, F, std=F ** -0.5)]

        def whole(x, wn, w12, w3):
            return ops.mlp_gated(x, wn, 1e-6, "te", w12, w3, None, "silu")

        def parts(x, wn, w12, w3):
            y, res = ops.rmsnorm_residual(x, wn, 1e-6)
            return ops.linear(ops.glu_act_packed(ops.linear(y, w12), "silu"), w3, None, residual=res)
    else:
        ws = [_rand(3 * D, D, std=D ** -0.5)]

        def whole(x, wn, w):
            y, res = ops.norm_linear(x, wn, 1e-6, "te", w, None)
            return torch.cat([y, res], -1)

        def parts(x, wn, w):
            y, res = ops.rmsnorm_residual(x, wn, 1e-6)
            return torch.cat([ops.linear(y, w), res], -1)
    return [x, wn] + ws, whole, parts


def _leaves(ts, frozen=()):
    return [t.clone().requires_grad_(i not in frozen) for i, t in enumerate(ts)]


@pytest.mark.parametrize("kind", ["mlp", "norm_linear"])
@pytest.mark.parametrize("frozen", [(), (2,), (3,), (0, 1)])
def test_joined_nodes_need_no_more_memory_than_their_parts(kind, frozen):
    ts, whole, parts = _joined(kind)
    peak = []
    for fn in (whole, parts, whole, parts):
        leaves = _leaves(ts, frozen)
        out = fn(*leaves)
        g = torch.randn_like(out)
        del fn
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        out.backward(g)
        torch.cuda.synchronize()
        peak.append(torch.cuda.max_memory_allocated() - before)
        del out, g, leaves
    # the parts allocate the same tensors; a megabyte for the norm's partial sums, of which both have one set
    assert min(peak[0], peak[2]) <= max(peak[1], peak[3]) + 2 ** 20, [p / 2 ** 20 for p in peak]


@pytest.mark.parametrize("kind", ["mlp", "norm_linear"])
def test_joined_nodes_keep_their_graph_when_asked(kind):
    ts, whole, _ = _joined(kind)
    leaves = _leaves([t[:, :64] if i == 0 else t for i, t in enumerate(ts)])
    out = whole(*leaves)
    g = torch.randn_like(out)
    a, b, c = (torch.autograd.grad(out, leaves, g, retain_graph=r) for r in (True, True, False))
    assert all(torch.equal(x, y) and torch.equal(x, z) for x, y, z in zip(a, b, c))
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(out, leaves, g)


def test_only_the_residual_branch_is_used():
    x = _rand(2, 8, 128).requires_grad_()
    _, res = ops.norm_linear(x, _rand(128), 1e-6, "te", _rand(64, 128))
    res.float().sum().backward()
    assert torch.equal(x.grad, torch.ones_like(x))


def _block(x, wn, w):
    return ops.linear(ops.rmsnorm(x, wn, 1e-6), w).float().square().sum()


def test_traced_graph_runs_the_kernels_on_new_inputs():
    wn, w = _rand(256), _rand(512, 256, std=0.05)
    f = torch.jit.trace(lambda t: _block(t, wn, w), (_rand(4, 256).requires_grad_(),), check_trace=False)
    x = _rand(4, 256)
    a, b = x.clone().requires_grad_(), x.clone().requires_grad_()
    ya, yb = f(a), _block(b, wn, w)
    ya.backward()
    yb.backward()
    assert torch.equal(ya, yb) and torch.equal(a.grad, b.grad)


def test_saved_tensor_hooks_see_every_saved_tensor():
    n = [0, 0]

    def pack(t):
        n[0] += 1
        return t.cpu()

    def unpack(t):
        n[1] += 1
        return t.cuda()
    wn, w, x = _rand(256), _rand(512, 256, std=0.05), _rand(4, 256)
    a, b = x.clone().requires_grad_(), x.clone().requires_grad_()
    with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
        y, _ = ops.norm_linear(a, wn, 1e-6, "te", w)
    y.float().sum().backward()
    ops.norm_linear(b, wn, 1e-6, "te", w)[0].float().sum().backward()
    assert n == [5, 5] and torch.equal(a.grad, b.grad)


def test_refusals():
    x, wn, w = _rand(4, 256), _rand(256), _rand(512, 256)
    with pytest.raises(RuntimeError):
        torch.vmap(lambda t: ops.rmsnorm(t, wn, 1e-6))(torch.stack([x, x]))
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: _block(t, wn, w))(x)
    a, v = x.clone().requires_grad_(), w.clone().requires_grad_()
    y = ops.linear(a, v)
    with torch.no_grad():
        v.mul_(2)
    with pytest.raises(RuntimeError):
        y.sum().backward()                           # a saved operand was changed
    z = _block(a, wn, w)
    z.backward()
    with pytest.raises(RuntimeError):
        z.backward()                                 # the saved tensors are gone


def test_refusals_name_what_was_handed_over():
    """A weight two bytes off a 16-byte boundary and a rotary width that the kernels do not have: refused on the host, with the operands."""
    from savanna_b200.ops import flash_sm100
    x, w = _rand(4, 128), _rand(64 * 128 + 1)[1:].view(64, 128)
    with pytest.raises(RuntimeError, match=r"gemm_bf16 failed \(code -4.*M=4 N=64 K=128 .*a\[4, 128\]/\[128, 1\] at 0x\w+, b\[64, 128\]/\[128, 1\] at 0x\w+2, out\[4, 64\]"):
        ops.linear(x, w)
    qkv, t = _rand(1, 8, 2, 384), torch.zeros(8, 24, device=DEV)
    with pytest.raises(RuntimeError, match=r"rotary embedding failed \(code -3\): cos\[8, 24\].*from\[1, 8, 2, 128\]/\[6144, 768, 384, 1\]"):
        flash_sm100.attention_packed(qkv, t, t, True)
    assert torch.equal(ops.linear(x, w.clone()), ops.linear(x, w.clone()))


@pytest.mark.parametrize("kind,marked", [("mlp", (2,)), ("mlp", (3,)), ("mlp", (2, 3)), ("norm_linear", (2,))])
def test_joined_nodes_add_into_marked_gradients(kind, marked):
    """Weights whose gradient lives in a persistent buffer get theirs added into it, each into its own; the others get one of their own."""
    ts, whole, parts = _joined(kind)
    ts[0] = ts[0][:, :100]
    g = [_rand(*whole(*ts).shape) for _ in range(2)]
    leaves, plain = _leaves(ts), _leaves(ts)
    buffers = {}
    for i in marked:
        leaves[i].grad = buffers[i] = torch.zeros_like(leaves[i])
        leaves[i]._fuse_grad_accum = True                # what the optimizers with flat buffers set
    for dy in g:
        whole(*leaves).backward(dy)
    want = [torch.autograd.grad(parts(*plain), plain, dy) for dy in g]
    for i, (a, w) in enumerate(zip(leaves, zip(*want))):
        # the buffer's second addition and the sum of the two bf16 gradients round once more than fp32: 2^-8
        total = w[0].float() + w[1].float()
        assert (a.grad.float() - total).norm() <= 2 ** -8 * total.norm(), i
        assert i not in buffers or a.grad is buffers[i]
    assert all(leaves[i].grad.abs().sum() > 0 for i in range(len(ts)))


FIRST_CALL_CAPTURED = """
import torch
from savanna_b200 import ops
from savanna_b200.ops import cuda_ops
torch.manual_seed(0)
args = [torch.randn(2, 300, 192, device="cuda").bfloat16(), torch.randn(4, 64, device="cuda") / 8, torch.randn(64, device="cuda")]
graph = torch.cuda.CUDAGraph()
with torch.no_grad():
    with torch.cuda.graph(graph):
        z = ops.hyena_mr_inner(*args)
    want = ops.hyena_mr_inner(*args)
graph.replay()
assert torch.equal(z, want) and cuda_ops.check_status() == 0
cuda_ops.status_word(z.device).fill_(7 << 24)
graph.replay()
try:
    cuda_ops.check_status()
except RuntimeError as e:
    assert "code 7" in str(e)
    print("kept")
"""


def test_first_call_of_a_process_under_capture():
    """The word for timed-out waits is made at the first call that wants it.  Made on the capturing stream, every replay would clear it."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", FIRST_CALL_CAPTURED], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "kept", r.stdout + r.stderr[-2000:]


FIRST_NORM = """
import sys, torch
from savanna_b200 import ops
D, residual = int(sys.argv[1]), sys.argv[2] == "True"
torch.manual_seed(0)
x, w = (torch.randn(*s, device="cuda").bfloat16() for s in ((37, D), (D,)))
x.requires_grad_(), w.requires_grad_()
y, res = ops.rmsnorm_residual(x, w, 1e-6) if residual else (ops.rmsnorm(x, w, 1e-6), None)
loss = y.float().pow(2).sum() + (res.float().sum() if residual else 0)
loss.backward()
xd, wd = (t.detach().double().requires_grad_() for t in (x, w))
yd = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6) * wd
(yd.pow(2).sum() + (xd.sum() if residual else 0)).backward()
for a, b in ((x.grad, xd.grad), (w.grad, wd.grad)):
    assert (a - b).norm() < 1e-2 * b.norm()
print("ok")
"""


@pytest.mark.parametrize("D,residual", [(3072, False), (2048, True), (2040, True), (2056, True), (3064, False), (3080, False)])
def test_norm_backward_as_the_first_of_a_process(D, residual):
    """A ring of exactly 48 KB, and widths next to it: beside the kernel's own shared memory that is more than a launch gets unasked, and
    asking lasts for the process, so only a process of its own shows it.  bf16 gradients: 2^-9 each of dy, y and the result."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", FIRST_NORM, str(D), str(residual)], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr[-2000:]
