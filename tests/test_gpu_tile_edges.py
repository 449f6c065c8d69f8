"""Tile edges of the sequence kernels: sizes around one tile, partial channel blocks, the shortest and longest filters,
against the fp32 PyTorch statements (ops/reference.py; the decode step: the same decoder stepping operator by operator)."""
import math
import os

import pytest
import torch

from savanna_b200 import ops
from savanna_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV, BF = "cuda", torch.bfloat16
TINY = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "configs", "baseline", "tiny_sh2_gpu.yml")


def _close(a, b, tol, what):
    """Every element within tol of its value plus tol of the tensor's rms (bf16 results: half an ulp is 2^-9 = 0.2 %)."""
    a, b = a.float(), b.float()
    rms = b.pow(2).mean().sqrt().clamp(min=1e-12)
    excess = ((a - b).abs() - tol * (rms + b.abs())).max().item()
    assert excess <= 0, f"{what}: {excess:.4g} outside the bound (rms {rms.item():.4g})"


@pytest.mark.parametrize("B,L,D,O", [(1, 1, 8, 16), (2, 15, 24, 1), (1, 16, 128, 16), (1, 63, 136, 5), (2, 64, 8, 16), (1, 65, 264, 16),
                                     (3, 129, 120, 16), (1, 2049, 16, 8)])
def test_li_scan(B, L, D, O):
    torch.manual_seed(L * 31 + D)
    args = [(torch.randn(B, L, 3 * D, device=DEV) * 0.7).to(BF), (torch.rand(D, O, device=DEV) * 0.09 + 0.01).log(),
            torch.randn(D, O, device=DEV) / math.sqrt(O), -torch.ones(D, O, device=DEV), torch.randn(D, device=DEV)]
    leaves = [t.clone().requires_grad_() for t in args]
    z = ops.hyena_li_modal(*leaves)
    g = torch.randn_like(z)
    z.backward(g)
    rl = [t.float().clone().requires_grad_() for t in args]
    zr = ref.hyena_li_modal(*rl)
    zr.backward(g.float())
    # fp32 recurrence, one bf16 rounding of z / dfeat: 2^-9; 4x for the fp32 FFT of the oracle and cancelling sums
    _close(z, zr, 8e-3, "z")
    _close(leaves[0].grad, rl[0].grad, 8e-3, "dfeat")
    if L > 1:                                            # at L = 1 the pole gradients are zero up to the oracle's FFT noise
        for i, n in ((1, "dgamma"), (3, "dp")):
            _close(leaves[i].grad, rl[i].grad, 2e-3, n)
    _close(leaves[2].grad, rl[2].grad, 2e-3, "dR")
    _close(leaves[4].grad, rl[4].grad, 2e-3, "dbias")


@pytest.mark.parametrize("state", [False, True])
def test_li_scan_pole_gradient_precision(state):
    """Long memories over many chunks, against 64 bits.  In fp32 the poles themselves are rounded: 2^-25 on average, times the length
    of the memory (1 / 0.0037 = 270 steps for the slowest of these poles), is 8e-6 for that mode and 4e-6 over all of them if the
    recurrences use them throughout.  The scan uses exp(T log(pole)) between chunks and corrects what is left of the rounding
    within one: 1.1e-6 by simulation with correctly rounded poles, where the uncorrected sum has 1.5e-6.  The device's expf is
    documented to 2 ulp, so a pole may be off by twice as much and more: 2.2e-6 and 3.0e-6."""
    torch.manual_seed(21)
    B, L, D, O = 1, 4096, 64, 16
    feat, dz = (torch.randn(B, L, 3 * D, device=DEV) * 0.7).to(BF), torch.randn(B, L, D, device=DEV).to(BF)
    g, R, p, b = (torch.rand(D, O, device=DEV) * 0.09 + 0.01).log(), 0.1 * torch.randn(D, O, device=DEV) / 4, -torch.ones(D, O, device=DEV), \
        torch.randn(D, device=DEV)
    gs = torch.randn(B, D, O, device=DEV) if state else None
    leaves = [t.clone().requires_grad_() for t in (g, R, p)]
    z, s = ops.hyena_li_modal(feat, *leaves, b, None, True)
    (z.float() * dz.float()).sum().backward() if gs is None else torch.autograd.backward([z, s], [dz, gs])
    l64 = [t.double().requires_grad_() for t in (g, R, p)]
    x1, x2, v = (feat[..., i::3].double() for i in range(3))
    ll = -torch.exp(l64[2]) * torch.exp(l64[0])
    u = (x2 * v).transpose(1, 2)                                       # [B, D, L]
    t = torch.arange(L, device=DEV, dtype=torch.float64)
    pw = torch.exp(ll[..., None] * t)                                  # [D, O, L]
    h = (l64[1][..., None] * pw).sum(1)
    y = torch.fft.irfft(torch.fft.rfft(u, n=2 * L) * torch.fft.rfft(h, n=2 * L), n=2 * L)[..., :L].transpose(1, 2)
    loss = (x1 * (y + b.double() * u.transpose(1, 2)) * dz.double()).sum()
    if state:
        loss = loss + (torch.einsum("dol,bdl->bdo", pw.flip(-1), u) * gs.double()).sum()
    loss.backward()
    for got, want in ((leaves[0], l64[0]), (leaves[2], l64[2])):
        err = ((got.grad.double() - want.grad).norm() / want.grad.norm()).item()
        assert err <= 2.25e-6, err


@pytest.mark.parametrize("D", [24, 20])                  # the tiled scan, the per-thread one
@pytest.mark.parametrize("gs,Rs,ps,bs,ss", [("DO", "DO", "D1", "D", None), ("DO", "DO", "11", "D", "1DO"), ("DO", "DO", "", "1", "DO"),
                                            ("1O", "DO", "DO", "", "BD1"), ("D1", "1O", "O", "D", "1"), ("1O", "1O", "1O", "D", "11DO")])
def test_li_scan_broadcast_operands(D, gs, Rs, ps, bs, ss):
    """Operands that broadcast to [D, O], [D] and [B, D, O], with their gradients, against the same call with them spelled out."""
    torch.manual_seed(7)
    B, L, O = 3, 70, 5
    n = {"D": D, "O": O, "B": B, "1": 1}

    def rand(form, scale=1.0):
        return (torch.randn([n[c] for c in form], device=DEV) * scale).requires_grad_() if form is not None else None
    feat = (torch.randn(B, L, 3 * D, device=DEV) * 0.7).to(BF)
    args = [rand(gs, 0.3), rand(Rs), rand(ps, 0.3), rand(bs), rand(ss)]
    full = [t.detach().expand(s).clone().requires_grad_() if t is not None else None
            for t, s in zip([*args[:4], args[4][0] if ss == "11DO" else args[4]], [(D, O)] * 3 + [(D,), (B, D, O)])]
    gz, gs_ = torch.randn(B, L, D, device=DEV), torch.randn(B, D, O, device=DEV)
    for a in (args, full):
        z, s = ops.hyena_li_modal(feat, *a, True)
        a.append((z, s))
        ((z.float() * gz).sum() + (s * gs_).sum()).backward()
    assert torch.equal(args[5][0], full[5][0]) and torch.equal(args[5][1], full[5][1])
    for t, f in zip(args[:5], full[:5]):
        if t is not None:
            # the same gradient, summed over the broadcast dimensions (fp32 sums in another order)
            want = f.grad.sum_to_size(t.shape[1:] if t.dim() == 4 else t.shape).view(t.shape)
            assert (t.grad - want).norm() <= 1e-5 * want.norm().clamp(min=1e-3)
    with torch.no_grad():                                # against the fp32 statement
        zr = ref.hyena_li_modal(feat.float(), *[t.detach() if t is not None else None for t in full[:5]])
    _close(full[5][0], zr, 8e-3, "z")


def test_li_scan_host_operands():
    """A host scalar for p is accepted, as PyTorch's operators accept it; a host tensor has no address for the kernels."""
    D, O = 16, 4
    feat, g, R, b = torch.randn(1, 9, 3 * D, device=DEV).to(BF), torch.randn(D, O, device=DEV), torch.randn(D, O, device=DEV), torch.randn(D, device=DEV)
    assert torch.equal(ops.hyena_li_modal(feat, g, R, torch.tensor(-1.0), b), ops.hyena_li_modal(feat, g, R, -torch.ones(D, O, device=DEV), b))
    for i in range(4):
        args = [g, R, -torch.ones(D, O, device=DEV), b]
        args[i] = args[i].cpu()
        with pytest.raises(RuntimeError):
            ops.hyena_li_modal(feat, *args)


@pytest.mark.parametrize("D", [24, 20])
def test_li_scan_state_buffer_reused(D):
    """The caller's state buffer may be overwritten between forward and backward (a running state carried in place)."""
    torch.manual_seed(9)
    B, L, O = 2, 40, 16
    feat = (torch.randn(B, L, 3 * D, device=DEV) * 0.7).to(BF)
    a = [(torch.rand(D, O, device=DEV) * 0.09 + 0.01).log(), torch.randn(D, O, device=DEV) / 4, -torch.ones(D, O, device=DEV),
         torch.randn(D, device=DEV)]
    s0, grads = torch.randn(B, D, O, device=DEV), []
    for overwrite in (False, True):
        leaves, buf = [t.clone().requires_grad_() for t in a], s0.clone()
        z = ops.hyena_li_modal(feat, *leaves, buf)
        if overwrite:
            buf.zero_()
        z.float().sum().backward()
        grads.append([t.grad for t in leaves])
    assert all(torch.equal(x, y) for x, y in zip(*grads))


def test_li_scan_unaligned_view():
    """A contiguous view that starts off a 16-byte boundary."""
    torch.manual_seed(5)
    L, D, O = 40, 16, 16
    buf = torch.randn(L * 3 * D + 1, device=DEV).to(BF)
    feat = buf[1:].view(1, L, 3 * D)
    a = [(torch.rand(D, O, device=DEV) * 0.09 + 0.01).log(), torch.randn(D, O, device=DEV) / 4, -torch.ones(D, O, device=DEV),
         torch.randn(D, device=DEV)]
    assert torch.equal(ops.hyena_li_modal(feat, *a), ops.hyena_li_modal(feat.clone(), *a))


def _same(a, b, what):
    assert torch.equal(torch.nan_to_num(a.float()), torch.nan_to_num(b.float())), what


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_li_scan_non_finite_values_stay_where_they_belong(bad):
    """A non-finite input reaches the outputs of its own channel from its own step on (the adjoint: up to it), and nothing else:
    not the channel that shares its registers, not earlier chunks."""
    torch.manual_seed(11)
    B, L, D, O, t0, c = 2, 300, 24, 16, 133, 5
    feat, dz = (torch.randn(B, L, n * D, device=DEV).to(BF) for n in (3, 1))
    a = [(torch.rand(D, O, device=DEV) * 0.09 + 0.01).log(), torch.randn(D, O, device=DEV) / 4, -torch.ones(D, O, device=DEV),
         torch.randn(D, device=DEV)]

    def run(f, g):
        leaves = [t.clone().requires_grad_() for t in (f, *a)]
        z = ops.hyena_li_modal(*leaves)
        z.backward(g)
        return [z.detach()] + [t.grad for t in leaves]
    clean = run(feat, dz)
    f = feat.clone()
    f[1, t0, 3 * c + 1] = bad
    z, df, dg, dR, dp, db = run(f, dz)
    others = [i for i in range(D) if i != c]
    _same(z[0], clean[0][0], "other sequence"), _same(z[1][:, others], clean[0][1][:, others], "other channels")
    _same(z[1, :t0, c], clean[0][1, :t0, c], "earlier steps")
    assert not z[1, t0:, c].isfinite().any()
    d, dc = df.view(B, L, D, 3), clean[1].view(B, L, D, 3)
    _same(d[:, :, others], dc[:, :, others], "dfeat, other channels"), _same(d[1, :t0, c], dc[1, :t0, c], "dfeat, earlier steps")
    for got, want in zip((dg, dR, dp, db), clean[2:]):
        _same(got[others], want[others], "parameter gradients, other channels")
    assert (dg[c] == 0).all() and (dp[c] == 0).all()               # non-finite pole gradients are dropped
    g = dz.clone()
    g[1, t0, c] = bad
    z, df, *_ = run(feat, g)
    d = df.view(B, L, D, 3)
    _same(z, clean[0], "z"), _same(d[:, :, others], dc[:, :, others], "adjoint, other channels")
    _same(d[1, t0 + 1:, c], dc[1, t0 + 1:, c], "adjoint, later steps")
    assert not d[1, :t0, c, 1:].isfinite().any()


def test_mr_fir_non_finite_values_stay_in_their_column():
    """The Toeplitz products take sixteen steps at a time, zero taps included: a non-finite value reaches its own channel, from the
    start of its sixteen steps to the end of the last sixteen that its taps touch."""
    torch.manual_seed(12)
    B, L, D, G, K, t0, c = 1, 500, 64, 4, 128, 203, 9
    feat, h, b = torch.randn(B, L, 3 * D, device=DEV).to(BF), torch.randn(G, K, device=DEV) / 11, torch.randn(D, device=DEV)
    clean = ops.hyena_mr_inner(feat, h, b)
    feat[0, t0, 3 * c + 2] = float("nan")
    z = ops.hyena_mr_inner(feat, h, b)
    others = [i for i in range(D) if i != c]
    lo, hi = t0 // 16 * 16, t0 // 16 * 16 + 16 + 128
    _same(z[..., others], clean[..., others], "other channels"), _same(z[:, :lo, c], clean[:, :lo, c], "earlier steps")
    _same(z[:, hi:, c], clean[:, hi:, c], "beyond the taps")
    assert z[0, t0:t0 + K, c].isnan().all()


def _mr_grads(halo, *args):
    leaves = [t.clone().requires_grad_() for t in args[:3]]
    z = ops.hyena_mr_inner(*leaves, halo)
    z.backward(args[3])
    return [z.detach()] + [t.grad for t in leaves]


# one row; a tile less one, whole, and one more; an odd and an even number of tiles; several runs per block; a filter for 64 channels
@pytest.mark.parametrize("B,L,D,G,K", [(1, 1, 16, 1, 128), (2, 127, 32, 2, 128), (1, 128, 16, 1, 1), (1, 129, 48, 3, 31), (1, 1025, 64, 1, 128),
                                       (2, 2304, 128, 2, 113), (3, 777, 2048, 128, 128), (5, 300, 1024, 16, 7)])
def test_mr_fir_tiles_of_128_rows_match_the_16_row_blocks(B, L, D, G, K):
    """Without halo rows the products come from whole tiles, with (zero) halo rows from 16-row blocks: the same roundings of the
    operands, fp32 sums in another order, one rounding of the result, which may fall on either side."""
    torch.manual_seed(L + D)
    a = [torch.randn(B, L, 3 * D, device=DEV).to(BF), torch.randn(G, K, device=DEV) / math.sqrt(K), torch.randn(D, device=DEV),
         torch.randn(B, L, D, device=DEV).to(BF)]
    new = _mr_grads(None, *a)
    for got, want, tol, what in zip(new, _mr_grads(torch.zeros(B, K - 1, 3 * D, device=DEV, dtype=BF), *a), (2 ** -7, 2 ** -7, 1e-5, 1e-5),
                                    ("z", "dfeat", "dh", "dbias")):
        _close(got, want, tol, what)
    assert torch.equal(new[0], _mr_grads(None, *a)[0])


# one row and one more than 32; filters of 32 and 33 taps; sizes on both sides of where a short filter keeps the 16-row blocks
@pytest.mark.parametrize("B,L,D,G,K,blocks", [(1, 1, 32, 2, 3, True), (2, 32, 48, 3, 32, True), (1, 33, 48, 3, 32, False), (1, 32, 48, 3, 33, False),
                                              (1, 1023, 1024, 64, 7, False), (1, 1024, 1024, 64, 16, True), (1, 1024, 1024, 64, 17, False),
                                              (4, 2048, 256, 4, 32, True), (4, 2047, 256, 4, 32, False), (4, 2048, 256, 4, 33, False)])
def test_mr_fir_short_filters(B, L, D, G, K, blocks):
    torch.manual_seed(L + K)
    feat, h, bias = torch.randn(B, L, 3 * D, device=DEV).to(BF), torch.randn(G, K, device=DEV) / math.sqrt(K), torch.randn(D, device=DEV)
    with torch.no_grad():
        z, tiled = ops.hyena_mr_inner(feat, h, bias), ops.hyena_mr_inner(feat, h, bias, torch.zeros(B, K - 1, 3 * D, device=DEV, dtype=BF))
    if blocks:
        assert torch.equal(z, tiled)
    _close(z, tiled, 2 ** -7, "z")                        # fp32 sums in another order, one rounding of the result either way
    want = ref.hyena_mr_inner(feat.double(), h.to(BF).double(), bias.double())
    # u rounded to bf16: y is off by 2^-9 / sqrt(3) of its rms (one sigma); that and x1 at most 4.5 sigma; one rounding of the result, 2^-9
    _close(z, want, 4.5 * 4.5 * 2 ** -9 / 3 ** 0.5, "z")


@pytest.mark.parametrize("off", [1, 2, 3])
def test_mr_fir_parameters_off_16_byte_boundaries(off):
    """Taps and bias as views into the middle of a flat buffer, as an optimizer lays them out: the results of aligned copies."""
    from savanna_b200.ops import cuda_ops
    torch.manual_seed(off)
    B, L, D, G, K = 2, 300, 64, 4, 31
    feat, dz = torch.randn(B, L, 3 * D, device=DEV).to(BF), torch.randn(B, L, D, device=DEV).to(BF)
    flat = torch.randn(off + D + off + G * K, device=DEV)
    h, bias = flat[off + D + off:].view(G, K), flat[off:off + D]
    assert bias.data_ptr() % 16 and h.is_contiguous()
    got, want = [], []
    for out, hh, bb in ((got, h, bias), (want, h.clone(), bias.clone())):
        leaves = [feat.clone().requires_grad_(), hh.detach().requires_grad_(), bb.detach().requires_grad_()]
        z = ops.hyena_mr_inner(*leaves)
        z.backward(dz)
        out += [z.detach()] + [t.grad for t in leaves]
    _same(got[0], want[0], "z")
    _same(got[1], want[1], "dfeat")
    for a, b, what in zip(got[2:], want[2:], ("dh", "dbias")):          # atomic sums: any order
        _close(a, b, 1e-5, what)
    # the entry itself takes no such bias (refused on the host, nothing is launched)
    dfeat, dh, db = torch.empty_like(feat), torch.zeros(G, K, device=DEV), torch.zeros(D, device=DEV)
    rc = cuda_ops.require().sb_mr_umma_bwd(feat.data_ptr(), h.data_ptr(), bias.data_ptr(), dz.data_ptr(), dfeat.data_ptr(), dh.data_ptr(),
                                           db.data_ptr(), B, L, D, G, K, cuda_ops.status_word(feat.device).data_ptr(),
                                           torch.cuda.current_stream().cuda_stream)
    assert rc == -1
    cuda_ops.check_status()


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("t0", [130, 200, 511])
def test_mr_fir_non_finite_values_reach_only_what_their_taps_touch(bad, t0):
    torch.manual_seed(13)
    B, L, D, G, K, c = 1, 900, 64, 4, 100, 21
    a = [torch.randn(B, L, 3 * D, device=DEV).to(BF), torch.randn(G, K, device=DEV) / 11, torch.randn(D, device=DEV),
         torch.randn(B, L, D, device=DEV).to(BF)]
    clean = _mr_grads(None, *a)
    a[0][0, t0, 3 * c + 2] = bad
    z, df = _mr_grads(None, *a)[:2]
    others = [i for i in range(D) if i != c]
    _same(z[..., others], clean[0][..., others], "other channels")
    assert not z[0, t0:t0 + K, c].isfinite().any()
    for part in (slice(0, t0), slice(t0 + K, L)):      # formed again tap by tap next to the bad value: fp32 sums in another order
        _close(z[:, part, c], clean[0][:, part, c], 2 ** -7, "beyond the taps")
    a[0][0, t0, 3 * c + 2] = 1.0
    a[3][0, t0, c] = bad
    df = _mr_grads(None, *a)[1].view(B, L, D, 3)
    want = clean[1].view(B, L, D, 3)
    _same(df[:, :, others], want[:, :, others], "dfeat, other channels")
    assert not df[0, t0 - K + 1:t0 + 1, c, 1:].isfinite().any()
    for part in (slice(0, t0 - K + 1), slice(t0 + K, L)):
        _close(df[:, part, c], want[:, part, c], 2 ** -7, "dfeat beyond the taps")
    _close(df[:, t0 + 1:, c, 1:], want[:, t0 + 1:, c, 1:], 2 ** -7, "gradients of x2 and v behind the value")     # anticausal: not reached


# near both ends of the sequence and of its tiles and of the runs of tiles that a block takes
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("L,t0", [(900, 0), (900, 50), (900, 127), (900, 128), (900, 768), (900, 801), (900, 850), (900, 899), (130, 125), (128, 127),
                                  (20, 3), (4096, 4090)])
def test_mr_fir_non_finite_values_reach_only_the_taps_they_meet(bad, L, t0):
    """A non-finite u[t0] meets g[t0 + s] in the gradient of tap s, a non-finite g[t0] meets u[t0 - s]: taps without such a row stay as they are."""
    torch.manual_seed(17)
    B, D, G, K, c = 2, 64, 4, 100, 21
    a = [torch.randn(B, L, 3 * D, device=DEV).to(BF), torch.randn(G, K, device=DEV) / 11, torch.randn(D, device=DEV),
         torch.randn(B, L, D, device=DEV).to(BF)]
    g, others, taps = c // (D // G), [i for i in range(D) if i != c], torch.arange(K, device=DEV)
    v0, clean = a[0][1, t0, 3 * c + 2].item(), _mr_grads(None, *a)
    for what, met in (("u", taps <= L - 1 - t0), ("g", taps <= t0)):
        a[0][1, t0, 3 * c + 2] = bad if what == "u" else v0
        a[3][1, t0, c] = a[3][1, t0, c] if what == "u" else bad
        dh, db = _mr_grads(None, *a)[2:]
        _close(dh[[i for i in range(G) if i != g]], clean[2][[i for i in range(G) if i != g]], 1e-5, what + ": dh, other groups")
        _close(db[others], clean[3][others], 1e-5, what + ": dbias, other channels")
        assert not dh[g, met].isfinite().any() and not db[c].isfinite()
        if (~met).any():                                  # formed again row by row: fp32 sums in another order
            _close(dh[g, ~met], clean[2][g, ~met], 1e-5, what + ": dh, taps that meet no such value")


@pytest.mark.parametrize("D,offset,tiled", [(24, 0, True), (136, 0, True), (20, 0, False), (24, 1, False)])
@pytest.mark.parametrize("state", [False, True])
def test_li_c_entries(D, offset, tiled, state):
    """`sb_li_fwd` / `sb_li_bwd` on prepared log-poles: the tiled kernels where the shape and the alignment allow, the per-thread
    ones elsewhere, the same numbers from both."""
    from savanna_b200.ops import cuda_ops
    lib = cuda_ops.require()
    torch.manual_seed(D + offset)
    B, L, O, st = 2, 200, 16, torch.cuda.current_stream().cuda_stream

    def buf(*shape, dtype=torch.float32):
        n = math.prod(shape)
        t = torch.zeros(n + offset, device=DEV, dtype=dtype)[offset:].view(shape) if dtype == BF else torch.zeros(shape, device=DEV)
        return t
    feat, dz, z = buf(B, L, 3 * D, dtype=BF), buf(B, L, D, dtype=BF), buf(B, L, D, dtype=BF)
    feat.copy_(torch.randn(B, L, 3 * D, device=DEV) * 0.7), dz.copy_(torch.randn(B, L, D, device=DEV))
    g, R, p, bias = (torch.rand(D, O, device=DEV) * 0.09 + 0.01).log(), torch.randn(D, O, device=DEV) / 4, -torch.ones(D, O, device=DEV), \
        torch.randn(D, device=DEV)
    s_in = torch.randn(B, D, O, device=DEV) if state else None
    ll = -torch.exp(p) * torch.exp(g)

    def ptr(t):
        return t.data_ptr() if t is not None else None
    tc = lib.sb_li_bwd_chunk(D, 128)
    assert tc == (64 if D % 8 == 0 else 128)
    nf, nb = -(-L // 96), -(-L // tc)
    S, sout = buf(B, nf, D, 16), buf(B, D, 16)
    Sb, W, A, dRp, dLp = (buf(B, nb, D, 16) for _ in range(5))
    dBp, tmp, df, dsi = buf(B, nb, D), buf(B, L, D, dtype=BF), buf(B, L, 3 * D, dtype=BF), buf(B, D, 16)
    torch.cuda.synchronize()
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        assert lib.sb_li_fwd(ptr(feat), ptr(ll), ptr(R), ptr(bias), ptr(s_in), ptr(sout), ptr(S), ptr(z), B, L, D, 96, st) == 0
        assert lib.sb_li_bwd(ptr(feat), ptr(dz), ptr(ll), ptr(R), ptr(bias), ptr(s_in), None, ptr(Sb), ptr(W), ptr(A), ptr(dRp), ptr(dLp),
                             ptr(dBp), ptr(tmp), ptr(df), None, ptr(dsi) if state else None, B, L, D, tc, st) == 0
        torch.cuda.synchronize()
    names = [e.key for e in prof.key_averages()]
    if any("li_" in n for n in names):                   # (no kernel names where the profiler has no access to the device)
        assert all(("tiled" in n) == tiled for n in names if "li_" in n), names
    leaves = [t.float().clone().requires_grad_() for t in (feat, g, R, p, bias)]
    sr = s_in.clone().requires_grad_() if state else None
    zr, sor = ref.hyena_li_modal(*leaves, sr, True)
    zr.backward(dz.float())
    lam = torch.exp(ll)
    _close(z, zr, 8e-3, "z")                             # as in test_li_scan
    _close(df, leaves[0].grad, 8e-3, "dfeat")
    _close(sout, sor, 2e-3, "state_out")
    _close(dRp.sum((0, 1)), leaves[2].grad, 2e-3, "dR")
    _close(dLp.sum((0, 1)) * lam * ll, leaves[1].grad, 2e-3, "dgamma")
    _close(dBp.sum((0, 1)), leaves[4].grad, 2e-3, "dbias")
    if state:
        _close(dsi, sr.grad, 2e-3, "dstate_in")


@pytest.mark.parametrize("B,L,D,G,K", [(1, 1, 16, 1, 128), (2, 31, 16, 1, 1), (1, 32, 80, 5, 16), (1, 33, 64, 1, 17), (2, 160, 48, 3, 113),
                                       (1, 161, 144, 9, 128), (1, 700, 64, 4, 31)])
@pytest.mark.parametrize("halo", [False, True])
def test_mr_fir(B, L, D, G, K, halo):
    torch.manual_seed(L * 7 + K)
    f, h, b = torch.randn(B, L, 3 * D, device=DEV).to(BF), torch.randn(G, K, device=DEV) / math.sqrt(K), torch.randn(D, device=DEV)
    hal = torch.randn(B, K - 1, 3 * D, device=DEV).to(BF) if halo and K > 1 else None
    leaves = [t.clone().requires_grad_() for t in (f, h, b)] + ([hal.clone().requires_grad_()] if hal is not None else [])
    z = ops.hyena_mr_inner(*leaves)
    g = torch.randn_like(z)
    z.backward(g)
    rl = [t.float().clone().requires_grad_() for t in (f, h, b)] + ([hal.float().clone().requires_grad_()] if hal is not None else [])
    zr = ref.hyena_mr_inner(*rl)
    zr.backward(g.float())
    # bf16 operands of the Toeplitz products (u, taps): two roundings of up to 2^-9 per term leave y and du an error of 0.2 %
    # of their rms, 4 sigma over the elements, and z, dfeat multiply it by a factor of up to 4 times its rms: 3.2 %
    _close(z, zr, 3.2e-2, "z")
    _close(leaves[0].grad, rl[0].grad, 3.2e-2, "dfeat")
    if hal is not None:
        _close(leaves[3].grad, rl[3].grad, 3.2e-2, "dhalo")
    # dh sums bf16-rounded products: relative to the norm of the whole gradient
    assert (leaves[1].grad - rl[1].grad).norm() <= 1e-2 * rl[1].grad.norm()
    assert (leaves[2].grad - rl[2].grad).norm() <= 1e-4 * rl[2].grad.norm()


@pytest.mark.parametrize("B,T,steps", [(1, 1, 3), (2, 5, 70), (3, 130, 5), (8, 64, 4)])
def test_decode_step(B, T, steps):
    """The native decode step against the operator-by-operator one: short prompts (rings that start zero-padded), key caches
    that grow, every batch size class.  Each is within 1.1 % (relative 2-norm of the logits) of the model in 64 bits, bf16
    activations being the cause, and they round at different places (a residual addition once or twice): 2.2 % apart."""
    from savanna_b200.config import GlobalConfig
    from savanna_b200.inference.cached import CachedDecoder
    from savanna_b200.models import build_model
    cfg = GlobalConfig.from_ymls([TINY], {"global_num_gpus": 1})
    cfg.build_tokenizer()
    torch.manual_seed(0)
    model = build_model(cfg, device=DEV)
    with torch.no_grad():
        for n, p in model.named_parameters():
            if n.endswith("filter.h"):
                p.mul_(3e4)
    toks = torch.randint(0, 256, (B, T + steps), device=DEV)
    fast, slow = CachedDecoder(model), CachedDecoder(model)
    a, b = fast.prefill(toks[:, :T]), slow.prefill(toks[:, :T])
    assert fast._fused is not None and torch.equal(a, b)
    from savanna_b200.inference import cached
    build = cached._FusedStep.build
    cached._FusedStep.build = staticmethod(lambda *_: None)
    try:
        slow.prefill(toks[:, :T])
    finally:
        cached._FusedStep.build = build
    for i in range(steps):
        a, b = fast.step(toks[:, T + i]), slow.step(toks[:, T + i])
        assert a.shape == b.shape and a.dtype == b.dtype
        assert (a - b).norm() <= 2.2e-2 * b.norm(), (i, ((a - b).norm() / b.norm()).item())
    with pytest.raises(ValueError):
        fast.step(toks[:1, 0].repeat(B + 1))


@pytest.mark.parametrize("L", [1, 63, 64, 65, 127, 128, 129, 256, 300, 641])
@pytest.mark.parametrize("causal", [True, False])
def test_attention_tiles(L, causal):
    """One tile more or less than the 64- and 128-row tiles of the kernels, forward and backward."""
    torch.manual_seed(L)
    q, k, v = (torch.randn(2, L, 3, 128, device=DEV).to(BF).requires_grad_() for _ in range(3))
    o = ops.attention(q, k, v, causal)
    g = torch.randn_like(o)
    o.backward(g)
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    orf = ref.attention(qr, kr, vr, causal)
    orf.backward(g.float())
    from savanna_b200.ops import cuda_ops
    cuda_ops.check_status()
    # bf16 probabilities and score gradients as MMA operands, one rounding (up to 2^-8) in each of three factors of a term and
    # one of the result; the terms of dq and dk cancel to about half their size: 4 % of value plus rms
    for got, want, n in ((o, orf, "o"), (q.grad, qr.grad, "dq"), (k.grad, kr.grad, "dk"), (v.grad, vr.grad, "dv")):
        if L == 1 and n in ("dq", "dk"):                     # one key: the softmax is constant, the gradients are zero
            assert got.abs().max() <= 1e-5, n
        else:
            _close(got, want, 4e-2, n)


def test_packed_attention_rotary():
    """Partial rotary dimensions and odd lengths of the packed projection, against the unpacked statement."""
    for rd, L, H in ((16, 5, 1), (64, 70, 3), (128, 129, 33)):
        torch.manual_seed(rd)
        qkv = torch.randn(1, L, H, 384, device=DEV).to(BF).requires_grad_()
        cos, sin = ref.rope_tables(torch.arange(L, device=DEV), rd)
        o = ops.attention_packed(qkv, cos, sin, True)
        g = torch.randn_like(o)
        o.backward(g)
        qr = qkv.detach().float().requires_grad_()
        orf = ref.attention(ref.apply_rope(qr[..., :128], cos, sin), ref.apply_rope(qr[..., 128:256], cos, sin), qr[..., 256:], True)
        orf.backward(g.float())
        _close(o, orf, 2e-2, "o")                        # bf16 rotated q, k and probabilities: three roundings of up to 2^-8
        _close(qkv.grad, qr.grad, 4e-2, "dqkv")          # as in test_attention_tiles, and the rounded q, k enter the scores


@pytest.mark.parametrize("H,rd", [(4, 128), (5, 32), (130, 64)])
def test_rotary_heads(H, rd):
    """Head counts that leave a thread of the packed rotary kernel short of its four heads (5) or send it round again (130): the
    rotated queries and keys are written in place, the rest of the packed tensor stays as it was."""
    import ctypes
    from savanna_b200.ops import cuda_ops
    cuda_ops.require()
    entry = ctypes.CDLL(cuda_ops._LIB_PATH).sb_attn_rope
    L = 3
    torch.manual_seed(H)
    qkv = torch.randn(2, L, H, 384, device=DEV).to(BF)
    cos, sin = ref.rope_tables(torch.arange(L, device=DEV), rd)
    out = qkv.clone()
    views = [out[..., :128], out[..., 128:256]]
    ptrs = (ctypes.c_void_p * 2)(*[v.data_ptr() for v in views])
    strides = (ctypes.c_longlong * 6)(*[s for v in views for s in v.stride()[:3]])
    cos, sin = cos.float().contiguous(), sin.float().contiguous()
    assert entry(ptrs, ptrs, strides, strides, (ctypes.c_int * 2)(0, 0), 2, ctypes.c_void_p(cos.data_ptr()),
                 ctypes.c_void_p(sin.data_ptr()), 2, L, H, rd, 0, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    for i, v in enumerate(views):
        want = ref.apply_rope(qkv[..., 128 * i:128 * i + 128].float(), cos, sin)
        _close(v, want, 2.0 ** -8, "qk"[i])              # one rounding to bf16
    assert torch.equal(out[..., 256:], qkv[..., 256:])


def _conv_grads(B, L, D, G, K, halo, pre=True, post=True, bf16_taps=False):
    torch.manual_seed(L + K)
    feat, w = torch.randn(B, L, 3 * D, device=DEV).to(BF), torch.randn(G, K, device=DEV) * 0.4
    if bf16_taps:
        w = w.to(BF)
    h = torch.randn(B, K - 1, 3 * D, device=DEV).to(BF) if halo else None
    g = torch.randn(B, L, D, device=DEV).to(BF)
    out = []
    for f32 in (False, True):
        a = [None if t is None else (t.float() if f32 else t.clone()).requires_grad_() for t in (feat, w, h)]
        z = (ref if f32 else ops).hyena_se_inner(a[0], a[1], a[2], pre, post)
        z.backward(g.float() if f32 else g)
        out.append([z.detach()] + [t.grad for t in a if t is not None])
    return out


# rows of 128 channels per SM: at least 200 on a chip of 148 SMs, where the streaming kernels start; runs that end on an odd row, strips
# of 128 channels that are not full, groups of fewer than four channels (their taps differ within a lane), every filter length
@pytest.mark.parametrize("B,L,D,G,K", [(1, 3703, 1024, 64, 7), (2, 1901, 1016, 127, 2), (3, 1301, 1000, 500, 3), (1, 1, 8, 1, 7),
                                       (1, 3801, 1016, 254, 4), (2, 1999, 904, 452, 5), (1, 4001, 1024, 8, 6), (5, 797, 1024, 1024, 8)])
@pytest.mark.parametrize("halo", [False, True])
def test_se_streaming(B, L, D, G, K, halo):
    got, want = _conv_grads(B, L, D, G, K, halo, bf16_taps=K == 7)
    # fp32 sums, one bf16 rounding of the result: 2^-9; bf16 taps round their gradient once more
    for a, b, n in zip(got, want, ("z", "dfeat", "dtaps", "dhalo")):
        _close(a, b, 4e-3, n)


@pytest.mark.parametrize("pre,post", [(False, True), (True, False), (False, False)])
def test_se_streaming_gates(pre, post):
    for a, b in zip(*_conv_grads(1, 3701, 1024, 64, 7, True, pre, post)):
        _close(a, b, 4e-3, (pre, post))


@pytest.mark.parametrize("B,L,C,K", [(1, 1301, 3072, 3), (2, 1901, 1016, 2), (3, 1301, 1000, 4), (1, 3801, 1016, 8), (2, 1999, 904, 5), (1, 2, 8, 3)])
@pytest.mark.parametrize("halo", [False, True])
def test_featuriser_streaming(B, L, C, K, halo):
    torch.manual_seed(L + K)
    x, w = torch.randn(B, L, C, device=DEV).to(BF), torch.randn(C, K, device=DEV).to(BF)
    h, g = torch.randn(B, K - 1, C, device=DEV).to(BF) if halo else None, torch.randn(B, L, C, device=DEV).to(BF)
    out = []
    for f32 in (False, True):
        a = [None if t is None else (t.float() if f32 else t.clone()).requires_grad_() for t in (x, w, h)]
        y = (ref if f32 else ops).causal_conv1d(*a)
        y.backward(g.float() if f32 else g)
        out.append([y.detach()] + [t.grad for t in a if t is not None])
    for a, b, n in zip(*out, ("y", "dx", "dtaps", "dhalo")):
        _close(a, b, 4e-3, n)


@pytest.mark.parametrize("L,D,K", [(3702, 1024, 7), (3710, 1088, 4)])
def test_conv_streaming_chunks(L, D, K):
    """Two chunks of one sequence as batch rows, their edge rows handed over as the context-parallel entry points take them: rows before
    each chunk, and rows after it for the backward; the pieces together are the whole sequence's results."""
    from savanna_b200.ops import cuda_ops
    from savanna_b200.parallel import halo_fused
    import ctypes
    torch.manual_seed(L)
    lib, c, H, G, C, st = cuda_ops.require(), L // 2, K - 1, D // 16, 3 * D, torch.cuda.current_stream().cuda_stream
    P, I, S = ctypes.c_void_p, ctypes.c_int, ctypes.POINTER(halo_fused.HaloSrc)
    lib.sb_dwconv_bwd_cp.argtypes = [P, S, P, P, S, P, P, I, I, I, I, P]
    lib.sb_se_fwd_cp.argtypes = [P, S, P, P, I, I, I, I, I, I, I, P]
    lib.sb_se_bwd_cp.argtypes = [P, S, P, P, S, S, P, P, I, I, I, I, I, I, I, P]
    f, g, gx = (torch.randn(1, L, n, device=DEV).to(BF) for n in (C, D, C))
    w, wc = torch.randn(G, K, device=DEV) * 0.4, torch.randn(C, K, device=DEV)

    def edges(t, after):
        zero = torch.zeros(1, H, t.shape[2], device=DEV, dtype=BF)
        e = torch.cat([t[:, c:c + H], zero] if after else [zero, t[:, c - H:c]]).contiguous()
        return e, halo_fused.HaloSrc(e.data_ptr(), e.data_ptr(), 0, 0, 0)

    (k0, bf_), (k1, af), (k2, ag), (k3, agx) = edges(f, False), edges(f, True), edges(g, True), edges(gx, True)
    z, df, dx = torch.empty_like(g), torch.empty_like(f), torch.empty_like(f)
    dw, dwc = torch.zeros_like(w), torch.zeros_like(wc)
    assert lib.sb_se_fwd_cp(f.data_ptr(), ctypes.byref(bf_), w.data_ptr(), z.data_ptr(), 2, c, D, G, K, 1, 1, st) == 0
    assert lib.sb_se_bwd_cp(f.data_ptr(), ctypes.byref(bf_), w.data_ptr(), g.data_ptr(), ctypes.byref(af), ctypes.byref(ag), df.data_ptr(),
                            dw.data_ptr(), 2, c, D, G, K, 1, 1, st) == 0
    assert lib.sb_dwconv_bwd_cp(f.data_ptr(), ctypes.byref(bf_), wc.data_ptr(), gx.data_ptr(), ctypes.byref(agx), dx.data_ptr(), dwc.data_ptr(),
                                2, c, C, K, st) == 0
    torch.cuda.synchronize()
    a, b = f.float().requires_grad_(), w.clone().requires_grad_()
    zr = ref.hyena_se_inner(a, b)
    zr.backward(g.float())
    x, v = f.float().requires_grad_(), wc.clone().requires_grad_()
    ref.causal_conv1d(x, v).backward(gx.float())
    for got, want, n in ((z, zr, "z"), (df, a.grad, "dfeat"), (dw, b.grad, "dtaps"), (dx, x.grad, "dx"), (dwc, v.grad, "dconv")):
        _close(got.view(want.shape), want, 4e-3, n)


# rows in pairs: one row, odd counts, more and fewer pairs than blocks; widths of one vector per thread (not a multiple of a warp among them,
# the widest 4096) and beyond
@pytest.mark.parametrize("T,D", [(1, 64), (3, 72), (2, 4096), (597, 2816), (1185, 256), (37, 4104), (2371, 1024)])
@pytest.mark.parametrize("form", ["te", "classic"])
def test_rmsnorm_rows_in_pairs(T, D, form):
    torch.manual_seed(T)
    x, w, g, gr = (torch.randn(*s, device=DEV).to(BF) for s in ((T, D), (D,), (T, D), (T, D)))
    a, b = x.clone().requires_grad_(), w.clone().requires_grad_()
    y, res = ops.rmsnorm_residual(a, b, 1e-6, form)
    torch.autograd.backward([y, res], [g, gr])
    ar, br = x.float().requires_grad_(), w.float().requires_grad_()
    yr = ref.rmsnorm(ar, br, 1e-6, form)
    torch.autograd.backward([yr, ar * 1], [g.float(), gr.float()])
    # fp32 sums, one bf16 rounding of each result: 2^-9
    for got, want, n in ((y, yr, "y"), (a.grad, ar.grad, "dx"), (b.grad, br.grad, "dw")):
        _close(got, want, 4e-3, n)


# outputs with few 256 x 256 tiles take 128 x 128 or 128 x 64 tiles: partial tiles in both directions, contractions shorter than the ring
# of stages and with a ragged end, every operand order, bias, residual and accumulation
@pytest.mark.parametrize("M,N,K", [(8, 8, 8), (999, 1024, 2816), (130, 72, 64), (512, 4096, 1000), (768, 256, 2048), (1, 200, 4096), (257, 136, 520)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_gemm_narrow_tiles(M, N, K, a_mn, b_mn):
    from savanna_b200.ops import cuda_ops
    torch.manual_seed(M + N)
    if (a_mn and M % 8) or (b_mn and N % 8):
        pytest.skip("rows of a transposed operand start on 16-byte boundaries")
    assert cuda_ops.gemm_tile(M, N) in (64, 128)
    a, b = torch.randn(M, K, device=DEV).to(BF), torch.randn(N, K, device=DEV).to(BF)
    bias, res = torch.randn(N, device=DEV).to(BF), torch.randn(M, N, device=DEV).to(BF)
    out = res.clone()
    cuda_ops.gemm(a.t().contiguous() if a_mn else a, b.t().contiguous() if b_mn else b, out, a_mn, b_mn, bias=bias, accumulate=True, residual=res)
    want = a.float() @ b.float().t() + bias.float() + 2 * res.float()
    # fp32 accumulation, one bf16 rounding (two where the old value is added after the first): 2^-8
    _close(out, want, 8e-3, "gemm")


# blocks of the backward's passes against the SMs: each with an SM of its own, more prefix blocks than SMs, one row of blocks short of a full
# chip and a full one (148 SMs: D = 1024 has 8 blocks for a chunk of 64 steps)
@pytest.mark.parametrize("B,L,D", [(1, 300, 256), (2, 300, 256), (1, 1152, 1024), (1, 1217, 1024)])
@pytest.mark.parametrize("state", [False, True])
def test_li_backward_launch_forms(B, L, D, state):
    torch.manual_seed(L + D)
    O = 16
    args = [(torch.randn(B, L, 3 * D, device=DEV) * 0.7).to(BF), (torch.rand(D, O, device=DEV) * 0.09 + 0.01).log(),
            torch.randn(D, O, device=DEV) / math.sqrt(O), -torch.ones(D, O, device=DEV), torch.randn(D, device=DEV)]
    args += [torch.randn(B, D, O, device=DEV)] if state else []
    g, gs = torch.randn(B, L, D, device=DEV).to(BF), torch.randn(B, D, O, device=DEV)

    def grads(fn, f32):
        leaves = [(t.float() if f32 else t).clone().requires_grad_() for t in args]
        out = fn(*leaves, *([True] if state else []))
        torch.autograd.backward(out, (g.float() if f32 else g, gs) if state else g.float() if f32 else g)
        return [t.grad for t in leaves]
    want = grads(ref.hyena_li_modal, True)
    first = grads(ops.hyena_li_modal, False)
    for _ in range(3):                                   # every sum has a fixed order
        assert all(torch.equal(a, b) for a, b in zip(first, grads(ops.hyena_li_modal, False)))
    for a, b, n in zip(first, want, ("dfeat", "dgamma", "dR", "dp", "dbias", "dstate")):
        _close(a, b, 8e-3 if n == "dfeat" else 2e-3, n)  # as in test_li_scan


def test_refused_launch_is_reported_once():
    """More sequences than a grid has layers: the scan's launch is refused, and the next operator on this thread is none the wiser."""
    B, D, O = 65536, 8, 16
    x, w = torch.randn(4, 128, device=DEV).to(BF), torch.ones(128, device=DEV, dtype=BF)
    want = ops.rmsnorm(x, w, 1e-6)
    feat, g = torch.randn(B, 1, 3 * D, device=DEV).to(BF), torch.zeros(D, O, device=DEV)
    with torch.no_grad():
        with pytest.raises(RuntimeError, match="code -2"):
            ops.hyena_li_modal(feat, g, g, g, torch.zeros(D, device=DEV))
        assert torch.equal(ops.rmsnorm(x, w, 1e-6), want)
        assert ops.hyena_li_modal(feat[:4], g, g, g, torch.zeros(D, device=DEV)).shape == (4, 1, D)


# narrow tiles of which a CTA takes two or more (148 SMs): both accumulators, their barriers' phases, a ring of stages that goes on into the
# next tile; partial tiles at both edges, contractions shorter and longer than the ring
@pytest.mark.parametrize("M,N,K,width", [(384, 10240, 520, 128), (333, 22528, 200, 128), (19001, 56, 200, 64), (38301, 64, 1032, 64)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("fp8", [False, True])
def test_gemm_narrow_tiles_in_turn(M, N, K, width, a_mn, b_mn, fp8):
    from savanna_b200.ops import cuda_ops
    torch.manual_seed(M + N)
    unit = 16 if fp8 else 8
    if fp8:
        K += -K % 16                                     # rows of an fp8 operand start on 16-byte boundaries
    if a_mn:
        M += -M % unit
    if b_mn:
        N += -N % unit
    want_width = 128 if fp8 and b_mn else width          # an MN-major fp8 operand comes in boxes of 128 columns
    assert cuda_ops.gemm_tile(M, N, fp8, b_mn) == want_width and -(-M // 128) * -(-N // want_width) > 148
    a, b = torch.randn(M, K, device=DEV).to(BF), torch.randn(N, K, device=DEV).to(BF)
    out = torch.full((M, N), float("nan"), device=DEV, dtype=BF)
    if fp8:
        (aq, sa), (bq, sb_) = (cuda_ops.quantize_fp8(t.t().contiguous() if mn else t, 0) for t, mn in ((a, a_mn), (b, b_mn)))
        cuda_ops.gemm_fp8(aq, bq, out, sa, alpha2=sb_, a_mn=a_mn, b_mn=b_mn)
        a, b = (q.view(torch.float8_e4m3fn).float() * s for q, s in ((aq, sa), (bq, sb_)))
        a, b = a.t() if a_mn else a, b.t() if b_mn else b
    else:
        cuda_ops.gemm(a.t().contiguous() if a_mn else a, b.t().contiguous() if b_mn else b, out, a_mn, b_mn)
    cuda_ops.check_status()
    _close(out, a.float() @ b.float().t(), 4e-3, "gemm")  # fp32 accumulation, one bf16 rounding: 2^-9


# the forward norm takes four rows of one warp to a block, or a row to a block of 2 to 16 warps, by its width and the rows per SM: the widths at
# which that changes and the next one up, rows that fill the last block of four and rows that do not, few and many
@pytest.mark.parametrize("form", ["te", "classic"])
@pytest.mark.parametrize("D", [8, 264, 512, 520, 1024, 1032, 2048, 2056, 4096, 4104, 8192, 8200, 16384])
@pytest.mark.parametrize("T", [1, 3, 4, 5, 3001])
def test_norm_rows_and_widths(T, D, form):
    from savanna_b200.ops import cuda_ops
    torch.manual_seed(T + D)
    x, w = torch.randn(T + 1, D, device=DEV).to(BF), (1 + 0.1 * torch.randn(D, device=DEV)).to(BF)
    x[T] = float("nan")                                   # the row behind the last one
    _, _, a, y = cuda_ops._rmsnorm_fwd(x[:T], w, 1e-6, 0 if form == "te" else 1)
    ms = x[:T].double().pow(2).mean(-1)
    want_a = (ms + 1e-6).rsqrt() if form == "te" else 1 / (ms.sqrt() + 1e-6)
    # a lane adds up to 64 squares, then 8 more sums: 72 * 2^-24, halved by the root, and two ulp of the root itself
    assert ((a.double() - want_a).abs() / want_a).max() < 2.5e-6
    _close(y, x[:T].double() * want_a[:, None] * w.double(), 2.0 ** -8, "y")   # one bf16 rounding, 2^-9

    # one byte out: the bf16 result under the scale that the history gives (its maximum, 3, outside this call's two slots)
    hist, si = torch.tensor([3.0, 0.5, 0.0, 9.0], device=DEV), torch.empty(1, device=DEV)
    q, a8 = torch.full((T + 1, D), 0x55, device=DEV, dtype=torch.uint8), torch.empty(T, device=DEV)
    rc = cuda_ops.require().sb_rmsnorm_fwd_fp8(x.data_ptr(), w.data_ptr(), q.data_ptr(), a8.data_ptr(), T, D, 1e-6, 0 if form == "te" else 1,
                                               hist.data_ptr(), 4, 2, si.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and torch.equal(a8, a) and (q[T] == 0x55).all()
    got, want = q[:T].view(torch.float8_e4m3fn).float() * (3.0 / 448), y.float().clamp(-3, 3)
    assert ((got - want).abs() <= 2.0 ** -4 * 1.00001 * want.abs() + 2.0 ** -10 * 3 / 448).all()     # half a step of e4m3; below 2^-6 2^-10
    assert hist.tolist() == [3.0, 0.5, y.float().abs().max().item(), 0.0]


def _sum_of_squares(x):
    """fp32 sum of a row's squares (exact products of bf16 values) in the order of a block with a thread for each of 512 vectors of eight."""
    T, D = x.shape
    p = torch.nn.functional.pad(x.float().square(), (0, -D % 4096)).view(T, -1, 512, 8)
    s = torch.zeros(T, 512, device=x.device)
    for g in range(p.shape[1]):
        for j in range(8):
            s = s + p[:, g, :, j]
    s = s.view(T, 16, 32)
    for o in (16, 8, 4, 2, 1):
        s = s[..., :o] + s[..., o:2 * o]
    s = s[..., 0]
    for o in (8, 4, 2, 1):
        s = s[..., :o] + s[..., o:2 * o]
    return s[:, 0]


@pytest.mark.parametrize("D", [8, 256, 264, 512, 520, 768, 1024, 1032, 2040, 2048, 2056, 4096, 4104, 8192, 8200, 12296, 16384])
@pytest.mark.parametrize("T", [1, 5, 149, 741, 1037, 1500, 15000])
def test_norm_sums_have_one_order_at_all_widths(T, D):
    from savanna_b200.ops import cuda_ops
    torch.manual_seed(T + D)
    x, w = torch.randn(T, D, device=DEV).to(BF), torch.ones(D, device=DEV, dtype=BF)
    _, _, a, _ = cuda_ops._rmsnorm_fwd(x, w, 1e-6, 1)
    mean = _sum_of_squares(x) / torch.full((T,), float(D), device=DEV)
    assert torch.equal(a, torch.ones_like(mean) / (mean.sqrt() + torch.full_like(mean, 1e-6)))


@pytest.mark.parametrize("M,N,K", [(64, 64, 64), (999, 1024, 264), (512, 4096, 4096), (8192, 512, 512), (8192, 2048, 256)])
@pytest.mark.parametrize("captured", [False, True])
def test_gemm_behind_the_kernel_that_feeds_it(M, N, K, captured):
    """A GEMM's launch does not wait for the kernel before it to be done: what it reads (operands, residual, C) and writes over is what it
    would be with the device idle between the launches, behind other kernels and another GEMM, eagerly and in a graph.  None of these lets
    its successor start before its own last block ends; the kernels of the next test do."""
    from savanna_b200.ops import cuda_ops
    torch.manual_seed(M + K)
    x, w, v = (torch.randn(*s, device=DEV).to(BF) for s in ((M, K), (N, K), (K, N)))
    a, y, z, c = torch.empty_like(x), torch.empty(M, N, device=DEV, dtype=BF), torch.empty(M, K, device=DEV, dtype=BF), torch.empty(M, N, device=DEV, dtype=BF)

    def steps(between=lambda: None):
        for i in range(4):
            torch.mul(x, 1.0 + 0.5 * i, out=a); between()
            cuda_ops.gemm(a, w, y); between()
            cuda_ops.gemm(y, v, z); between()                        # [M, N] x [K, N]^T
            torch.add(z, a, out=a); between()
            c.zero_(); between()
            cuda_ops.gemm(a, w, c, residual=y); between()            # the residual is two kernels old
            cuda_ops.gemm(x, w, c, accumulate=True); between()
            torch.mul(c, 0.01, out=y); between()
    for t in (a, y, z, c):
        t.zero_()
    steps(torch.cuda.synchronize)
    want = [t.clone() for t in (a, y, z, c)]
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            steps()
    for _ in range(3):
        for t in (a, y, z, c):
            t.fill_(float("nan"))
        graph.replay() if captured else steps()
        assert all(torch.equal(p, q) for p, q in zip((a, y, z, c), want))
    cuda_ops.check_status()


@pytest.mark.parametrize("B,L,H", [(1, 1, 1), (2, 333, 3), (1, 1024, 8), (1, 2600, 16)])
@pytest.mark.parametrize("captured", [False, True])
def test_attention_behind_the_kernel_that_feeds_it(B, L, H, captured):
    """As above for the rotary embedding of what a kernel has just written and the attention behind it."""
    torch.manual_seed(B * L + H)
    x = (torch.randn(B, L, 3 * H * 128, device=DEV) * 0.5).to(BF)
    cos, sin = (f(torch.rand(L, 128, device=DEV) * 6) for f in (torch.cos, torch.sin))
    qkv = torch.empty_like(x)

    def steps(between=lambda: None):
        out = []
        for i in range(4):
            torch.mul(x, 1.0 - 0.2 * i, out=qkv); between()
            out.append(ops.attention_packed(qkv.view(B, L, H, 384), cos, sin)); between()
        return out
    with torch.no_grad():
        want = [t.clone() for t in steps(torch.cuda.synchronize)]
        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                got = steps()
        for _ in range(3):
            qkv.fill_(float("nan"))
            if captured:
                graph.replay()
            else:
                got = steps()
            assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("captured", [False, True])
def test_dependents_of_a_kernel_that_lets_them_start(captured):
    """The scan on short chunks lets the next kernel start as soon as all its own blocks run, so the dependent is there long before its
    operand is: GEMMs that read the scan's output as A, in either layout, as residual and as C, the rotary kernel with the attention behind
    it, and a GEMM behind a memset.  Buffers hold NaN before each pass, so a value read too early shows."""
    import ctypes
    from savanna_b200.ops import cuda_ops
    torch.manual_seed(23)
    lib, memset = cuda_ops.require(), ctypes.CDLL("libcudart.so.12").cudaMemsetAsync
    memset.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_size_t, ctypes.c_void_p]
    L, H, N, TC = 2048, 3, 512, 64
    D = 3 * H * 128
    feat = (torch.randn(L, 3 * D, device=DEV) * 0.7).to(BF)
    gamma, p = (torch.rand(D, 16, device=DEV) * 0.09 + 0.01).log(), -torch.ones(D, 16, device=DEV)
    R, bias = torch.randn(D, 16, device=DEV) / 4, torch.randn(D, device=DEV)
    modal, S = torch.empty(4 * D * 16, device=DEV), torch.empty(L // TC * D * 16, device=DEV)
    w, x, v = (torch.randn(*s, device=DEV).to(BF) for s in ((N, D), (L, N), (D, N)))
    cos, sin = (f(torch.rand(L, 128, device=DEV) * 6) for f in (torch.cos, torch.sin))
    scans = [torch.empty(L, D, device=DEV, dtype=BF) for _ in range(5)]
    outs = [torch.empty(*s, device=DEV, dtype=BF) for s in ((L, N), (D, N), (L, D), (L, D))]

    def scan(z):
        rc = lib.sb_li_fwd_tiled(feat.data_ptr(), gamma.data_ptr(), p.data_ptr(), R.data_ptr(), bias.data_ptr(), None, None, modal.data_ptr(),
                                 S.data_ptr(), z.data_ptr(), 1, L, D, 16, TC, torch.cuda.current_stream().cuda_stream)
        assert rc == 0

    def steps(between=lambda: None):
        scan(scans[0]); between()
        cuda_ops.gemm(scans[0], w, outs[0]); between()
        scan(scans[1]); between()
        cuda_ops.gemm(scans[1], x, outs[1], a_mn=True, b_mn=True); between()        # as a weight gradient
        scan(scans[2]); between()
        cuda_ops.gemm(x, v, outs[2], residual=scans[2]); between()
        scan(scans[3]); between()
        cuda_ops.gemm(x, v, scans[3], accumulate=True); between()
        scan(scans[4]); between()
        att = ops.attention_packed(scans[4].view(1, L, H, 384), cos, sin); between()
        assert memset(outs[3].data_ptr(), 0, outs[3].nbytes, torch.cuda.current_stream().cuda_stream) == 0; between()
        cuda_ops.gemm(x, v, outs[3], accumulate=True); between()
        return att

    with torch.no_grad():
        att = steps(torch.cuda.synchronize)
        want = [t.clone() for t in (*scans, *outs, att)]
        assert all(t.isfinite().all() for t in want)
        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                att = steps()
        for _ in range(5):
            for t in (*scans, *outs):
                t.fill_(float("nan"))
            if captured:
                graph.replay()
            else:
                att = steps()
            assert all(torch.equal(a, b) for a, b in zip((*scans, *outs, att), want))
    cuda_ops.check_status()


@pytest.mark.parametrize("B,L,H", [(1, 1, 1), (2, 333, 3), (1, 1024, 8)])
@pytest.mark.parametrize("captured", [False, True])
def test_attention_backward_behind_the_kernels_that_feed_it(B, L, H, captured):
    """The backward's main kernel, a dependent of the one that forms its row statistics, behind a kernel that writes the output's gradient."""
    torch.manual_seed(B * L + H)
    qkv = (torch.randn(B, L, H, 384, device=DEV) * 0.5).to(BF).requires_grad_()
    cos, sin = (f(torch.rand(L, 128, device=DEV) * 6) for f in (torch.cos, torch.sin))
    g0, go = torch.randn(B, L, H, 128, device=DEV).to(BF), torch.empty(B, L, H, 128, device=DEV, dtype=BF)

    def steps(between=lambda: None):
        grads = []
        for i in range(3):
            out = ops.attention_packed(qkv, cos, sin); between()
            torch.mul(g0, 1.0 - 0.3 * i, out=go); between()
            grads += torch.autograd.grad(out, qkv, go); between()
        return grads
    stream = torch.cuda.Stream()                          # captures want a stream of their own, warmed up
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        want = [t.clone() for t in steps(torch.cuda.synchronize)]
    torch.cuda.synchronize()
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            got = steps()
    for _ in range(3):
        go.fill_(float("nan"))
        if captured:
            graph.replay()
        else:
            got = steps()
        torch.cuda.synchronize()
        for a, b in zip(got, want):                       # dq adds up over key blocks in any order, in fp32: one rounding, either side
            _close(a, b, 2 ** -8, "dqkv")
