"""Kernels at the sizes where they can go wrong - edges of tiles, ragged remainders, the smallest and largest of a range -
against fp64 / fp32 PyTorch.  Tolerances: 2^-9 is half a unit in the last place of bf16 relative to the largest value
(fp16: 2^-12); a result that is rounded k times on its way may be off by k such steps."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"
ULP = {torch.bfloat16: 2.0 ** -9, torch.float16: 2.0 ** -12, torch.float32: 2.0 ** -24}


@pytest.fixture(scope="module")
def K():
    from mindspore_b200 import _native
    from mindspore_b200.ops import kernels
    assert _native.cuda() is not None, "native CUDA library is not loaded"
    torch.manual_seed(3)
    return kernels


def _near(got, exp, steps, dtype, rel=True):
    """Largest difference within ``steps`` roundings of the largest value."""
    got, exp = got.double(), exp.double()
    bound = steps * ULP[dtype] * (exp.abs().max().item() if rel else 1.0)
    assert torch.isfinite(got).all()
    err = (got - exp).abs().max().item()
    assert err <= bound, "error %g, bound %g" % (err, bound)


def _status_ok():
    from mindspore_b200 import _native
    torch.cuda.synchronize()
    assert _native.device_status() == 0


# ------------------------------------------------------------------------------------------------ attention
@pytest.mark.parametrize("B,S,H,Hk,causal", [(1, 128, 2, 1, True), (2, 384, 4, 2, True), (1, 384, 4, 1, False),
                                              (1, 640, 40, 40, True), (1, 2176, 12, 3, True), (3, 5, 2, 2, True),
                                              (2, 100, 2, 1, False), (1, 129, 4, 2, True), (2, 1000, 4, 4, False)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_flash_attention_grouped_heads_and_odd_tiles(K, B, S, H, Hk, causal, dtype):
    """One tile, an odd number of query tiles (the second of a pair lies beyond the sequence), more items than SMs,
    grouped k / v heads, sequences that end inside a tile: forward, log-sum-exp and all gradients."""
    from mindspore_b200.ops import flash_attn_kernel as FK
    D = 128
    q = torch.randn(B, S, H, D, device=DEV).to(dtype)
    k, v = (torch.randn(B, S, Hk, D, device=DEV).to(dtype) for _ in range(2))
    do = torch.randn(B, S, H, D, device=DEV).to(dtype)
    sc = 1 / math.sqrt(D)
    o, lse, q2, k2, v2 = FK.fwd(q, k, v, causal, sc)
    dq, dk, dv = FK.bwd(do, q2, k2, v2, o, lse, causal, sc)
    qf, kf, vf = (t.double().requires_grad_(True) for t in (q, k, v))
    s = torch.einsum("bqhd,bkhd->bhqk", qf, kf.repeat_interleave(H // Hk, 2)) * sc
    if causal:
        s = s.masked_fill(torch.ones(S, S, device=DEV, dtype=torch.bool).triu(1), -math.inf)
    ref = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), vf.repeat_interleave(H // Hk, 2))
    ref.backward(do.double())
    _near(o, ref, 4, dtype)                                  # P and O rounded; P's error averages over the keys
    _near(lse, torch.logsumexp(s, -1), 64, torch.float32)    # exp2 / log2 of the fast unit: 2 ulp each
    for got, t in ((dq, qf), (dk, kf), (dv, vf)):
        _near(got, t.grad, 6, dtype)                         # P, dS, O and the result rounded
    _status_ok()


@pytest.mark.parametrize("S,H,Hk", [(256, 4, 2), (200, 4, 4), (77, 4, 1)])
def test_rotary_attention_keeps_its_input(K, S, H, Hk):
    """RotaryFlashAttention with grouped heads or a ragged sequence: gradient against fp64, the packed projection left as it
    was."""
    from mindspore_b200.ops.llm_ops import RotaryFlashAttention
    from mindspore_b200.ops import fused
    D = 128
    qkv = torch.randn(2 * S, (H + 2 * Hk) * D, device=DEV).bfloat16()
    cos, sin = fused.rope_tables(S, D, device=DEV)
    do = torch.randn(2 * S, H * D, device=DEV).bfloat16()
    x = qkv.clone().requires_grad_(True)
    y = RotaryFlashAttention(H, Hk, D)(x, cos, sin)
    (g,) = torch.autograd.grad(y, x, do)
    assert torch.equal(x.detach(), qkv)
    r = qkv.double().requires_grad_(True)
    q, k, v = (t.reshape(2, S, -1, D) for t in r.split([H * D, Hk * D, Hk * D], -1))
    c, s = cos.double()[None, :, None], sin.double()[None, :, None]
    rot = lambda t: torch.cat([t[..., :64] * c - t[..., 64:] * s, t[..., 64:] * c + t[..., :64] * s], -1)  # noqa: E731
    p = torch.einsum("bqhd,bkhd->bhqk", rot(q), rot(k).repeat_interleave(H // Hk, 2)) / math.sqrt(D)
    p = p.masked_fill(torch.ones(S, S, device=DEV, dtype=torch.bool).triu(1), -math.inf)
    ref = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(p, -1), v.repeat_interleave(H // Hk, 2)).reshape(2 * S, H * D)
    ref.backward(do.double())
    _near(y, ref, 6, torch.bfloat16)
    _near(g, r.grad, 10, torch.bfloat16)
    _status_ok()


# ------------------------------------------------------------------------------------------------ cross entropy
@pytest.mark.parametrize("rows,V", [(1, 1), (3, 7), (5, 4099), (64, 32000), (9, 50257)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_cross_entropy_ragged_vocabulary(K, rows, V, dtype):
    """Vocabularies that leave rows misaligned, ignored rows, -inf logits, an in-place gradient."""
    from mindspore_b200.ops import fused
    x = (2 * torch.randn(rows, V, device=DEV)).to(dtype)
    if V > 100:
        x[:, 3::5] = -math.inf
    lab = torch.randint(0, V, (rows, 2), device=DEV, dtype=torch.int32)[:, 0]
    lab[lab % 5 == 3] -= 1
    lab[1::4] = -100
    a = x.clone().requires_grad_(True)
    loss = fused.softmax_cross_entropy(a, lab)
    (3 * loss).backward()
    r = x.double().requires_grad_(True)
    ref = torch.nn.functional.cross_entropy(r, lab.long())
    (3 * ref).backward()
    assert abs(float(loss) - float(ref)) <= 1e-5 * max(1.0, abs(float(ref)))
    _near(a.grad, r.grad, 2 if dtype == torch.bfloat16 else 256, dtype)      # fp32: exp of the fast unit
    st = K.ce_stats(a.detach(), lab.contiguous())
    buf = x.clone()
    K.ce_loss_grad(buf, lab.contiguous(), st, torch.full((1,), 0.5, device=DEV), dlogits=buf)
    valid = int((lab != -100).sum())
    _near(buf, r.grad * (0.5 * valid / 3), 2 if dtype == torch.bfloat16 else 256, dtype)


def test_cross_entropy_without_a_valid_row(K):
    from mindspore_b200.ops import fused
    x = torch.randn(4, 40, device=DEV).bfloat16().requires_grad_(True)
    loss = fused.softmax_cross_entropy(x, torch.full((4,), -100, device=DEV, dtype=torch.int32))
    loss.backward()
    assert float(loss) == 0 and not x.grad.any()


# ------------------------------------------------------------------------------------------------ norms
@pytest.mark.parametrize("rows,H", [(1, 8), (3, 248), (700, 256), (5, 1032), (1031, 2560), (2, 5064), (601, 4096),
                                    (7, 8200), (3, 16384)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_norms_over_the_range_of_widths(K, rows, H, dtype):
    """A warp per row, groups of a block, whole blocks of every size; fewer rows than SMs and several per CTA."""
    x, r, dy, ds = (torch.randn(rows, H, device=DEV).to(dtype) for _ in range(4))
    w, b = ((1 + 0.1 * torch.randn(H, device=DEV)).to(dtype) for _ in range(2))
    y, rstd, s = K.rmsnorm_fwd(x, w, 1e-5, residual=r)
    dx, dw = K.rmsnorm_bwd(dy, s, w, rstd, dresidual=ds)
    acc = torch.ones(H, device=DEV)
    K.rmsnorm_bwd(dy, s, w, rstd, dw_out=acc, accumulate=True)
    sd, wd = s.double().requires_grad_(True), w.double().requires_grad_(True)
    ref = sd * torch.rsqrt(sd.pow(2).mean(-1, keepdim=True) + 1e-5) * wd
    ref.backward(dy.double())
    assert torch.equal(s, (x.float() + r.float()).to(dtype))
    _near(y, ref, 2, dtype)
    _near(dx, sd.grad + ds.double(), 2, dtype)
    _near(dw, wd.grad, 2, dtype)
    _near(acc - 1, wd.grad, 2, dtype)
    y, mean, rstd = K.layernorm_fwd(x, w, b, 1e-5)
    dx, dw, db = K.layernorm_bwd(dy, x, w, mean, rstd)
    xd, wd, bd = (t.double().requires_grad_(True) for t in (x, w, b))
    ref = torch.nn.functional.layer_norm(xd, (H,), wd, bd, 1e-5)
    ref.backward(dy.double())
    for got, exp in ((y, ref), (dx, xd.grad), (dw, wd.grad), (db, bd.grad)):
        _near(got, exp, 2, dtype)


# ------------------------------------------------------------------------------------------------ streaming kernels
@pytest.mark.parametrize("rows,F", [(1, 8), (3, 24), (77, 11008), (1000, 1408)])
def test_swiglu_sizes(K, rows, F):
    gu, d = torch.randn(rows, 2 * F, device=DEV).bfloat16(), torch.randn(rows, F, device=DEV).bfloat16()
    x = gu.double().requires_grad_(True)
    ref = torch.nn.functional.silu(x[:, :F]) * x[:, F:]
    ref.backward(d.double())
    _near(K.swiglu_fwd(gu), ref, 2, torch.bfloat16)
    _near(K.swiglu_bwd(gu, d), x.grad, 2, torch.bfloat16)


@pytest.mark.parametrize("tokens,heads,D,seq", [(5, 1, 16, 5), (6, 3, 80, 3), (64, 9, 128, 32), (8, 40, 128, 8)])
def test_rope_in_and_out_of_place(K, tokens, heads, D, seq):
    """Widths that do not divide the block, odd numbers of heads, a pitch wider than the row, misaligned tables."""
    wide = torch.randn(tokens, heads * D + 64, device=DEV).bfloat16()
    x = wide[:, :heads * D]
    ang = torch.randn(seq, D // 2, device=DEV)
    store = torch.empty(2 * ang.numel() + 1, device=DEV)
    cos, sin = (store[1 + i * ang.numel():1 + (i + 1) * ang.numel()].view_as(ang) for i in range(2))
    cos.copy_(ang.cos())
    sin.copy_(ang.sin())
    p = torch.arange(tokens, device=DEV) % seq
    c, s = cos.double()[p][:, None], sin.double()[p][:, None]
    xd = x.double().view(tokens, heads, D)
    a, b = xd[..., :D // 2], xd[..., D // 2:]
    ref = torch.cat([a * c - b * s, b * c + a * s], -1).reshape(tokens, heads * D)
    before = wide.clone()
    _near(K.rope(x, cos, sin, heads, D, seq), ref, 2, torch.bfloat16)
    assert torch.equal(wide, before)
    K.rope_(x, cos, sin, heads, D, seq)
    _near(x, ref, 2, torch.bfloat16)
    assert torch.equal(wide[:, heads * D:], before[:, heads * D:])


@pytest.mark.parametrize("n,off", [(1, 0), (3, 1), (17, 3), (100003, 1), (1 << 22, 0)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_sum_of_squares_of_slices(K, n, off, dtype):
    x = torch.randn(n + off, device=DEV).to(dtype)[off:]
    out, bad = torch.zeros(1, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    K.sumsq_finite(x, out, bad)
    assert int(bad) == 0
    _near(out, x.double().pow(2).sum().reshape(1), 1024, torch.float32)
    for value in (math.inf, -math.inf, math.nan):
        y = x.clone()
        y[n // 2] = value
        bad.zero_()
        K.sumsq_finite(y, out, bad)
        assert int(bad) == 1
    big = torch.full((n,), 3e38, device=DEV).to(dtype)            # finite values whose squares are not
    bad.zero_()
    K.sumsq_finite(big, out, bad)
    assert int(bad) == 0


def test_fill_scalars(K):
    h = torch.zeros(8, device=DEV)
    K.fill_scalars(h[2:5], [0.1, 1e-8, 3])
    assert torch.equal(h.cpu(), torch.tensor([0, 0, 0.1, 1e-8, 3, 0, 0, 0]))


# ------------------------------------------------------------------------------------------------ GEMM
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("M,N,Kd,batch", [(8, 8, 8, 1), (24, 4096, 4096, 1), (136, 72, 328, 1), (128, 64, 520, 3),
                                          (1, 200, 2048, 1), (300, 512, 1408, 2)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gemm_with_few_tiles(K, a_mn, b_mn, M, N, Kd, batch, dtype):
    """Split over clusters of 1 to 8 CTAs, ragged M / N / K, bias, fp32 accumulation into an existing output."""
    if a_mn and M % 8:
        pytest.skip("a stored [K, M] needs a row pitch of whole 16 bytes")
    mk = lambda r, c, t: (torch.randn(*((batch,) if batch > 1 else ()), *((c, r) if t else (r, c)), device=DEV) /  # noqa: E731
                          math.sqrt(Kd)).to(dtype)
    a, b = mk(M, Kd, a_mn), mk(N, Kd, b_mn)
    bias = torch.randn(N, device=DEV).to(dtype)
    ad = a.double().transpose(-1, -2) if a_mn else a.double()
    bd = b.double().transpose(-1, -2) if b_mn else b.double()
    ref = ad @ bd.transpose(-1, -2)
    _near(K.gemm(a, b, a_mn=a_mn, b_mn=b_mn, bias=bias, alpha=2.0), 2 * ref + bias.double(), 2, dtype)
    out = torch.ones(ref.shape, device=DEV)
    K.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=out, accumulate=True)
    _near(out, ref + 1, 256, torch.float32)                     # fp32 sums of up to 4096 products in another order
    _status_ok()


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("M,N,Kd", [(1032, 776, 200), (1280, 2560, 72)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gemm_cta_pair_batched(K, a_mn, b_mn, M, N, Kd, dtype):
    """Batched problems on CTA pairs, both element types, ragged tiles, accumulation."""
    batch = 8
    mk = lambda r, c, t: (torch.randn(batch, *((c, r) if t else (r, c)), device=DEV) / math.sqrt(Kd)).to(dtype)  # noqa: E731
    a, b = mk(M, Kd, a_mn), mk(N, Kd, b_mn)
    out = torch.empty(batch, M, N, device=DEV, dtype=dtype)
    assert K._pair_gemm_ok(M, N, Kd, batch, out, out[0], False, 0)
    ad = a.double().transpose(-1, -2) if a_mn else a.double()
    bd = b.double().transpose(-1, -2) if b_mn else b.double()
    ref = ad @ bd.transpose(-1, -2)
    _near(K.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=out), ref, 2, dtype)
    acc = torch.ones(ref.shape, device=DEV)
    K.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=acc, accumulate=True)
    _near(acc, ref + 1, 256, torch.float32)
    _status_ok()


# ------------------------------------------------------------------------------------------------ convolution
@pytest.mark.parametrize("N,C,H,W,Cout,k,stride", [(1, 64, 7, 7, 64, 3, 1), (3, 64, 13, 9, 256, 1, 1),
                                                  (2, 128, 15, 15, 128, 3, 2), (5, 64, 3, 5, 320, 1, 1),
                                                  (2, 320, 9, 6, 72, 1, 1), (1, 64, 9, 21, 200, 3, 1)])
def test_convolution_edges(K, N, C, H, W, Cout, k, stride):
    """Pixel tiles that overhang the image on every side, one and several column blocks: output, the statistics that the
    epilogue gathers, and the weight gradient."""
    from mindspore_b200.ops import conv_kernel as CK
    x = torch.randn(N, C, H, W, device=DEV).bfloat16().to(memory_format=torch.channels_last)
    w = (torch.randn(Cout, C, k, k, device=DEV) / math.sqrt(C * k * k)).bfloat16()
    y, stats = CK._ConvFn.apply(x, w, stride, k // 2, k // 2, True)
    ref = torch.nn.functional.conv2d(x.double(), w.double(), None, stride, k // 2)
    _near(y, ref, 2, torch.bfloat16)
    yd = y.double()
    _near(stats[:Cout], yd.sum((0, 2, 3)), 4096, torch.float32)
    _near(stats[Cout:], yd.pow(2).sum((0, 2, 3)), 4096, torch.float32)
    dy = torch.randn_like(ref).bfloat16().to(memory_format=torch.channels_last)
    dw = CK.conv_wgrad_raw(x, dy, k, k, stride, k // 2, k // 2).permute(0, 3, 1, 2)
    refw = torch.nn.grad.conv2d_weight(x.double(), w.shape, dy.double(), stride, k // 2)
    _near(dw, refw, 1024, torch.float32)
    _status_ok()


@pytest.mark.parametrize("N,C,H,W,Cout,k,stride", [(1, 64, 7, 7, 64, 3, 1), (2, 320, 5, 9, 64, 3, 1), (38, 192, 28, 28, 64, 1, 1),
                                                  (3, 128, 8, 6, 320, 1, 2), (2, 128, 9, 9, 192, 3, 2), (2, 64, 9, 9, 72, 3, 1)])
def test_convolution_data_gradient(K, N, C, H, W, Cout, k, stride):
    """The data gradient by the weights of the forward pass in their own order (72 channels: a padded copy), one and several
    column blocks, strides included."""
    from mindspore_b200.ops import conv_kernel as CK
    x = torch.randn(N, C, H, W, device=DEV).bfloat16().to(memory_format=torch.channels_last).requires_grad_()
    w = (torch.randn(Cout, C, k, k, device=DEV) / math.sqrt(C * k * k)).bfloat16()
    y, _ = CK._ConvFn.apply(x, w, stride, k // 2, k // 2, False)
    dy = torch.randn_like(y)
    y.backward(dy)
    ref = torch.nn.grad.conv2d_input(x.shape, w.double(), dy.double(), stride, k // 2)
    _near(x.grad, ref, 2, torch.bfloat16)
    _status_ok()


def test_batch_norm_affine_gradients(K):
    """Gradients of 16-bit gamma and beta, which the backward kernel writes itself."""
    from mindspore_b200.ops import conv_kernel as CK
    N, C, H, W = 3, 72, 5, 7
    x = torch.randn(N, C, H, W, device=DEV).bfloat16().to(memory_format=torch.channels_last)
    xd = x.double()
    stats = torch.cat([xd.sum((0, 2, 3)), xd.pow(2).sum((0, 2, 3))]).float()
    gamma, beta = ((torch.randn(C, device=DEV) * 0.1 + o).bfloat16().requires_grad_() for o in (1, 0))
    y = CK._BnActFn.apply(x, stats, gamma, beta, None, False, 1e-5, (torch.zeros(C, device=DEV), torch.ones(C, device=DEV), 0.9))
    dy = torch.randn_like(y)
    y.backward(dy)
    xhat = (xd - xd.mean((0, 2, 3), keepdim=True)) * torch.rsqrt(xd.var((0, 2, 3), unbiased=False, keepdim=True) + 1e-5)
    _near(gamma.grad, (dy.double() * xhat).sum((0, 2, 3)), 2, torch.bfloat16)
    _near(beta.grad, dy.double().sum((0, 2, 3)), 2, torch.bfloat16)
    _status_ok()
