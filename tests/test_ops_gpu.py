"""Each CUDA kernel against a plain PyTorch fp32 reference of the same op."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _close(a, b, rtol, atol, what=""):
    a, b = a.float(), b.float()
    err = (a - b).abs()
    tol = atol + rtol * b.abs()
    bad = (err > tol).float().mean().item()
    assert bad < 1e-3, f"{what}: {bad:.4%} elements out of tolerance, max err {err.max().item():.4g}"


@pytest.mark.parametrize("T,H", [(64, 256), (1000, 4096), (33, 5120), (17, 8192)])
@pytest.mark.parametrize("with_res", [False, True])
def test_rmsnorm_fwd_bwd(T, H, with_res):
    from xorl_b200.ops.norm import rmsnorm
    torch.manual_seed(0)
    x = torch.randn(T, H, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    r = torch.randn(T, H, device=DEV, dtype=torch.bfloat16, requires_grad=True) if with_res else None
    w = (1 + 0.1 * torch.randn(H, device=DEV)).to(torch.bfloat16).requires_grad_()
    gy = torch.randn(T, H, device=DEV, dtype=torch.bfloat16)
    gh = torch.randn(T, H, device=DEV, dtype=torch.bfloat16)
    if with_res:
        y, h = rmsnorm(x, w, 1e-6, residual=r)
        (y.float() * gy.float()).sum().add((h.float() * gh.float()).sum()).backward()
    else:
        y = rmsnorm(x, w, 1e-6)
        (y.float() * gy.float()).sum().backward()
    # fp32 reference
    xr = x.detach().float().requires_grad_()
    rr = r.detach().float().requires_grad_() if with_res else None
    wr = w.detach().float().requires_grad_()
    hr = xr + rr if with_res else xr
    if with_res:
        hr = hr + (hr.to(torch.bfloat16).float() - hr).detach()  # residual stream is stored in bf16
    yr = hr * torch.rsqrt(hr.pow(2).mean(-1, keepdim=True) + 1e-6) * wr
    lossr = (yr * gy.float()).sum()
    if with_res:
        lossr = lossr + (hr * gh.float()).sum()
    lossr.backward()
    _close(y, yr, 2e-2, 2e-2, "y")
    _close(x.grad, xr.grad, 3e-2, 3e-2, "dx")
    _close(w.grad, wr.grad, 3e-2, 0.05 * wr.grad.abs().max().item(), "dw")
    if with_res:
        _close(r.grad, rr.grad, 3e-2, 3e-2, "dres")


@pytest.mark.parametrize("T,I", [(77, 768), (512, 12288)])
def test_swiglu(T, I):
    from xorl_b200.ops.activation import swiglu
    torch.manual_seed(0)
    gu = torch.randn(T, 2 * I, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    go = torch.randn(T, I, device=DEV, dtype=torch.bfloat16)
    out = swiglu(gu)
    out.backward(go)
    gr = gu.detach().float().requires_grad_()
    ref = torch.nn.functional.silu(gr[:, :I]) * gr[:, I:]
    ref.backward(go.float())
    _close(out, ref, 2e-2, 2e-2, "out")
    _close(gu.grad, gr.grad, 2e-2, 2e-2, "dgu")


@pytest.mark.parametrize("rows,V", [(64, 1024), (130, 151936), (16, 32003)])
def test_cross_entropy_chunk(rows, V):
    from xorl_b200.ops.loss import ce_chunk_
    torch.manual_seed(0)
    ldv = (V + 7) // 8 * 8
    buf = torch.randn(rows, ldv, device=DEV, dtype=torch.bfloat16) * 3
    logits = buf[:, :V]
    labels = torch.randint(0, V, (rows,), device=DEV)
    labels[::7] = -100
    lr = logits.detach().float().requires_grad_()
    ref = torch.nn.functional.cross_entropy(lr, labels, ignore_index=-100, reduction="none")
    (ref.sum() * 0.5).backward()
    loss, lse = ce_chunk_(logits, labels, 0.5, True)
    _close(loss, ref, 1e-3, 1e-3, "loss")
    _close(logits, lr.grad, 2e-2, 1e-4, "dlogits")


def test_fused_linear_ce():
    from xorl_b200.ops.loss import fused_linear_cross_entropy
    torch.manual_seed(0)
    T, H, V = 300, 256, 5000
    h = (torch.randn(T, H, device=DEV) * 0.5).to(torch.bfloat16).requires_grad_()
    w = (torch.randn(V, H, device=DEV) * 0.05).to(torch.bfloat16).requires_grad_()
    labels = torch.randint(0, V, (T,), device=DEV)
    labels[:5] = -100
    loss = fused_linear_cross_entropy(h, w, labels, grad_scale=1.0 / T, chunk_tokens=128)
    loss.backward()
    hr, wr = h.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    ref = torch.nn.functional.cross_entropy(hr @ wr.t(), labels, ignore_index=-100, reduction="sum") / T
    ref.backward()
    assert abs(loss.item() - ref.item()) < 2e-2 * abs(ref.item())
    _close(h.grad, hr.grad, 5e-2, 0.03 * hr.grad.abs().max().item(), "dh")
    _close(w.grad, wr.grad, 5e-2, 0.03 * wr.grad.abs().max().item(), "dw")


@pytest.mark.parametrize("kept_chunks", [0, 1, 2, 4, 9])
@pytest.mark.parametrize("buffer", [None, "fresh", "adds"])
@pytest.mark.parametrize("token_loss", [False, True])
def test_lm_head_gradients_over_groups_of_chunks(kept_chunks, buffer, token_loss):
    """Five chunks, the last one ragged, in groups of one, two (2 + 2 + 1), four (4 + 1) and all: hidden and weight
    gradients, the latter also in an engine's fp32 buffer, and the memory that the logits take.  bf16 logits and
    gradients of logits: each within 2^-9, 4e-3 of the norm together with the fp32 sums."""
    from xorl_b200.ops.loss import fused_linear_cross_entropy, fused_linear_token_loss
    torch.manual_seed(0)
    T, H, V, chunk = 1100, 128, 1000, 256
    h = (torch.randn(T, H, device=DEV) * 0.5).bfloat16().requires_grad_()
    w = (torch.randn(V, H, device=DEV) * 0.05).bfloat16().requires_grad_()
    labels = torch.randint(0, V, (T,), device=DEV)
    labels[::9] = -100
    start = torch.randn(V, H, device=DEV)
    if buffer:
        w._xb_grad_buf, w._xb_grad_fresh = start.clone(), buffer == "fresh"
    kept = kept_chunks * chunk * V * 2
    if token_loss:
        loss, _, _ = fused_linear_token_loss(h, w, labels, lambda lp, mask: (-(lp * mask).sum(), {}), 1.0,
                                             chunk_tokens=chunk, kept_logits_bytes=kept)
    else:
        loss = fused_linear_cross_entropy(h, w, labels, chunk_tokens=chunk, kept_logits_bytes=kept)
    loss.backward()
    hr, wr = h.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    ref = torch.nn.functional.cross_entropy(hr @ wr.t(), labels, ignore_index=-100, reduction="sum")
    ref.backward()
    dw = w._xb_grad_buf - (start if buffer == "adds" else 0) if buffer else w.grad.float()
    assert abs(loss.item() - ref.item()) < 4e-3 * ref.item()
    for name, g, r in (("dh", h.grad.float(), hr.grad), ("dw", dw, wr.grad)):
        assert (g - r).norm() < 4e-3 * r.norm(), (name, float((g - r).norm() / r.norm()))


def test_lm_head_logits_stay_within_the_chunk_that_was_asked_for():
    from xorl_b200.ops.loss import fused_linear_cross_entropy
    T, H, V = 4096, 64, 16384
    h = torch.randn(T, H, device=DEV).bfloat16().requires_grad_()
    w = (torch.randn(V, H, device=DEV) * 0.05).bfloat16().requires_grad_()
    labels = torch.randint(0, V, (T,), device=DEV)

    def peak(**kw):
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        base = torch.cuda.memory_allocated()
        fused_linear_cross_entropy(h, w, labels, **kw).backward()
        h.grad = w.grad = None
        return torch.cuda.max_memory_allocated() - base

    slack = 4 * (V * H * 4 + T * H * 4)                       # gradients of weight and hidden states, in fp32
    assert peak(chunk_tokens=256) < 256 * V * 2 + slack
    assert peak(chunk_tokens=1024, kept_logits_bytes=0) < 1024 * V * 2 + slack
    assert peak() > T * V * 2                                 # nothing asked for: all of it at once


def test_embedding():
    from xorl_b200.ops.embedding import embedding
    torch.manual_seed(0)
    V, H, T = 1000, 256, 513
    table = torch.randn(V, H, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    ids = torch.randint(0, V, (T,), device=DEV)
    go = torch.randn(T, H, device=DEV, dtype=torch.bfloat16)
    out = embedding(ids, table)
    out.backward(go)
    tr = table.detach().float().requires_grad_()
    ref = torch.nn.functional.embedding(ids, tr)
    ref.backward(go.float())
    assert torch.equal(out.float(), ref)
    _close(table.grad, tr.grad, 2e-2, 2e-2, "dtable")


def test_adamw_and_norm():
    from xorl_b200.ops import optim
    torch.manual_seed(0)
    n = 1_000_003
    p = torch.randn(n, device=DEV)
    g = torch.randn(n, device=DEV) * 0.1
    m = torch.zeros(n, device=DEV)
    v = torch.zeros(n, device=DEV)
    pr = p.clone().requires_grad_()
    opt = torch.optim.AdamW([pr], lr=1e-3, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.01)
    bf = torch.empty(n, device=DEV, dtype=torch.bfloat16)
    for step in range(1, 4):
        pr.grad = g.clone()
        opt.step()
        optim.adamw_step_(p, m, v, g, bf, lr=1e-3, beta1=0.9, beta2=0.95, eps=1e-8,
                          weight_decay=0.01, step=step)
    assert torch.allclose(p, pr.detach(), rtol=1e-5, atol=1e-6)
    assert torch.equal(bf, p.to(torch.bfloat16))
    tot = torch.zeros(1, device=DEV)
    optim.sumsq_(g, tot, False)
    assert abs(tot.item() - g.double().pow(2).sum().item()) < 1e-3 * tot.item()
    norm = torch.zeros(1, device=DEV)
    coef = torch.zeros(1, device=DEV)
    optim.clip_coef_(tot, 1.0, norm, coef)
    assert abs(norm.item() - math.sqrt(tot.item())) < 1e-3
    assert abs(coef.item() - min(1.0, 1.0 / (norm.item() + 1e-6))) < 1e-5


def _make_cu(lens):
    cu = [0]
    for l in lens:
        cu.append(cu[-1] + l)
    return torch.tensor(cu, device=DEV, dtype=torch.int32)


@pytest.fixture(params=["split", "fused"])
def bwd_mode(request):
    from xorl_b200.ops import _lib, attention
    prev = attention.set_backward_mode(request.param)
    yield request.param
    attention.set_backward_mode(prev)
    assert all(v == 0 for v in _lib.read_status()[:4])


@pytest.mark.parametrize("lens,Hq,Hkv,causal", [
    ([128], 2, 1, True), ([256], 4, 2, True), ([200, 56, 384], 4, 1, True), ([1000], 8, 2, True),
    ([300, 100], 2, 2, False), ([4096], 8, 2, True), ([1, 63, 65, 129, 700], 4, 2, True)])
def test_flash_attention_fwd_bwd(lens, Hq, Hkv, causal, bwd_mode):
    from xorl_b200.ops.attention import attention_reference, flash_attn_varlen
    torch.manual_seed(0)
    D = 128
    T = sum(lens)
    cu = _make_cu(lens)
    q = torch.randn(T, Hq, D, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    k = torch.randn(T, Hkv, D, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    v = torch.randn(T, Hkv, D, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    go = torch.randn(T, Hq, D, device=DEV, dtype=torch.bfloat16)
    out = flash_attn_varlen(q, k, v, cu, causal=causal)
    out.backward(go)
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    ref = attention_reference(qr, kr, vr, cu, causal=causal)
    ref.backward(go.float())
    _close(out, ref, 2e-2, 2e-2, "out")
    _close(v.grad, vr.grad, 3e-2, 0.02 * vr.grad.abs().max().item(), "dv")
    _close(k.grad, kr.grad, 3e-2, 0.02 * kr.grad.abs().max().item(), "dk")
    _close(q.grad, qr.grad, 3e-2, 0.02 * qr.grad.abs().max().item(), "dq")


@pytest.mark.parametrize("lens,Hq,Hkv,D,window,sinks", [
    ([333, 691], 4, 2, 128, 128, False),      # window = one tile; documents that end inside a tile
    ([1024], 2, 2, 128, 200, False),          # window that straddles tiles
    ([700, 100], 4, 1, 128, 8, False),        # window far below the tile size
    ([515], 2, 1, 128, 4096, False),          # window longer than the document: plain causal
    ([333, 691], 4, 2, 128, 0, True),         # sink logits only
    ([300, 212, 512], 8, 2, 64, 128, True),   # gpt-oss layer: 64-wide heads, window and sinks
])
def test_flash_attention_window_sinks_head_dim(lens, Hq, Hkv, D, window, sinks):
    from xorl_b200.ops import attention as A
    torch.manual_seed(0)
    T = sum(lens)
    cu = _make_cu(lens)
    q = torch.randn(T, Hq, D, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    k = torch.randn(T, Hkv, D, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    v = torch.randn(T, Hkv, D, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    sk = (torch.randn(Hq, device=DEV) * 2).to(torch.bfloat16).requires_grad_() if sinks else None
    go = torch.randn(T, Hq, D, device=DEV, dtype=torch.bfloat16)
    before = A.launch_count()
    out = A.flash_attn_varlen(q, k, v, cu, causal=True, window=window or None, sinks=sk)
    out.backward(go)
    assert A.launch_count() - before == 4, "the tcgen05 kernels must serve windows, sinks and 64-wide heads"
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    skr = sk.detach().float().requires_grad_() if sinks else None
    ref = A.attention_reference(qr, kr, vr, cu, causal=True, window=window or None, sinks=skr)
    ref.backward(go.float())
    _close(out, ref, 2e-2, 2e-2, "out")
    _close(v.grad, vr.grad, 3e-2, 0.02 * vr.grad.abs().max().item(), "dv")
    _close(k.grad, kr.grad, 3e-2, 0.02 * kr.grad.abs().max().item(), "dk")
    _close(q.grad, qr.grad, 3e-2, 0.02 * qr.grad.abs().max().item(), "dq")
    if sinks:
        _close(sk.grad, skr.grad, 3e-2, 0.03 * skr.grad.abs().max().item(), "dsinks")


@pytest.mark.parametrize("do_norm", [True, False])
def test_qk_norm_rope_attention(do_norm):
    from xorl_b200.ops.attention import (qk_norm_rope_attention,
                                         qk_norm_rope_attention_reference)
    torch.manual_seed(0)
    Hq, Hkv, D = 4, 2, 128
    lens = [300, 212]
    T = sum(lens)
    cu = _make_cu(lens)
    qkv = torch.randn(T, (Hq + 2 * Hkv) * D, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    wq = (1 + 0.1 * torch.randn(D, device=DEV)).to(torch.bfloat16).requires_grad_() if do_norm else None
    wk = (1 + 0.1 * torch.randn(D, device=DEV)).to(torch.bfloat16).requires_grad_() if do_norm else None
    pos = torch.cat([torch.arange(l, device=DEV) for l in lens]).float()
    inv = 1.0 / (1e6 ** (torch.arange(0, D, 2, device=DEV).float() / D))
    ang = pos[:, None] * inv[None, :]
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    go = torch.randn(T, Hq * D, device=DEV, dtype=torch.bfloat16)
    out = qk_norm_rope_attention(qkv, wq, wk, cos, sin, cu, Hq, Hkv, D)
    out.backward(go)
    qkvr = qkv.detach().float().requires_grad_()
    wqr = wq.detach().float().requires_grad_() if do_norm else None
    wkr = wk.detach().float().requires_grad_() if do_norm else None
    ref = qk_norm_rope_attention_reference(qkvr, wqr, wkr, cos, sin, cu, Hq, Hkv, D, 1e-6, True,
                                           1.0 / math.sqrt(D))
    ref.backward(go.float())
    _close(out, ref, 3e-2, 3e-2, "out")
    _close(qkv.grad, qkvr.grad, 5e-2, 0.03 * qkvr.grad.abs().max().item(), "dqkv")
    if do_norm:
        _close(wq.grad, wqr.grad, 5e-2, 0.05 * wqr.grad.abs().max().item(), "dwq")
        _close(wk.grad, wkr.grad, 5e-2, 0.05 * wkr.grad.abs().max().item(), "dwk")


@pytest.mark.parametrize("lens,Hq,Hkv,causal,window", [
    ([1], 1, 1, True, 0), ([127, 129, 256, 257], 8, 1, True, 0), ([2000, 40], 16, 2, True, 0), ([8192], 8, 8, True, 0),
    ([513], 12, 4, False, 0), ([900], 8, 1, True, 300), ([128, 640], 4, 1, False, 130), ([3000, 3000, 2192], 32, 8, True, 0)])
def test_attention_128_against_the_single_backward_kernel(lens, Hq, Hkv, causal, window):
    """Two query tiles per forward CTA, 128-row key tiles and heads dealt over clusters of 1, 2 and 4 in the
    backward, on long and ragged documents: against float32 sums of the same bf16 values (short calls) and
    against the kernel with 64-row tiles and P in shared memory (long ones).  Both round P and dS to bf16, so
    results agree to about two of its roundings, 2^-8 of their norm."""
    from xorl_b200.ops import _lib, attention as A
    torch.manual_seed(1)
    T, D = sum(lens), 128
    cu = _make_cu(lens)
    q, k, v = (torch.randn(T, h, D, device=DEV, dtype=torch.bfloat16) for h in (Hq, Hkv, Hkv))
    go = torch.randn(T, Hq, D, device=DEV, dtype=torch.bfloat16)
    out, lse = A._attn_fwd(q, k, v, cu, causal, D ** -0.5, window)
    dv = torch.empty_like(v)
    dq, dk = A._attn_bwd(q, k, v, out, go, lse, cu, causal, D ** -0.5, dv, window)
    again = A._attn_bwd(q, k, v, out, go, lse, cu, causal, D ** -0.5, torch.empty_like(v), window)
    assert torch.equal(dq, again[0]) and torch.equal(dk, again[1])      # sums in a fixed order
    got = [out, dq, dk, dv]
    if T <= 2048 or window:
        ins = [t.float().requires_grad_() for t in (q, k, v)]
        ref = A.attention_reference(*ins, cu, causal=causal, window=window or None)
        ref.backward(go.float())
        refs = [ref.detach()] + [t.grad for t in ins]
    else:
        prev = A.set_backward_mode("fused")
        try:
            dv2 = torch.empty_like(v)
            dq2, dk2 = A._attn_bwd(q, k, v, out, go, lse, cu, causal, D ** -0.5, dv2, window)
        finally:
            A.set_backward_mode(prev)
        refs = [A.attention_reference(q.float(), k.float(), v.float(), cu, causal=causal), dq2, dk2, dv2]
    for name, g, r in zip(("out", "dq", "dk", "dv"), got, refs):
        err = (g.float() - r.float()).norm().item() / max(r.float().norm().item(), 1e-3 * go.float().norm().item())
        assert err < 2 ** -7, (name, err)
    assert _lib.read_status()[0] == 0


@pytest.mark.parametrize("lens,pad,Hq,Hkv", [([128, 300], 0, 4, 2), ([77, 1, 513], 40, 8, 1), ([640], 128, 2, 2)])
def test_block_attention_against_key_blocks(lens, pad, Hq, Hkv):
    """What ring attention asks of the 128-wide kernels: keys that start elsewhere in a longer tensor, blocks that take
    no part, and dq added to in a second call.  Float32 on the CPU is the oracle; P and dS are bf16, 2^-7 of the norm."""
    from xorl_b200.parallel.sequence_parallel import block_attention, block_attention_bwd
    torch.manual_seed(5)
    D, T, B = 128, sum(lens), len(lens)
    cu = _make_cu(lens)
    Tk = 2 * T + pad                                          # two key sets behind `pad` rows that nobody sees
    starts = torch.tensor([0] + lens[:-1]).cumsum(0).to(torch.int32)
    own, other = (starts + pad).to(DEV), (starts + pad + T).to(DEV)
    if B > 1:
        other[0] = -1
    q, go = (torch.randn(T, Hq, D, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(Tk, Hkv, D, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    scale = D ** -0.5
    parts = {dev: [block_attention(*(t.to(dev) if dev == DEV else t.cpu().float() for t in (q, k, v)),
                                   cu.to(dev), ks.to(dev), causal, scale) for ks, causal in ((own, True), (other, False))]
             for dev in (DEV, "cpu")}
    close = lambda name, a, b: (a.cpu().float() - b.float()).norm() <= 2 ** -7 * b.float().norm() or pytest.fail(name)
    for (o, l), (ro, rl) in zip(parts[DEV], parts["cpu"]):
        close("out", o, ro)
        seen = rl.isfinite()
        assert torch.equal(l.cpu().isfinite(), seen) and (l.cpu() - rl)[seen].abs().max() < 1e-2
    (o1, l1), (o2, l2) = parts["cpu"]
    lse = torch.logaddexp(l1, l2)
    mix = lambda o, l: o.float() * torch.exp(l - lse).transpose(0, 1).unsqueeze(-1)
    out = (mix(o1, l1) + mix(o2, l2)).bfloat16()
    got = {}
    for dev in (DEV, "cpu"):
        cast = (lambda t: t.to(dev)) if dev == DEV else (lambda t: t.cpu().float())
        delta = torch.full((Hq, T), float("nan"), device=dev)
        dq = torch.full((T, Hq, D), float("nan"), device=dev)
        got[dev] = []
        for i, (ks, causal) in enumerate(((own, True), (other, False))):
            got[dev] += block_attention_bwd(cast(q), cast(k), cast(v), cast(out), cast(go), lse.to(dev), delta, dq,
                                            cu.to(dev), ks.to(dev), causal, scale, i == 0)
        got[dev].append(dq)
    for name, a, b in zip(("dk", "dv", "dk other", "dv other", "dq"), got[DEV], got["cpu"]):
        close(name, a, b)


@pytest.mark.parametrize("D", [64, 128])
def test_gradient_rows_outside_every_document_are_zero(D, monkeypatch):
    """Documents that begin behind the first token and end before the last; every allocation holds NaN before."""
    from xorl_b200.ops import attention as A
    torch.manual_seed(6)
    T, Hq, Hkv = 400, 4, 2
    cu = torch.tensor([30, 190, 371], device=DEV, dtype=torch.int32)
    q, k, v = (torch.randn(T, h, D, device=DEV, dtype=torch.bfloat16) for h in (Hq, Hkv, Hkv))
    go = torch.randn(T, Hq, D, device=DEV, dtype=torch.bfloat16)
    dv = torch.full_like(v, float("nan"))
    monkeypatch.setattr(torch, "empty", lambda *a, **kw: torch.full(*a, float("nan"), **kw))
    if D == 64:
        out, lse, f32 = A._attn_fwd_hd64(q, k, v, cu, True, D ** -0.5, True)
        dq, dk = A._attn_bwd_hd64(q, k, v, f32, go, lse, cu, True, D ** -0.5, dv)
    else:
        out, lse = A._attn_fwd(q, k, v, cu, True, D ** -0.5)
        dq, dk = A._attn_bwd(q, k, v, out, go, lse, cu, True, D ** -0.5, dv)
    monkeypatch.undo()
    ins = [t[30:371].float().requires_grad_() for t in (q, k, v)]
    ref = A.attention_reference(*ins, cu - 30)
    ref.backward(go[30:371].float())
    for a, r in zip((out, dq, dk, dv), [ref.detach()] + [t.grad for t in ins]):
        assert (a[30:371].float() - r).norm() < 2 ** -7 * r.norm()
    for t in (dq, dk, dv) if D == 64 else (dq,):
        assert not t[:30].any() and not t[371:].any()


def test_attention_128_takes_more_tiles_than_a_grid_is_high():
    """66,000 documents of one token: every query sees its own key only."""
    from xorl_b200.ops import attention as A
    T, D = 66000, 128
    cu = torch.arange(T + 1, device=DEV, dtype=torch.int32)
    q, k, v, go = (torch.randn(T, 1, D, device=DEV, dtype=torch.bfloat16) for _ in range(4))
    out, lse = A._attn_fwd(q, k, v, cu, True, D ** -0.5)
    assert torch.equal(out, v)
    dv = torch.empty_like(v)
    dq, dk = A._attn_bwd(q, k, v, out, go, lse, cu, True, D ** -0.5, dv)
    # P and dP - delta: the two fp32 sums over 128 products and the lse round differently
    assert (dv.float() - go.float()).abs().max() <= 2 ** -8 * go.float().abs().max()
    assert dq.abs().max() < 1e-4 and dk.abs().max() < 1e-4


def _attention_float64(qkv, wq, wk, cos, sin, lens, Hq, Hkv, D, eps, causal):
    """The block in float64 without any rounding inside."""
    T = qkv.shape[0]
    q, k, v = (t.reshape(T, -1, D) for t in qkv.split([Hq * D, Hkv * D, Hkv * D], dim=-1))
    norm = lambda t, w: t if w is None else t * torch.rsqrt(t.pow(2).mean(-1, keepdim=True) + eps) * w

    def rope(t):
        a, b, c, s = t[..., :D // 2], t[..., D // 2:], cos.double()[:, None], sin.double()[:, None]
        return torch.cat([a * c - b * s, b * c + a * s], -1)

    q, k = rope(norm(q, wq)), rope(norm(k, wk))
    out, s = [], 0
    for n in lens:
        qb, kb, vb = (t[s:s + n].transpose(0, 1) for t in (q, k, v))
        kb, vb = kb.repeat_interleave(Hq // Hkv, 0), vb.repeat_interleave(Hq // Hkv, 0)
        sc = qb @ kb.transpose(1, 2) / math.sqrt(D)
        if causal:
            sc = sc.masked_fill(~torch.ones(n, n, dtype=torch.bool, device=sc.device).tril(), float("-inf"))
        out.append((sc.softmax(-1) @ vb).transpose(0, 1).reshape(n, Hq * D))
        s += n
    return torch.cat(out)


@pytest.mark.parametrize("lens,Hq,Hkv,causal,do_norm", [
    ([1], 2, 1, True, True), ([63, 1, 65], 4, 4, True, False), ([128, 64, 129], 8, 2, False, False),
    ([257, 700, 3], 16, 4, True, True), ([511], 6, 2, False, True)])
def test_hd64_attention_loses_no_precision(lens, Hq, Hkv, causal, do_norm):
    """64-wide heads: the kernels against float64, next to the reference path with its fp32
    probabilities.  Without norm and rotation only the rounding of outputs and gradients to bf16 is left,
    1.6e-3 of the norm; bf16 probabilities would add as much again (1.4x).  In three parts they keep their 24 bits,
    and what the tensor core's fp32 sums add is below 2e-5."""
    from xorl_b200.ops import attention as A
    torch.manual_seed(0)
    D, T, eps = 64, sum(lens), 1e-6
    cu = _make_cu(lens)
    base = torch.randn(T, (Hq + 2 * Hkv) * D, device=DEV, dtype=torch.bfloat16)
    ws = [(1 + 0.1 * torch.randn(D, device=DEV)).bfloat16() if do_norm else None for _ in range(2)]
    pos = torch.cat([torch.arange(l, device=DEV) for l in lens]).float()
    ang = pos[:, None] / (1e4 ** (torch.arange(0, D, 2, device=DEV).float() / D))[None] * float(do_norm)
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    go = torch.randn(T, Hq * D, device=DEV, dtype=torch.bfloat16)

    def grads(fn, dtype=None):
        ins = [t if t is None else t.detach().to(dtype or t.dtype).requires_grad_() for t in (base, *ws)]
        y = fn(*ins)
        y.backward(go.to(y.dtype))
        return [y.detach()] + [t.grad for t in ins if t is not None]

    before = A.launch_count()
    got = grads(lambda x, a, b: A.qk_norm_rope_attention(x, a, b, cos, sin, cu, Hq, Hkv, D, eps, causal))
    assert A.launch_count() > before
    ref = grads(lambda x, a, b: A.qk_norm_rope_attention_reference(x, a, b, cos, sin, cu, Hq, Hkv, D, eps, causal,
                                                                  D ** -0.5))
    exact = grads(lambda x, a, b: _attention_float64(x, a, b, cos, sin, lens, Hq, Hkv, D, eps, causal), torch.float64)
    for name, g, r, e in zip(("out", "dqkv", "dwq", "dwk"), got, ref, exact):
        # a gradient that cancels to zero (a document of one token) does so to the rounding of the fp32 sums
        # dP and delta over 64 products: 64 * 2^-24 = 4e-6 of their terms
        base_norm = max(e.norm().item(), 1e-4 * go.double().norm().item())
        eg, er = ((t.double() - e).norm().item() / base_norm for t in (g, r))
        # weight gradients: 64 values rounded once each to bf16, up to half an ulp (2^-9) off
        assert eg <= 1.02 * er + (2 ** -9 if name in ("dwq", "dwk") else 2e-5), (name, eg, er)


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("lens,causal", [([70, 65, 1, 200, 127], True), ([129, 300, 63], False), ([64, 128, 1], True)])
def test_hd64_documents_do_not_see_each_others_infinities(lens, causal, value):
    """One document holds a non-finite value, and so do rows behind the last document.  Tiles of its neighbours
    run on into those rows; outputs and gradients of every other document have the bits of the clean call."""
    from xorl_b200.ops import attention as A
    torch.manual_seed(2)
    Hq, Hkv, D, tail = 4, 2, 64, 30
    n = sum(lens)
    cu = _make_cu(lens)
    base = torch.randn(n + tail, (Hq + 2 * Hkv) * D, device=DEV, dtype=torch.bfloat16)
    go = torch.randn(n + tail, Hq * D, device=DEV, dtype=torch.bfloat16)
    cos, sin = torch.ones(n + tail, D // 2, device=DEV), torch.zeros(n + tail, D // 2, device=DEV)

    def run(x, g):
        x = x.clone().requires_grad_()
        y = A.qk_norm_rope_attention(x, None, None, cos, sin, cu, Hq, Hkv, D, 1e-6, causal)
        y.backward(g)
        return y.detach(), x.grad

    before = A.launch_count()
    clean = run(base, go)
    assert A.launch_count() > before
    for bad in range(len(lens)):
        s = sum(lens[:bad])
        x, g = base.clone(), go.clone()
        for t in (x, g):
            t[s] = t[s + lens[bad] - 1] = t[n:] = value
        got = run(x, g)
        keep = torch.ones(n + tail, dtype=torch.bool, device=DEV)
        keep[s:s + lens[bad]] = keep[n:] = False
        for a, b in zip(got, clean):
            assert torch.equal(a[keep], b[keep])
        assert not got[1][n:].any()                           # rows of no document have no gradient


def _shifted(t):
    """The same values behind an address that only the type's own alignment holds for."""
    flat = torch.empty(t.numel() + 1, device=t.device, dtype=t.dtype)
    return flat[1:].view_as(t).copy_(t)


@pytest.mark.parametrize("D", [64, 128])
def test_qk_norm_rope_attention_on_shifted_buffers(D):
    """Rotation tables (both widths), and for 64-wide heads activations and output gradients, at odd offsets."""
    from xorl_b200.ops import attention as A
    torch.manual_seed(3)
    lens, Hq, Hkv = [100, 61], 4, 2
    T, cu = sum(lens), _make_cu(lens)
    base = torch.randn(T, (Hq + 2 * Hkv) * D, device=DEV, dtype=torch.bfloat16)
    ws = [(1 + 0.1 * torch.randn(D, device=DEV)).bfloat16().requires_grad_() for _ in range(2)]
    ang = torch.rand(T, D // 2, device=DEV) * 6
    go = torch.randn(T, Hq * D, device=DEV, dtype=torch.bfloat16)

    def run(x, cos, sin, g):
        x.requires_grad_()
        y = A.qk_norm_rope_attention(x, *ws, cos, sin, cu, Hq, Hkv, D)
        return [y.detach(), *torch.autograd.grad(y, [x, *ws], g)]

    cos, sin = ang.cos(), ang.sin()
    clean = run(base.clone(), cos, sin, go)
    for a, b in zip(run(base.clone(), _shifted(cos), _shifted(sin), go), clean):
        assert torch.equal(a, b)
    if D == 64:
        for a, b in zip(run(base.clone(), cos, sin, _shifted(go)), clean):
            assert torch.equal(a, b)
        got = run(_shifted(base), cos, sin, go)               # served by the reference
        for a, b in zip(got, clean):
            assert (a.float() - b.float()).norm() < 2 ** -7 * b.float().norm()


def test_hd64_attention_outside_the_kernels_range():
    """A width that does not fit the heads stays an error; gradients of the tables, and of the gradient, exist."""
    from xorl_b200.ops import attention as A
    torch.manual_seed(4)
    lens, Hq, Hkv, D = [40, 25], 4, 2, 64
    T, cu = sum(lens), _make_cu(lens)
    x = torch.randn(T, (Hq + 2 * Hkv) * D, device=DEV, dtype=torch.bfloat16)
    ang = torch.rand(T, D // 2, device=DEV) * 6
    cos, sin = ang.cos(), ang.sin()
    with pytest.raises(RuntimeError):
        A.qk_norm_rope_attention(x[:, :-D].contiguous(), None, None, cos, sin, cu, Hq, Hkv, D)
    A.qk_norm_rope_attention(x, None, None, cos.requires_grad_(), sin, cu, Hq, Hkv, D).float().sum().backward()
    assert cos.grad is not None and cos.grad.abs().sum() > 0
    cos = cos.detach()

    def second(fn):
        leaf = x.clone().requires_grad_()
        y = fn(leaf)
        (g,) = torch.autograd.grad(y, leaf, torch.ones_like(y), create_graph=True)
        return torch.autograd.grad(g.float().pow(2).sum(), leaf)[0].float()

    before = A.launch_count()
    got = second(lambda t: A.qk_norm_rope_attention(t, None, None, cos, sin, cu, Hq, Hkv, D))
    assert A.launch_count() > before
    ref = second(lambda t: A.qk_norm_rope_attention_reference(t, None, None, cos, sin, cu, Hq, Hkv, D, 1e-6, True,
                                                              D ** -0.5))
    # first and second derivative are the reference's on both sides
    assert torch.equal(got, ref)


@pytest.mark.parametrize("scale", [0.0, -0.1])
def test_hd64_attention_with_a_scale_that_is_not_positive(scale):
    from xorl_b200.ops import attention as A
    torch.manual_seed(7)
    cu, D = _make_cu([90, 70]), 64
    x = torch.randn(160, 8 * D, device=DEV, dtype=torch.bfloat16)
    cos, sin = torch.ones(160, D // 2, device=DEV), torch.zeros(160, D // 2, device=DEV)
    got = A.qk_norm_rope_attention(x, None, None, cos, sin, cu, 4, 2, D, scale=scale)
    assert torch.equal(got, A.qk_norm_rope_attention_reference(x, None, None, cos, sin, cu, 4, 2, D, 1e-6, True, scale))


def test_status_words_clean():
    from xorl_b200.ops import _lib
    assert _lib.read_status()[0] == 0


@pytest.mark.parametrize("E,K,N,counts", [(4, 256, 512, [100, 0, 300, 129]), (16, 2048, 1536, None),
                                          (8, 768, 2048, None)])
def test_grouped_linear_fwd_bwd(E, K, N, counts):
    from xorl_b200.ops import moe as moe_ops
    torch.manual_seed(0)
    if counts is None:
        counts = torch.randint(0, 700, (E,)).tolist()
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(counts)).to(DEV)
    S = ids.numel()
    dest, seg, _ = moe_ops.aligned_sort_indices(ids, E)
    rows = moe_ops.buffer_rows(S, E)
    xs = (torch.randn(S, K, device=DEV) * 0.5).to(torch.bfloat16)
    buf = torch.zeros(rows, K, device=DEV, dtype=torch.bfloat16).index_copy(0, dest, xs).requires_grad_()
    w = (torch.randn(E, K, N, device=DEV) * 0.05).to(torch.bfloat16).requires_grad_()
    go_s = torch.randn(S, N, device=DEV, dtype=torch.bfloat16)
    go = torch.zeros(rows, N, device=DEV, dtype=torch.bfloat16).index_copy(0, dest, go_s)
    y = moe_ops.grouped_linear(buf, w, seg)
    y.backward(go)
    # fp32 reference per expert
    xr = buf.detach().float().requires_grad_()
    wr = w.detach().float().requires_grad_()
    s = seg.tolist()
    yr = torch.zeros(rows, N, device=DEV)
    parts = []
    for e in range(E):
        parts.append(xr[s[e]:s[e + 1]] @ wr[e])
    yr = torch.cat(parts + [torch.zeros(rows - s[E], N, device=DEV)], 0)
    yr.backward(go.float())
    _close(y, yr, 2e-2, 0.02 * yr.abs().max().item(), "y")
    _close(buf.grad, xr.grad, 3e-2, 0.02 * xr.grad.abs().max().item(), "dx")
    _close(w.grad, wr.grad, 3e-2, 0.02 * wr.grad.abs().max().item(), "dw")


def test_moe_block_gpu_matches_reference():
    from xorl_b200.models.config import preset
    from xorl_b200.models.context import StepContext
    from xorl_b200.models.moe import MoEBlock
    from xorl_b200.parallel.state import init_parallel_state, reset_parallel_state
    reset_parallel_state()
    init_parallel_state(device_type="cuda")
    cfg = preset("qwen3-30b-a3b", hidden_size=512, num_experts=16, num_experts_per_tok=4,
                 moe_intermediate_size=256, num_hidden_layers=1)
    torch.manual_seed(0)
    blk = MoEBlock(cfg, 0, dtype=torch.bfloat16, device=DEV)
    for p in blk.parameters():
        torch.nn.init.normal_(p, 0, 0.05)
    T = 777
    x = (torch.randn(T, 512, device=DEV) * 0.5).to(torch.bfloat16).requires_grad_()
    ctx = StepContext(cu_seqlens=torch.tensor([0, T], device=DEV, dtype=torch.int32),
                      position_ids=torch.arange(T, device=DEV))
    out = blk(x, ctx)
    go = torch.randn_like(out)
    out.backward(go)
    w, idx, _ = blk.gate(x.detach())
    xr = x.detach().float()
    ref = torch.zeros(T, 512, device=DEV)
    gu, dn = blk.experts.gate_up_proj.detach().float(), blk.experts.down_proj.detach().float()
    for e in range(16):
        tok, slot = (idx == e).nonzero(as_tuple=True)
        if tok.numel() == 0:
            continue
        h = xr[tok] @ gu[e]
        a = torch.nn.functional.silu(h[:, :256]) * h[:, 256:]
        ref.index_add_(0, tok, (a @ dn[e]) * w[tok, slot].unsqueeze(-1))
    _close(out, ref, 3e-2, 0.03 * ref.abs().max().item(), "moe out")
    assert x.grad is not None and torch.isfinite(x.grad.float()).all()
    assert torch.isfinite(blk.experts.gate_up_proj.grad.float()).all()


@pytest.mark.parametrize("T,slices,out,rank,scaling", [(512, ((0, 256),), 256, 16, 2.0), (100, ((0, 256),), 256, 8, 1.0),
                                                       (700, ((0, 256), (256, 320), (320, 384)), 384, 16, 0.3),
                                                       (385, ((64, 128),), 384, 24, 2.0), (1, ((0, 64), (128, 192)), 256, 8, 0.5)])
def test_lora_linear_against_float64(T, slices, out, rank, scaling):
    """Adapters on whole and on partial outputs, with rows that have no adapter, against float64 and next to
    one product per factor: no error may be larger (that path rounds each delta twice more)."""
    from xorl_b200.adapters.lora import LoraLinear
    from xorl_b200.models.layers import Linear
    from xorl_b200.ops import lora as L
    torch.manual_seed(T)
    fin = 320
    mod = LoraLinear(Linear(fin, out, dtype=torch.bfloat16, device=DEV), rank, scaling * rank,
                     [(str(i), s, e) for i, (s, e) in enumerate(slices)])
    for p in mod.parameters():
        torch.nn.init.normal_(p, 0, 0.05)
    x0 = torch.randn(T, fin, device=DEV, dtype=torch.bfloat16)
    go = torch.randn(T, out, device=DEV, dtype=torch.bfloat16)

    def run(fn, dtype):
        x = x0.detach().clone().to(dtype).requires_grad_()
        ps = [p.detach().to(dtype).requires_grad_() for d in (mod.lora_A, mod.lora_B) for p in d.values()]
        y = fn(x, ps)
        y.backward(go.to(dtype))
        return [y.detach(), x.grad] + [p.grad for p in ps]

    def plain(x, ps, lin):
        w, n = mod.weight.to(x.dtype), len(slices)
        y = lin(x, w)
        cols = [y[:, :0]]
        cur = 0
        for i, (s, e) in enumerate(slices):
            cols += [y[:, cur:s], y[:, s:e] + lin(lin(x, ps[i]), ps[n + i]) * scaling]
            cur = e
        return torch.cat(cols + [y[:, cur:]], -1)

    from xorl_b200.ops.gemm import linear
    before = L.launch_count()
    got = run(lambda x, ps: L.lora_linear(x, mod.weight, scaling, slices, ps[:len(slices)], ps[len(slices):]), torch.bfloat16)
    assert T < 384 or L.launch_count() > before
    old = run(lambda x, ps: plain(x, ps, linear), torch.bfloat16)
    exact = run(lambda x, ps: plain(x, ps, torch.nn.functional.linear), torch.float64)
    assert L.lora_linear_ok(x0, mod.weight, slices, list(mod.lora_A.values()), list(mod.lora_B.values()))
    for g, o, e in zip(got, old, exact):
        eg, eo = ((t.double() - e).norm().item() / e.norm().item() for t in (g, o))
        assert eg <= 1.05 * eo + 2 ** -12, (eg, eo)


@pytest.mark.parametrize("M,I,K", [(384, 128, 64), (1000, 264, 328), (4096, 1536, 512), (2500, 5000, 192), (513, 8, 72)])
def test_linear_swiglu_has_the_bits_of_both_kernels(M, I, K):
    """The activation in the GEMM's epilogue: whole and cut tiles, widths that end inside one."""
    from xorl_b200.ops import _lib, activation as act, gemm as g
    torch.manual_seed(M)
    x = torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    w = (torch.randn(2 * I, K, device=DEV) * K ** -0.5).bfloat16()
    with torch.no_grad():
        before = g.launch_count() + act.launch_count()
        got = act.linear_swiglu(x, w)
        assert g.launch_count() + act.launch_count() - before == 2      # one kernel, counted by both
        assert torch.equal(got, act.swiglu(g.linear(x, w)))
    assert _lib.read_status()[0] == 0
