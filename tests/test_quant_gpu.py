"""fp8 block-scaled GEMM and quantisation kernels, token-loss head and Muon GEMM path on a B200,
each against a plain PyTorch fp32 reference of the same op."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from xorl_b200.ops import _lib
    _lib.cuda_lib()          # fail loudly if the native library is missing on a GPU box
    yield
    assert all(v == 0 for v in _lib.read_status()[:4]), _lib.read_status()


@pytest.mark.parametrize("M,K", [(256, 512), (1000, 1024), (3, 128)])
def test_quant_rows_matches_reference(M, K):
    from xorl_b200.ops import fp8_gemm, quantize as Q
    torch.manual_seed(M + K)
    x = (torch.randn(M, K, device="cuda") * 3).bfloat16()
    q, s = fp8_gemm.quantize_rows(x)
    q_ref, s_ref = Q.block_fp8_quantize_1x128(x)
    torch.testing.assert_close(s, s_ref, rtol=1e-6, atol=0)
    # a value on a rounding boundary may fall either way: compare after dequantisation
    d, d_ref = q.float() * s.repeat_interleave(128, 1), q_ref.float() * s_ref.repeat_interleave(128, 1)
    assert (d - d_ref).abs().max() <= 0.07 * x.float().abs().max()
    assert (q.view(torch.uint8) != q_ref.view(torch.uint8)).float().mean() < 3e-3
    assert (d - x.float()).abs().max() <= 0.07 * x.float().abs().max()


@pytest.mark.parametrize("N,K", [(256, 384), (300, 200)])
def test_quant_blocks_roundtrip(N, K):
    from xorl_b200.ops import fp8_gemm, quantize as Q
    torch.manual_seed(N + K)
    w = torch.randn(N, K, device="cuda").bfloat16()
    q, s = fp8_gemm.quantize_blocks(w)
    q_ref, s_ref = Q.block_fp8_quantize_128x128(w)
    torch.testing.assert_close(s, s_ref, rtol=1e-6, atol=0)
    # x * (1 / scale) against x / scale: values on a rounding boundary may fall either way
    assert (q.view(torch.uint8) != q_ref.view(torch.uint8)).float().mean() < 3e-3
    back = fp8_gemm.dequantize_blocks(q, s)
    ref = Q.block_fp8_dequantize_128x128(q, s)
    torch.testing.assert_close(back.float(), ref.float(), rtol=0, atol=0)


@pytest.mark.parametrize("M,N,K", [(128, 128, 128), (256, 384, 1024), (1000, 200, 512), (4096, 4096, 4096)])
def test_block_fp8_gemm_matches_fp32_reference(M, N, K):
    from xorl_b200.ops import fp8_gemm, quantize as Q
    torch.manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda").bfloat16()
    # give K blocks very different magnitudes so a wrong scale index cannot hide
    a = a * (1 + torch.arange(K // 128, device="cuda").repeat_interleave(128)).bfloat16()
    b = torch.randn(N, K, device="cuda").bfloat16() * 0.05
    aq, as_ = fp8_gemm.quantize_rows(a)
    bq, bs = fp8_gemm.quantize_blocks(b)
    out = fp8_gemm.block_fp8_gemm(aq, as_, bq, bs)
    ref = Q.block_fp8_gemm_reference(aq, as_, bq, bs, out_dtype=torch.float32)
    err = (out.float() - ref).abs().max() / ref.abs().max()
    assert err < 1e-2, err                                    # bf16 output rounding only
    dense = a.float() @ b.float().t()
    assert (out.float() - dense).norm() / dense.norm() < 0.06  # fp8 quantisation noise


@pytest.mark.parametrize("shape", [(512, 256, 384), (200, 320, 200)])
def test_fp8_linear_training_step(shape):
    """Forward and input-gradient GEMMs on e4m3 operands (cached weight codes, transposed for dgrad), weight
    gradient in bf16; sizes that are not multiples of 128 are padded."""
    from xorl_b200.adapters.fp8 import _FP8LinearFn
    from xorl_b200.ops import fp8_grouped
    M, K, N = shape
    torch.manual_seed(0)
    x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = (torch.randn(N, K, device="cuda") * 0.05).bfloat16().requires_grad_()
    g = torch.randn(M, N, device="cuda", dtype=torch.bfloat16)
    for fp8_backward in (True, False):
        x.grad = w.grad = None
        y = _FP8LinearFn.apply(x, w, fp8_backward)
        y.backward(g)
        ref = x.detach().float() @ w.detach().float().t()
        dx_ref = g.float() @ w.detach().float()
        dw_ref = g.float().t() @ x.detach().float()
        assert (y.float() - ref).norm() / ref.norm() < 0.06
        assert (x.grad.float() - dx_ref).norm() / dx_ref.norm() < (0.06 if fp8_backward else 0.01)
        assert (w.grad.float() - dw_ref).norm() / dw_ref.norm() < 0.01
    cache = w._xb_fp8_cache
    _FP8LinearFn.apply(x, w, True)
    assert w._xb_fp8_cache is cache                           # weights unchanged: codes reused
    fp8_grouped.invalidate_weight_cache()
    _FP8LinearFn.apply(x, w, True)
    assert w._xb_fp8_cache is not cache


def test_token_loss_head_matches_autograd():
    from xorl_b200.ops import rl_losses
    from xorl_b200.ops.loss import fused_linear_token_loss
    torch.manual_seed(0)
    T, H, V = 700, 256, 1000
    h = (torch.randn(T, H, device="cuda") * 0.5).bfloat16().requires_grad_()
    w = (torch.randn(V, H, device="cuda") * 0.05).bfloat16().requires_grad_()
    labels = torch.randint(0, V, (T,), device="cuda")
    labels[::7] = -100
    old = torch.full((T,), -6.5, device="cuda")
    adv = torch.randn(T, device="cuda")
    fn = lambda lp, mask: rl_losses.importance_sampling(lp, mask, old_logprobs=old, advantages=adv)
    loss, lp, _ = fused_linear_token_loss(h, w, labels, fn, 1.0, chunk_tokens=256)
    loss.backward()
    h32 = h.detach().float().requires_grad_()
    w32 = w.detach().float().requires_grad_()
    logits = h32 @ w32.t()
    lp_ref = -torch.nn.functional.cross_entropy(logits, labels, ignore_index=-100, reduction="none")
    loss_ref, _ = fn(lp_ref, (labels != -100).float())
    loss_ref.backward()
    torch.testing.assert_close(lp, lp_ref.detach(), rtol=2e-2, atol=3e-2)
    assert abs(loss.item() - loss_ref.item()) < 2e-2 * max(1.0, abs(loss_ref.item()))
    assert (h.grad.float() - h32.grad).norm() / h32.grad.norm() < 3e-2
    assert (w.grad.float() - w32.grad).norm() / w32.grad.norm() < 3e-2


def test_muon_newton_schulz_on_tcgen05_gemm():
    from xorl_b200.optim.muon import gram_newton_schulz, newton_schulz
    torch.manual_seed(0)
    G = torch.randn(256, 1024, device="cuda")
    X = newton_schulz(G).float()
    Y = gram_newton_schulz(G).float()
    Xc = newton_schulz(G.cpu()).float()
    sv = torch.linalg.svdvals(X)
    assert sv.min() > 0.5 and sv.max() < 1.3
    assert (X.cpu() - Xc).norm() / Xc.norm() < 0.05
    assert (X - Y).norm() / X.norm() < 0.06


@pytest.mark.parametrize("M,K,block,dt", [(2048, 512, 512, torch.bfloat16), (1000, 256, 256, torch.float32),
                                          (2304, 1024, 1024, torch.bfloat16)])
def test_symmetric_gemm_matches_full_product(M, K, block, dt):
    """Lower panels through the GEMM kernel + mirror kernel against the full product and fp32."""
    from xorl_b200.ops import gemm as G
    torch.manual_seed(0)
    x = (torch.randn(M, K, device="cuda") * 0.1).bfloat16()
    before = G.launch_count()
    c = G.gemm_symmetric(x, out_dtype=dt, block=block, min_rows=0)
    panels = -(-M // block)
    assert G.launch_count() == before + panels + 1
    full = G.gemm(x, x, out_dtype=dt)
    low = torch.tril(torch.ones(M, M, device="cuda", dtype=torch.bool))
    assert (c[low].float() - full[low].float()).abs().max() <= 1e-2 * full.float().abs().max()
    assert torch.equal(c, c.t())                             # exactly symmetric after the mirror
    ref = x.float() @ x.float().t()
    assert (c.float() - ref).abs().max() <= 2e-2 * ref.abs().max()
    # a product of two commuting symmetric factors
    a = full.to(torch.bfloat16)
    s2 = G.gemm_symmetric(a, a, block=block, min_rows=0).float()
    ref2 = a.float() @ a.float().t()
    assert (s2 - ref2).abs().max() <= 3e-2 * ref2.abs().max()


def test_muon_on_large_matrix_uses_symmetric_panels(monkeypatch):
    from xorl_b200.ops import gemm as G
    from xorl_b200.optim.muon import newton_schulz
    monkeypatch.setattr(G, "SYMMETRIC_MIN_ROWS", 0)          # the default keeps small matrices on the plain GEMM
    torch.manual_seed(1)
    Gm = torch.randn(2048, 2560, device="cuda")
    before = G.launch_count()
    X = newton_schulz(Gm, steps=5).float()
    # per step: 2 symmetric products (2 panels + mirror each) + 1 plain GEMM
    assert G.launch_count() - before == 5 * (2 * 3 + 1)
    sv = torch.linalg.svdvals(X)
    assert sv.min() > 0.4 and sv.max() < 1.3


@pytest.mark.parametrize("scoring,renorm,E,k,bias", [("softmax", True, 128, 8, False), ("softmax", False, 8, 2, False),
                                                     ("sigmoid", True, 256, 8, True), ("softmax_after_topk", False, 32, 4, False),
                                                     ("softmax", True, 60, 3, False)])
def test_moe_route_kernel_matches_torch(scoring, renorm, E, k, bias, monkeypatch):
    from xorl_b200.ops import moe
    torch.manual_seed(E + k)
    T = 1000
    logits = torch.randn(T, E, device="cuda")
    cb = torch.randn(E, device="cuda") * 0.3 if bias else None
    a = logits.clone().requires_grad_()
    w, idx, probs = moe.topk_route(a, k, renorm, scoring, 2.5, correction_bias=cb)           # kernel
    monkeypatch.setenv("XORL_B200_ROUTE_KERNEL", "0")
    b = logits.clone().requires_grad_()
    w2, idx2, probs2 = moe.topk_route(b, k, renorm, scoring, 2.5, correction_bias=cb)        # torch ops
    assert torch.equal(idx.sort(-1).values, idx2.sort(-1).values)
    torch.testing.assert_close(probs, probs2, rtol=1e-5, atol=1e-6)
    o1, o2 = idx.argsort(-1), idx2.argsort(-1)
    torch.testing.assert_close(w.gather(1, o1), w2.gather(1, o2), rtol=1e-5, atol=1e-6)
    gw, gp = torch.randn_like(w), torch.randn_like(probs)
    ((w.gather(1, o1) * gw).sum() + (probs * gp).sum()).backward()
    ((w2.gather(1, o2) * gw).sum() + (probs2 * gp).sum()).backward()
    torch.testing.assert_close(a.grad, b.grad, rtol=1e-4, atol=1e-5)


def test_moe_permute_combine_kernels_match_torch_path(monkeypatch):
    """The gather kernels (permute, weighted combine and their backward) against the index_select /
    index_copy formulation, forward and every gradient."""
    from xorl_b200.models.config import preset
    from xorl_b200.models.context import StepContext
    from xorl_b200.models.moe import MoEBlock
    from xorl_b200.parallel.state import init_parallel_state, reset_parallel_state
    reset_parallel_state()
    init_parallel_state(device_type="cuda")
    cfg = preset("qwen3-30b-a3b", hidden_size=256, num_experts=8, num_experts_per_tok=3,
                 moe_intermediate_size=128, num_hidden_layers=1)
    torch.manual_seed(0)
    blk = MoEBlock(cfg, 0, dtype=torch.bfloat16, device="cuda")
    for p in blk.parameters():
        torch.nn.init.normal_(p, 0, 0.05)
    T = 515
    x0 = (torch.randn(T, 256, device="cuda") * 0.5).to(torch.bfloat16)
    go = torch.randn(T, 256, device="cuda").to(torch.bfloat16)
    ctx = StepContext(cu_seqlens=torch.tensor([0, T], device="cuda", dtype=torch.int32),
                      position_ids=torch.arange(T, device="cuda"))
    res = {}
    for mode in ("1", "0"):
        monkeypatch.setenv("XORL_B200_MOE_KERNELS", mode)
        for p in blk.parameters():
            p.grad = None
        x = x0.clone().requires_grad_()
        out = blk(x, ctx)
        out.backward(go)
        res[mode] = (out.detach().float(), x.grad.float(), blk.gate.weight.grad.float(),
                     blk.experts.gate_up_proj.grad.float(), blk.experts.down_proj.grad.float())
    for a, b, name in zip(res["1"], res["0"], ("out", "dx", "dgate", "dgate_up", "ddown")):
        tol = 0.02 * b.abs().max().item() + 1e-4
        assert (a - b).abs().max().item() <= tol, (name, (a - b).abs().max().item(), tol)
    reset_parallel_state()


@pytest.mark.parametrize("N,rank,E,k,T", [(2, 1, 8, 2, 300), (8, 3, 128, 8, 4096), (4, 0, 16, 4, 1000)])
def test_ep_plan_kernel_matches_torch_formulation(N, rank, E, k, T):
    """Destination rank / row of every token slot and the local segment table, against the
    argsort / cumsum formulation (rows of an expert keep slot order in both)."""
    import ctypes
    from xorl_b200.ops import _lib
    torch.manual_seed(N * 100 + E)
    El = E // N
    idx = torch.randint(0, E, (T, k), device="cuda")
    flat = idx.reshape(-1)
    S = flat.numel()
    counts = torch.bincount(flat, minlength=E).to(torch.int32)
    table = torch.randint(0, 2 * S // E, (N, E), device="cuda", dtype=torch.int32)
    table[rank] = counts
    cap = (int(1.5 * S) + El * 127 + 127) // 128 * 128
    dr = torch.empty(S, device="cuda", dtype=torch.int32)
    drow = torch.empty(S, device="cuda", dtype=torch.int32)
    seg = torch.empty(El + 1, device="cuda", dtype=torch.int32)
    tot = torch.empty(El, device="cuda", dtype=torch.int32)
    ovf = torch.zeros(1, device="cuda", dtype=torch.int32)
    _lib.check(_lib.cuda_lib().xb_ep_plan(flat.data_ptr(), S, table.data_ptr(), rank, N, E, El, cap, dr.data_ptr(),
                                          drow.data_ptr(), seg.data_ptr(), tot.data_ptr(), ovf.data_ptr(),
                                          _lib.stream_ptr()), "xb_ep_plan")
    # torch formulation
    tl = table.long()
    t_all = tl.sum(0)
    padded = (t_all + 127) // 128 * 128
    pe = padded.view(N, El)
    seg_start = (pe.cumsum(1) - pe).reshape(-1)
    before = tl[:rank].sum(0) if rank > 0 else torch.zeros_like(t_all)
    base = seg_start + before
    order = torch.argsort(flat, stable=True)
    c64 = counts.long()
    starts = c64.cumsum(0) - c64
    rank_in_e = torch.empty_like(flat)
    rank_in_e[order] = torch.arange(S, device="cuda") - starts[flat[order]]
    ref_row = base[flat] + rank_in_e
    ref_rank = flat // El
    over = ref_row >= cap
    assert torch.equal(dr.long(), torch.where(over, torch.full_like(ref_rank, -1), ref_rank))
    assert torch.equal(drow.long()[~over], ref_row[~over])
    assert bool(ovf.item()) == bool(over.any().item())
    mine = slice(rank * El, (rank + 1) * El)
    ref_seg = torch.cat([padded.new_zeros(1), padded[mine].cumsum(0)]).clamp(max=cap // 128 * 128)
    assert torch.equal(seg.long(), ref_seg) and torch.equal(tot.long(), t_all[mine])


# ---- block-scaled fp8 grouped GEMM (power-of-two scales on the tensor core) ----------------------
def _mx_case(E, K, N, counts, seed=0):
    from xorl_b200.ops import moe as moe_ops
    g = torch.Generator(device="cpu").manual_seed(seed)
    ids = torch.cat([torch.full((c,), e, dtype=torch.int64) for e, c in enumerate(counts)])
    dest, seg, _ = moe_ops.aligned_sort_indices(ids.cuda(), E)
    rows = moe_ops.buffer_rows(ids.numel(), E)
    x = torch.zeros(rows, K, dtype=torch.bfloat16)
    x[dest.cpu()] = (torch.randn(ids.numel(), K, generator=g) * torch.rand(ids.numel(), 1, generator=g) * 3).bfloat16()
    w = (torch.randn(E, K, N, generator=g) * 0.05 * (1 + torch.arange(E).view(E, 1, 1))).bfloat16()
    return x.cuda(), w.cuda(), seg


def test_mx_quantisers_match_the_restatement():
    from xorl_b200.ops import fp8_grouped as fg
    x, w, _ = _mx_case(3, 384, 256, [100, 0, 300])
    q, sf = fg.quantize_rows(x)
    qr, er = fg.quantize_rows_ref(x.cpu())
    assert torch.equal(sf[:, :3].cpu().int() - 127, er)
    assert torch.equal(q.cpu().view(torch.float8_e4m3fn).float(), qr.float())
    qe = fg.quantize_experts(w)
    wq, we = fg.quantize_weight_ref(w.cpu())
    assert torch.equal(qe.sf_kn[:, :, :2].cpu().int() - 127, we)
    assert torch.equal(qe.sf_nk[:, :, :3].cpu().int() - 127, we.transpose(1, 2))
    assert torch.equal(qe.q_kn.cpu().view(torch.float8_e4m3fn).float(), wq.float())
    assert torch.equal(qe.q_nk.cpu().view(torch.float8_e4m3fn).float(), wq.float().transpose(1, 2))


@pytest.mark.parametrize("E,K,N,counts", [
    (3, 384, 256, [100, 0, 300]),                       # an empty expert, N not a multiple of 192
    (4, 768, 2048, [129, 640, 1, 255]),                 # down projection of Qwen3-30B-A3B
    (16, 2048, 1536, [2048 + 37 * (i % 5) - 64 * (i % 3) for i in range(16)]),   # gate_up projection, EP 8 load
])
def test_mx_grouped_gemm_matches_dequantised_matmul(E, K, N, counts):
    from xorl_b200.ops import _lib
    from xorl_b200.ops import fp8_grouped as fg
    x, w, seg = _mx_case(E, K, N, counts, seed=E)
    xq, sfx = fg.quantize_rows(x)
    qe = fg.quantize_experts(w)
    y = fg.grouped_rows_mx(xq, sfx, qe.q_nk, qe.sf_nk, seg)
    torch.cuda.synchronize()
    _lib.raise_on_status()
    ref = fg.grouped_rows_ref(x.cpu().float(), w.cpu().float(), seg.cpu())
    err = (y.cpu().float() - ref).abs().max() / ref.abs().max()
    assert err < 6e-3, err                               # bf16 rounding of the output only
    # against the unquantised product: the error of the fp8 scheme itself
    exact = torch.zeros_like(ref)
    s = seg.cpu().tolist()
    for e in range(E):
        exact[s[e]:s[e + 1]] = x.cpu().float()[s[e]:s[e + 1]] @ w.cpu().float()[e]
    rel = (y.cpu().float() - exact).norm() / exact.norm()
    assert rel < 0.05, rel


def test_mx_grouped_linear_gradients():
    """Forward and input gradient in fp8 against the bf16 grouped linear; weight gradient (bf16) equal."""
    from xorl_b200.ops import fp8_grouped as fg
    from xorl_b200.ops import moe as moe_ops
    x, w, seg = _mx_case(4, 256, 384, [200, 31, 0, 500], seed=5)
    outs = {}
    for mode in (None, "fp8", "bf16"):
        xi, wi = x.clone().requires_grad_(), w.clone().requires_grad_()
        y = moe_ops.grouped_linear(xi, wi, seg, mode)
        dy = torch.randn(y.shape, generator=torch.Generator().manual_seed(1)).bfloat16().cuda()
        valid = torch.zeros(y.shape[0], 1, device="cuda", dtype=torch.bfloat16)
        s = seg.tolist()
        valid[: s[-1]] = 1
        y.backward(dy * valid)
        outs[mode] = (y.float(), xi.grad.float(), wi.grad.float())
    for mode in ("fp8", "bf16"):
        for a, b, name, tol in zip(outs[mode], outs[None], ("y", "dx", "dw"), (0.05, 0.05, 1e-6)):
            if mode == "bf16" and name == "dx":
                tol = 1e-6
            rel = (a - b).norm() / b.norm()
            assert rel <= tol, (mode, name, float(rel))


@pytest.mark.parametrize("S,E", [(0, 4), (1, 1), (2, 8), (1000, 8), (1024, 16), (1025, 128), (32768, 16), (70000, 512),
                                 (160000, 1024)])
def test_moe_plan_matches_the_sorting_path(S, E):
    from xorl_b200.ops import _lib, moe
    torch.manual_seed(S)
    ids = torch.randint(0, E, (S,), device="cuda")
    ids[ids == E // 2] = 0                                   # an expert without rows, one with more than its share
    rows = moe.buffer_rows(S, E)
    dest, seg, slot = moe.sort_plan(ids, E, rows)
    d0, s0, _ = moe.aligned_sort_indices(ids, E)
    inv = torch.full((rows,), -1, device="cuda", dtype=torch.int32)
    inv[d0] = torch.arange(S, device="cuda", dtype=torch.int32)
    assert torch.equal(dest, d0) and torch.equal(seg, s0) and torch.equal(slot, inv)
    assert _lib.read_status()[0] == 0


def _moe_inputs(T, E, k, H=64, I=64):
    from types import SimpleNamespace
    gen = torch.Generator(device="cuda").manual_seed(T)
    rnd = lambda *shape: (torch.randn(*shape, generator=gen, device="cuda") * 0.1).bfloat16()
    experts = SimpleNamespace(gate_up_proj=rnd(E, H, 2 * I), down_proj=rnd(E, I, H))
    ids = torch.rand(T, E, generator=gen, device="cuda").topk(k, -1)[1]
    return rnd(T, H), torch.rand(T, k, generator=gen, device="cuda"), ids, experts


@pytest.mark.parametrize("bad", [-1, 8, 2 ** 31 - 1, -2 ** 40])
@pytest.mark.parametrize("T", [1, 700])
def test_expert_id_out_of_range_is_refused(T, bad):
    from xorl_b200.ops import moe
    x, w, ids, experts = _moe_inputs(T, 8, 2)
    good = moe.local_moe_forward(x, w, ids, experts, 8)
    broken = ids.clone()
    broken[T // 2, 1] = bad
    with pytest.raises(RuntimeError, match="1 of %d expert ids" % (2 * T)):
        moe.local_moe_forward(x, w, broken, experts, 8)
    assert torch.equal(moe.local_moe_forward(x, w, ids, experts, 8), good)


def test_slots_without_a_row_touch_no_other_token():
    """Where nobody can raise (a captured graph): NaN for the token of the slot, in both directions, and the
    values of the clean plan for every other token."""
    from xorl_b200.ops import moe
    T, E, k = 300, 8, 2
    x, w, ids, _ = _moe_inputs(T, E, k)
    w[17, 1] = 0.0                                            # a weight of zero hides nothing
    rows = moe.buffer_rows(T * k, E)
    dout = torch.randn_like(x)

    def run(ids):
        dest, _, slot = moe.sort_plan(ids.reshape(-1), E, rows)
        xi, wi = x.clone().requires_grad_(), w.clone().requires_grad_()
        y = moe._Combine.apply(moe._Permute.apply(xi, dest.view(T, k), slot), wi, dest.view(T, k), slot)
        y.backward(dout)
        return y.detach(), xi.grad, wi.grad

    broken = ids.clone()
    broken[17, 1], broken[250, 0] = E, -3
    hit = torch.zeros(T, dtype=torch.bool, device="cuda")
    hit[[17, 250]] = True
    clean, got = run(ids), run(broken)
    for c, g in zip(clean[:2], got[:2]):
        assert g[hit].isnan().all() and torch.equal(g[~hit], c[~hit])
    lost = broken != ids
    assert got[2][lost].isnan().all() and torch.equal(got[2][~lost], clean[2][~lost])


def test_router_on_logits_that_are_not_numbers_is_refused():
    from xorl_b200.models import ModelConfig
    from xorl_b200.models.context import StepContext
    from xorl_b200.models.moe import MoEBlock
    cfg = ModelConfig.from_dict(dict(model_type="qwen3_moe", vocab_size=64, hidden_size=64, num_hidden_layers=1,
                                     num_attention_heads=2, num_key_value_heads=2, head_dim=32, intermediate_size=64,
                                     num_experts=8, num_experts_per_tok=2, moe_intermediate_size=64))
    block = MoEBlock(cfg, 0, dtype=torch.bfloat16, device="cuda")
    for p in block.parameters():
        torch.nn.init.normal_(p, 0.0, 0.02)
    x = torch.randn(50, 64, device="cuda").bfloat16()
    ctx = StepContext(cu_seqlens=torch.tensor([0, 50], device="cuda", dtype=torch.int32),
                      position_ids=torch.arange(50, device="cuda"), causal=True, training=True)
    assert block(x, ctx).isfinite().all()
    x[7, 3] = float("nan")
    with pytest.raises(RuntimeError, match="expert ids"):
        block(x, ctx)


@pytest.mark.parametrize("T,E,k,renorm,scale", [(1, 1, 1, True, 1.0), (300, 8, 2, True, 1.0), (513, 128, 8, True, 2.5),
                                                (77, 60, 3, False, 0.5), (64, 512, 32, True, 1.0)])
def test_chosen_weights_and_balancing_loss_match_torch(T, E, k, renorm, scale):
    from xorl_b200.ops import moe
    torch.manual_seed(T)
    logits = torch.randn(T, E, device="cuda")
    idx = torch.randint(0, E, (T, k), device="cuda")         # with repeats: both slots contribute
    counts = moe.expert_histogram(idx, E)
    gw = torch.randn(T, k, device="cuda")

    def run(kernels):
        x = logits.clone().requires_grad_()
        p = torch.softmax(x, -1)
        if kernels:
            w, aux = moe.chosen_weights(p, idx, renorm, scale), moe.load_balancing_loss(p, idx, E, counts=counts, scale=0.3)
        else:
            w = moe._renorm_reference(p, idx, renorm, scale)
            aux = 0.3 * E * torch.dot(counts.float() / (T * k), p.mean(0))
        ((w * gw).sum() + 7 * aux).backward()
        return w.detach(), aux.detach(), x.grad

    for got, ref in zip(run(True), run(False)):
        torch.testing.assert_close(got, ref, rtol=2e-5, atol=2e-6)


@pytest.mark.parametrize("counts,K,N", [([0, 130, 1, 0], 256, 264), ([3], 128, 128), ([0, 0], 64, 512), ([100] * 130, 64, 72)])
@pytest.mark.parametrize("dtype,accumulate", [(torch.float32, False), (torch.float32, True), (torch.bfloat16, False),
                                              (torch.bfloat16, True)])
def test_grouped_gemm_writes_all_rows_and_experts(counts, K, N, dtype, accumulate):
    """Rows behind the last segment are zero without a fill; weight gradients of every output form, experts
    without rows and row counts of an expert that are no multiple of a tile included."""
    from xorl_b200.ops import _lib, moe
    torch.manual_seed(K)
    E = len(counts)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(counts)).cuda()
    dest, seg, _ = moe.aligned_sort_indices(ids, E)
    rows = moe.buffer_rows(ids.numel(), E)
    x = torch.zeros(rows, K, device="cuda", dtype=torch.bfloat16)
    x[dest] = torch.randn(ids.numel(), K, device="cuda").bfloat16()
    w = torch.randn(E, K, N, device="cuda", dtype=torch.bfloat16)
    y = torch.full((rows, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    moe._grouped_rows_cuda(x, w, seg, y, b_kmajor=False, zero_tail=True)
    s = seg.tolist()
    assert (y[s[E]:] == 0).all()
    out0 = torch.randn(E, K, N, device="cuda").to(dtype)
    out = out0.clone() if accumulate else torch.full_like(out0, float("nan"))
    dy = torch.randn(rows, N, device="cuda", dtype=torch.bfloat16)
    moe._grouped_wgrad_cuda(x, dy, seg, out, accumulate)
    for e in range(E):
        a = x[s[e]:s[e + 1]].double()
        # fp32 sums of up to 256 products, one bf16 rounding where the output has it
        torch.testing.assert_close(y[s[e]:s[e + 1]].double(), a @ w[e].double(), rtol=2 ** -8, atol=1e-3)
        ref = a.t() @ dy[s[e]:s[e + 1]].double() + (out0[e].double() if accumulate else 0)
        torch.testing.assert_close(out[e].double(), ref, rtol=2 ** -8 if dtype == torch.bfloat16 else 1e-4, atol=1e-3)
    assert _lib.read_status()[0] == 0


@pytest.mark.parametrize("K,N", [(8, 64), (40, 128), (168, 72)])
@pytest.mark.parametrize("dtype,accumulate", [(torch.float32, False), (torch.bfloat16, True)])
def test_grouped_weight_gradient_of_ragged_heights(K, N, dtype, accumulate):
    """Output rows that end inside a warp's 32, or before it."""
    from xorl_b200.ops import _lib, moe
    torch.manual_seed(K)
    seg = torch.tensor([0, 128, 384, 384], device="cuda", dtype=torch.int32)
    x, dy = (torch.randn(384, n, device="cuda").bfloat16() for n in (K, N))
    out0 = torch.randn(3, K, N, device="cuda").to(dtype)
    out = out0.clone() if accumulate else torch.full_like(out0, float("nan"))
    moe._grouped_wgrad_cuda(x, dy, seg, out, accumulate)
    for e, (a, b) in enumerate([(0, 128), (128, 384), (384, 384)]):
        ref = x[a:b].double().t() @ dy[a:b].double() + (out0[e].double() if accumulate else 0)
        # fp32 sums of up to 256 products, one bf16 rounding where the output has it
        torch.testing.assert_close(out[e].double(), ref, rtol=2 ** -8 if dtype == torch.bfloat16 else 1e-4, atol=1e-3)
    assert _lib.read_status()[0] == 0


def test_mx_scale_of_every_bf16_magnitude():
    """The power-of-two scale from the bits of the maximum, for every finite bf16 value of a block."""
    from xorl_b200.ops import fp8_grouped as fg
    vals = torch.arange(0, 0x7f80, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    x = torch.zeros(vals.numel(), 128, dtype=torch.bfloat16)
    x[:, 5] = -vals
    x[:, 9] = vals * 0.5
    q, sf = fg.quantize_rows(x.cuda())
    rq, re = fg.quantize_rows_ref(x)
    assert torch.equal(sf[:, 0].cpu().int(), re[:, 0] + 127)
    assert torch.equal(q.cpu().view(torch.float8_e4m3fn).float(), rq.float())
