"""tcgen05 GEMM against an fp32 PyTorch reference, all four operand layouts."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(a, b, a_mn, b_mn):
    A = a.float().t() if a_mn else a.float()
    B = b.float().t() if b_mn else b.float()
    return A @ B.t()


@pytest.fixture(params=["single", "pair"])
def variant(request):
    from xorl_b200.ops import gemm
    prev = gemm.set_variant(request.param)
    yield request.param
    gemm.set_variant(prev)
    from xorl_b200.ops import _lib
    assert all(v == 0 for v in _lib.read_status()[:4])


@pytest.mark.parametrize("a_mn,b_mn", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 512, 256), (4096, 6144, 4096), (304, 200, 136),
                                   (1000, 1256, 520), (72, 88, 40), (2048, 152064, 512), (4096, 4096, 256),
                                   (1536, 2304, 192), (5000, 640, 320)])
def test_gemm_layouts(M, N, K, a_mn, b_mn, variant):
    from xorl_b200.ops import gemm
    torch.manual_seed(0)
    dev = "cuda"
    a = torch.randn((K, M) if a_mn else (M, K), device=dev, dtype=torch.bfloat16)
    b = torch.randn((K, N) if b_mn else (N, K), device=dev, dtype=torch.bfloat16)
    c = gemm.gemm(a, b, a_mn=bool(a_mn), b_mn=bool(b_mn))
    torch.cuda.synchronize()
    ref = _ref(a, b, a_mn, b_mn)
    err = (c.float() - ref).abs().max().item()
    scale = ref.abs().max().item()
    assert err <= 1e-2 * scale + 1e-2, (err, scale)


def test_gemm_fp32_out_and_accumulate(variant):
    from xorl_b200.ops import gemm
    torch.manual_seed(1)
    a = torch.randn(512, 384, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(640, 384, device="cuda", dtype=torch.bfloat16)
    ref = a.float() @ b.float().t()
    c = gemm.gemm(a, b, out_dtype=torch.float32)
    assert torch.allclose(c, ref, rtol=1e-3, atol=1e-2)
    c2 = gemm.gemm(a, b, out=c.clone(), accumulate=True)
    assert torch.allclose(c2, 2 * ref, rtol=1e-3, atol=2e-2)
    cb = gemm.gemm(a, b)
    cb2 = gemm.gemm(a, b, out=cb.clone(), accumulate=True)
    assert torch.allclose(cb2.float(), 2 * ref, rtol=2e-2, atol=0.5)


@pytest.mark.parametrize("a_mn,b_mn", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("M,N,K", [(1, 8, 1024), (61, 4096, 4096), (16, 2048, 8192), (4096, 48, 4096), (136, 264, 1032),
                                   (128, 256, 4160), (520, 16, 12288), (8, 1000, 520)])
@pytest.mark.parametrize("out,accumulate", [(torch.bfloat16, False), (torch.bfloat16, True), (torch.float32, True)])
def test_gemm_with_few_tiles_splits_the_reduction(M, N, K, a_mn, b_mn, out, accumulate):
    """Cluster split-K: ragged tiles, remainders of K over the CTAs, every output form.  fp32 sums of K
    products differ by at most K * 2^-24 of the sum of their magnitudes; a bf16 result adds 2^-8."""
    from xorl_b200.ops import _lib, gemm
    if (a_mn and M % 8) or (b_mn and N % 8):
        pytest.skip("row pitch of an MN-major operand")
    torch.manual_seed(M + N)
    a = torch.randn((K, M) if a_mn else (M, K), device="cuda", dtype=torch.bfloat16)
    b = torch.randn((K, N) if b_mn else (N, K), device="cuda", dtype=torch.bfloat16)
    c0 = torch.randn(M, N, device="cuda").to(out)
    c = gemm.gemm(a, b, a_mn=bool(a_mn), b_mn=bool(b_mn), out=c0.clone(), accumulate=accumulate)
    again = gemm.gemm(a, b, a_mn=bool(a_mn), b_mn=bool(b_mn), out=c0.clone(), accumulate=accumulate)
    assert torch.equal(c, again)
    A, B = (a.t() if a_mn else a).double(), (b.t() if b_mn else b).double()
    ref = A @ B.t() + (c0.double() if accumulate else 0)
    bound = (A.abs() @ B.abs().t() + c0.double().abs()) * (K * 2.0 ** -24)
    if out == torch.bfloat16:
        bound = bound + ref.abs() * 2.0 ** -8
    assert ((c.double() - ref).abs() <= bound + 1e-6).all()
    assert all(v == 0 for v in _lib.read_status()[:4])


@pytest.mark.parametrize("M,N,K,K2", [(384, 256, 64, 8), (1000, 520, 520, 48), (4096, 6144, 1024, 72), (200, 512, 256, 16)])
@pytest.mark.parametrize("b_mn", [False, True])
def test_gemm_sum_of_two_products(M, N, K, K2, b_mn):
    from xorl_b200.ops import _lib
    from xorl_b200.ops.lora import gemm_sum
    torch.manual_seed(K2)
    x, x2 = (torch.randn(M, k, device="cuda", dtype=torch.bfloat16) for k in (K, K2))
    w, w2 = (torch.randn((k, N) if b_mn else (N, k), device="cuda", dtype=torch.bfloat16) for k in (K, K2))
    op = (lambda t: t.double()) if b_mn else (lambda t: t.double().t())
    ref = x.double() @ op(w) + x2.double() @ op(w2)
    mag = x.double().abs() @ op(w).abs() + x2.double().abs() @ op(w2).abs()
    # one bf16 rounding (2^-8 of the result), two where the second product is added to the first
    bound = mag * ((K + K2) * 2.0 ** -24) + (ref.abs() + (x.double() @ op(w)).abs()) * 2.0 ** -8
    assert ((gemm_sum(x, w, x2, w2, b_mn).double() - ref).abs() <= bound + 1e-6).all()
    assert all(v == 0 for v in _lib.read_status()[:4])


@pytest.mark.parametrize("rows", [(1024, 8), (8, 1024), (1024, 64, 1024, 8)])
def test_weight_used_at_several_lengths_sums_its_gradients(rows):
    """An engine's fp32 buffer with products on the side stream (2^31 multiply-adds and more) and on the main one.
    fp32 sums over all rows."""
    from xorl_b200.ops import gemm, grad_sink
    torch.manual_seed(0)
    N, K = 2048, 2048
    w = torch.nn.Parameter((torch.randn(N, K, device="cuda") * 0.02).bfloat16())
    xs = [torch.randn(r, K, device="cuda").bfloat16() for r in rows]
    dys = [torch.randn(r, N, device="cuda").bfloat16() for r in rows]
    ref = sum(d.double().t() @ x.double() for d, x in zip(dys, xs))
    bound = sum(d.double().abs().t() @ x.double().abs() for d, x in zip(dys, xs)) * (sum(rows) * 2.0 ** -24)
    for _ in range(10):
        w._xb_grad_buf, w._xb_grad_fresh = torch.full((N, K), float("nan"), device="cuda"), True
        for x, dy in zip(xs, dys):
            assert gemm.weight_grad(dy, x, w) is None
        grad_sink.join_wgrad_stream()
        assert ((w._xb_grad_buf.double() - ref).abs() <= bound + 1e-6).all()
