"""Linear layer with low-rank adapters on slices of its output, as one autograd function.

``y = x W^T + s (x A^T) B^T`` for every adapted slice of a fused projection.  The adapters of all slices
are stacked (``csrc/lora.cu``): ``d = s x Acat^T`` is one narrow GEMM, and ``x W^T + d Bcat^T`` one GEMM whose
reduction runs on over the ranks (``xb_gemm_bf16_pair_ext``), so the output is written once and no delta of its
size exists.  The input gradient has the same form, ``dy W + dd Acat`` with ``dd = s dy Bcat``.
Counterpart in the reference: src/xorl/lora/modules/linear.py:23-273.
"""
from __future__ import annotations

import ctypes

import torch

from . import _lib
from . import gemm as gemm_ops
from .gemm import gemm, weight_grad
from .grad_sink import current_wgrad_store, deliver_param_grad

_launches = 0


def launch_count() -> int:
    return _launches


def lora_linear_ok(x, w, slices, a, b) -> bool:
    """bf16 on the GPU, every extent and offset that a TMA copy or a packed vector starts at a multiple of
    eight elements; other layers take one product per factor."""
    if not (x.is_cuda and x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and x.shape[-1] % 8 == 0
            and w.shape[0] % 8 == 0 and 0 < len(slices) <= 8 and x.numel() > 0):
        return False
    if any(s0 < e1 and s1 < e0 for i, (s0, e0) in enumerate(slices) for s1, e1 in slices[:i]):
        return False
    return all(s % 8 == 0 and e % 8 == 0 and s < e and A.dtype == B.dtype == torch.bfloat16 and A.is_contiguous()
               and B.is_contiguous() and A.shape[0] % 8 == 0 and A.shape == (B.shape[1], x.shape[-1])
               and B.shape[0] == e - s for (s, e), A, B in zip(slices, a, b))


def _pack(a, b, slices, out_features: int):
    """(Acat [R, in], Bcat [out, R])."""
    global _launches
    if len(a) == 1 and slices[0] == (0, out_features):
        return a[0], b[0]
    n, fin = len(a), a[0].shape[1]
    ranks = [t.shape[0] for t in a]
    acat = torch.empty((sum(ranks), fin), device=a[0].device, dtype=torch.bfloat16)
    bcat = torch.empty((out_features, sum(ranks)), device=a[0].device, dtype=torch.bfloat16)
    ints = ctypes.c_int * n
    ptrs = ctypes.c_void_p * n
    _lib.check(_lib.cuda_lib().xb_lora_pack(
        ptrs(*[t.data_ptr() for t in a]), ptrs(*[t.data_ptr() for t in b]), ints(*ranks),
        ints(*[s for s, _ in slices]), ints(*[e for _, e in slices]), n, acat.data_ptr(), bcat.data_ptr(), fin,
        out_features, _lib.stream_ptr()), "xb_lora_pack")
    _launches += 1
    return acat, bcat


def gemm_sum(x, w, x2, w2, b_mn: bool = False):
    """``x @ op(w)^T + x2 @ op(w2)^T`` in bf16 with one rounding.  Below 384 rows, where the pair kernel has
    too few tiles, the second product is added to the first one's result."""
    global _launches
    M, K = x.shape
    N = w.shape[1] if b_mn else w.shape[0]
    if M < 384 and not gemm_ops._BATCH_INVARIANT or gemm_ops._VARIANT != "pair":
        return gemm(x2, w2, b_mn=b_mn, out=gemm(x, w, b_mn=b_mn), accumulate=True)
    x, x2, w, w2 = (t if t.stride(1) == 1 and t.stride(0) % 8 == 0 and t.data_ptr() % 16 == 0 else t.contiguous()
                    for t in (x, x2, w, w2))
    out = torch.empty((M, N), device=x.device, dtype=torch.bfloat16)
    _lib.check(_lib.cuda_lib().xb_gemm_bf16_pair_ext(
        x.data_ptr(), w.data_ptr(), x2.data_ptr(), w2.data_ptr(), out.data_ptr(), M, N, K, x2.shape[1], x.stride(0),
        w.stride(0), x2.stride(0), w2.stride(0), out.stride(0), int(b_mn), _lib.stream_ptr()), "xb_gemm_bf16_pair_ext")
    _launches += 1
    return out


class _LoraLinear(torch.autograd.Function):
    """Weights and factors are kept on ctx as plain attributes: ZeRO-3 fills their buffers again before the
    backward."""

    @staticmethod
    def forward(ctx, x, w, scaling, slices, *factors):
        a, b = factors[0::2], factors[1::2]
        x2 = x.reshape(-1, x.shape[-1])
        if not x2.is_contiguous():
            x2 = x2.contiguous()
        acat, bcat = _pack(a, b, slices, w.shape[0])
        d = gemm(x2, acat)
        if scaling != 1.0:
            d = d * scaling
        ctx.save_for_backward(x2, d)
        ctx.x_shape, ctx.w, ctx.scaling, ctx.slices, ctx.factors = x.shape, w, scaling, slices, factors
        return gemm_sum(x2, w, d, bcat).reshape(*x.shape[:-1], w.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x2, d = ctx.saved_tensors
        w, slices = ctx.w, ctx.slices
        a, b = ctx.factors[0::2], ctx.factors[1::2]
        need = ctx.needs_input_grad
        dy2 = dy.reshape(-1, dy.shape[-1])
        if not dy2.is_contiguous():
            dy2 = dy2.contiguous()
        dw = weight_grad(dy2, x2, w) if need[1] else None
        acat, bcat = _pack(a, b, slices, w.shape[0])
        dd = gemm(dy2, bcat, b_mn=True)
        if ctx.scaling != 1.0:
            dd = dd * ctx.scaling
        grads = []
        ga = None
        if any(need[4::2]) and current_wgrad_store() is None:
            ga = gemm(dd, x2, a_mn=True, b_mn=True, out_dtype=torch.float32)       # all slices at once
        r0 = 0
        for i, ((s, e), A, B) in enumerate(zip(slices, a, b)):
            r1 = r0 + A.shape[0]
            gA = gB = None
            if need[4 + 2 * i]:
                gA = deliver_param_grad(A, ga[r0:r1]) if ga is not None else weight_grad(dd[:, r0:r1], x2, A)
            if need[5 + 2 * i]:
                gB = weight_grad(dy2[:, s:e], d[:, r0:r1], B)
            grads += [gA, gB]
            r0 = r1
        dx = gemm_sum(dy2, w, dd, acat, b_mn=True).reshape(ctx.x_shape) if need[0] else None
        return (dx, dw, None, None, *grads)


def lora_linear(x, w, scaling: float, slices, a, b) -> torch.Tensor:
    """``slices``: tuple of (first, one past last) output row of every adapter; ``a`` [r, in], ``b`` [rows, r]."""
    factors = [t for pair in zip(a, b) for t in pair]
    return _lib.apply(_LoraLinear, x, w, float(scaling), tuple(slices), *factors)
