"""Dense GEMM entry points and the ``linear`` autograd op built on them.

Three operand layouts cover forward, dgrad and wgrad of ``y = x @ Wᵀ``
(``nn.Linear`` everywhere in the reference, e.g. `lit_gpt/attention.py:42-48`,
`lit_gpt/model.py:636-637`):

* ``matmul_nt(a[M,K], b[N,K])  = a @ bᵀ``  (forward; both operands K-major)
* ``matmul_nn(a[M,K], b[K,N])  = a @ b``   (dgrad; B is N-major)
* ``matmul_tn(a[K,M], b[K,N])  = aᵀ @ b``  (wgrad; both operands MN-major)

CUDA path: ``csrc/gemm2_bf16.cu`` by default — SM pairs (``cta_group::2``) share one 256×256
output tile: each CTA loads its half of both operands with TMA, the leader's elected thread
issues ``tcgen05.mma`` for the pair into double-buffered TMEM accumulators, epilogue warps of
both CTAs drain their 128 rows with ``tcgen05.ld``.  ``csrc/gemm_bf16.cu`` is the one-CTA
kernel of the same structure (128×256 tiles), kept for shapes the pair kernel does not take and
selectable with ``ARCHSCALE_B200_GEMM=1cta``.  All three layouts run the same kernels with
different TMA boxes and UMMA descriptor major-ness.
"""
from __future__ import annotations

import functools
import os
from typing import Optional

import torch
from torch.nn.modules.module import _has_any_global_hook

from . import backend


def _operands_ok(a: torch.Tensor, b: torch.Tensor) -> bool:
    return (a.dtype == torch.bfloat16 and b.dtype == torch.bfloat16 and a.dim() == 2 and b.dim() == 2
            and a.stride(-1) == 1 and b.stride(-1) == 1
            and a.stride(0) % 8 == 0 and b.stride(0) % 8 == 0
            and a.data_ptr() % 16 == 0 and b.data_ptr() % 16 == 0)


def _cuda_ok(a: torch.Tensor, b: torch.Tensor, M: int, N: int, K: int) -> bool:
    """Operands of ``y[M,N]`` with K products each: feature counts N and K multiples of 8 (rows of 16-byte multiples), any number
    of rows (tokens) M.  Whole training steps, ms, token counts that are no multiple of 8 through the library (whose weight
    gradient is a bf16 tensor to be added to the fp32 buffer, and which leaves SwiGLU to a kernel of its own) / through the own
    GEMM: dense 8 layers 1001 tokens 13.6 / 11.5, 4001 13.7 / 12.2, 16385 38.5 / 38.5; dense 16 layers 8191 92.9 / 88.5; hybrids of
    16 layers 2001 to 8193 tokens 69.3 / 64.8 to 104.8 / 100.5."""
    return K % 8 == 0 and N % 8 == 0 and K >= 64 and M >= 1 and _operands_ok(a, b)


def _cuda_ok_tn(a: torch.Tensor, b: torch.Tensor, M: int, N: int, K: int) -> bool:
    """The same for a weight gradient, whose K is the number of rows (tokens)."""
    return M % 8 == 0 and N % 8 == 0 and K >= 64 and M >= 1 and _operands_ok(a, b)


def bias_row(bias: torch.Tensor) -> torch.Tensor:
    """``bias`` as the GEMM epilogue reads it: dense bf16 on a 16-byte boundary."""
    bias = bias.to(torch.bfloat16).contiguous()
    return bias if bias.data_ptr() % 16 == 0 else bias.clone()


def matmul_nt(a: torch.Tensor, b: torch.Tensor, out_dtype: Optional[torch.dtype] = None, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """a:(M,K) b:(N,K) → a @ bᵀ : (M,N); ``bias`` (N,) (bf16 result) is added to the sums before they are rounded."""
    M, K = a.shape
    N = b.shape[0]
    if bias is not None:
        if _cuda_ok(a, b, M, N, K) and backend.use_cuda_kernel("gemm", a, b, bias):
            backend.count_launch()
            return backend.require_extension().gemm_bf16_bias(a, b, bias_row(bias))
        return torch.nn.functional.linear(a, b, bias.to(a.dtype))
    if _cuda_ok(a, b, M, N, K) and backend.use_cuda_kernel("gemm", a, b):
        backend.count_launch()
        return backend.require_extension().gemm_bf16(a, b, 0, out_dtype or torch.bfloat16, None)
    out = a @ b.t()
    return out if out_dtype is None else out.to(out_dtype)


def matmul_nn(a: torch.Tensor, b: torch.Tensor, out_dtype: Optional[torch.dtype] = None) -> torch.Tensor:
    """a:(M,K) b:(K,N) → a @ b : (M,N)."""
    M, K = a.shape
    N = b.shape[1]
    if _cuda_ok(a, b, M, N, K) and backend.use_cuda_kernel("gemm", a, b):
        backend.count_launch()
        return backend.require_extension().gemm_bf16(a, b, 1, out_dtype or torch.bfloat16, None)
    out = a @ b
    return out if out_dtype is None else out.to(out_dtype)


def matmul_tn(a: torch.Tensor, b: torch.Tensor, out_dtype: Optional[torch.dtype] = None) -> torch.Tensor:
    """a:(K,M) b:(K,N) → aᵀ @ b : (M,N)."""
    K, M = a.shape
    N = b.shape[1]
    if _cuda_ok_tn(a, b, M, N, K) and backend.use_cuda_kernel("gemm", a, b):
        backend.count_launch()
        return backend.require_extension().gemm_bf16(a, b, 2, out_dtype or torch.bfloat16, None)
    out = a.t() @ b
    return out if out_dtype is None else out.to(out_dtype)


def matmul_tn_acc_(c: torch.Tensor, a: torch.Tensor, b: torch.Tensor) -> torch.Tensor:
    """c (fp32, (M,N)) += aᵀ @ b with a:(K,M), b:(K,N)."""
    K, M = a.shape
    N = b.shape[1]
    if c.dtype == torch.float32 and c.is_contiguous() and _cuda_ok_tn(a, b, M, N, K) and backend.use_cuda_kernel("gemm", a, b, c):
        backend.count_launch()
        backend.require_extension().gemm_bf16(a, b, 2, torch.float32, c)
        return c
    if a.is_cuda:
        c.add_((a.t() @ b).to(c.dtype))
    else:
        c.add_(a.float().t() @ b.float())
    return c


class _LinearFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, bias):
        ctx.save_for_backward(x, weight)
        ctx.has_bias = bias is not None
        ctx.weight_ref = weight            # to find ``main_grad`` (fp32 flat-buffer view) in backward
        x2 = x.reshape(-1, x.shape[-1])
        g = getattr(weight, "_fsdp_group", None)
        if g is not None and getattr(g, "ag_pending", False):
            eng = weight._fsdp_engine
            if weight._fsdp_first and x2.shape[0] % 8 == 0 and _cuda_ok(x2, weight, x2.shape[0], weight.shape[0], x2.shape[1]):
                # FSDP forward: this GEMM also gathers the unit's matrix parameters from all ranks
                g.ag_pending = False
                y = eng.symm.ag_gemm(x2, g, weight.shape[0], bias=None if bias is None else bias_row(bias))
            else:
                eng.finish_pending_gather(g)
                y = matmul_nt(x2, weight, bias=bias)
        else:
            y = matmul_nt(x2, weight, bias=bias)
        return y.view(*x.shape[:-1], weight.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x, weight = ctx.saved_tensors
        dy2 = dy.reshape(-1, dy.shape[-1])
        main_grad = getattr(ctx.weight_ref, "main_grad", None)
        if torch.is_grad_enabled() and main_grad is None:                    # create_graph: the kernels have no backward of their own
            return (dy @ weight, dy2.t() @ x.reshape(-1, x.shape[-1]), dy2.float().sum(0).to(dy.dtype) if ctx.has_bias else None)
        if not dy2.is_contiguous():
            dy2 = dy2.contiguous()
        x2 = x.reshape(-1, x.shape[-1])
        dx = dw = db = None
        if ctx.needs_input_grad[0]:
            dx = matmul_nn(dy2, weight).view(x.shape)
        if ctx.needs_input_grad[1]:
            if main_grad is not None:
                matmul_tn_acc_(main_grad, dy2, x2)      # wgrad accumulates straight into fp32
            else:
                dw = matmul_tn(dy2, x2)
        if ctx.has_bias and ctx.needs_input_grad[2]:
            db = dy2.float().sum(0).to(dy.dtype)
        return dx, dw, db


class _LinearSwiGLUFn(torch.autograd.Function):
    """``silu(x·W_gateᵀ) ∘ (x·W_upᵀ)`` with the activation computed in the GEMM epilogue (``W = [gate rows | up rows]``).
    The pre-activation is written only when a backward pass will read it; the forward pass never reads it back."""

    @staticmethod
    def forward(ctx, x, weight, keep_h):
        x2 = x.reshape(-1, x.shape[-1])
        h, act = backend.require_extension().gemm_swiglu(x2, weight, keep_h)
        backend.count_launch()
        ctx.save_for_backward(x, weight, h)
        ctx.weight_ref = weight
        return act.view(*x.shape[:-1], weight.shape[0] // 2)

    @staticmethod
    def backward(ctx, dact):
        x, weight, h = ctx.saved_tensors
        da2 = dact.reshape(-1, dact.shape[-1])
        if not da2.is_contiguous():
            da2 = da2.contiguous()
        dh = backend.require_extension().swiglu_packed_bwd(h, da2)
        backend.count_launch()
        x2 = x.reshape(-1, x.shape[-1])
        dx = dw = None
        if ctx.needs_input_grad[0]:
            dx = matmul_nn(dh, weight).view(x.shape)
        if ctx.needs_input_grad[1]:
            main_grad = getattr(ctx.weight_ref, "main_grad", None)
            if main_grad is not None:
                matmul_tn_acc_(main_grad, dh, x2)
            else:
                dw = matmul_tn(dh, x2)
        return dx, dw, None


def fused_swiglu_enabled() -> bool:
    """SwiGLU in the epilogue of the SM-pair GEMM (off with ``ARCHSCALE_B200_FUSED_SWIGLU=0`` or the one-CTA GEMM)."""
    return (os.environ.get("ARCHSCALE_B200_FUSED_SWIGLU", "1") != "0" and os.environ.get("ARCHSCALE_B200_GEMM", "") != "1cta"
            and backend.has("gemm_swiglu"))


SKINNY_ROWS = 64


@functools.lru_cache(maxsize=None)
def _one_cta() -> bool:
    """``ARCHSCALE_B200_GEMM=1cta``: every product on the one-CTA GEMM, those of few rows too."""
    return os.environ.get("ARCHSCALE_B200_GEMM", "") == "1cta"


def _skinny_ok(x: torch.Tensor, ws) -> bool:
    """Whether the kernel for few rows (``csrc/gemm_skinny.cu``) takes ``x @ [w₀; w₁; …]ᵀ``: no gradients, at most 64 rows (one
    block of its tokens), dense bf16 rows that the TMA can read (16-byte base, widths that are multiples of 8)."""
    K = x.shape[-1]
    if not (x.is_cuda and x.dtype == torch.bfloat16 and 0 < x.numel() <= SKINNY_ROWS * K and K % 8 == 0 and backend.plain_call()
            and x.is_contiguous() and x.data_ptr() % 16 == 0 and not _one_cta() and backend.has("gemm_skinny")):
        return False
    for w in ws:
        if not (w.is_cuda and w.dtype == torch.bfloat16 and w.dim() == 2 and w.shape[0] % 8 == 0 and w.shape[0] > 0 and w.stride(1) == 1
                and w.stride(0) % 8 == 0 and w.stride(0) >= K and w.data_ptr() % 16 == 0):
            return False
        g = getattr(w, "_fsdp_group", None)
        if g is not None and getattr(g, "ag_pending", False):
            return False
    return backend.use_cuda_kernel("gemm", x, *ws)


def _skinny(x: torch.Tensor, ws, swiglu: bool) -> torch.Tensor:
    y = backend.require_extension().gemm_skinny(x.view(-1, x.shape[-1]), ws, swiglu)
    backend.count_launch()
    return y.view(*x.shape[:-1], y.shape[-1])


def linear_swiglu(x: torch.Tensor, weight: torch.Tensor) -> Optional[torch.Tensor]:
    """SwiGLU of ``x @ weightᵀ`` (gate = first half of the output features) in one GEMM launch, or ``None`` when the
    fused kernel does not take this case (the caller then runs ``linear`` + ``swiglu_packed``).

    Token counts that are no multiple of 8 take it without gradients too (unlike single products, see :func:`linear`): one launch
    instead of two.  Whole forward passes, launched one by one, ms, library and activation / fused: dense 8 layers 67 tokens 2.20 / 2.05,
    257 2.20 / 2.05.  In a graph, where only device time counts, the fused kernel's 256-row tiles lose below some 800 tokens: 67 0.428 /
    0.456, 257 0.484 / 0.505, 777 0.649 / 0.673, 1001 0.716 / 0.720; 16 layers 257 1.361 / 1.504, 513 1.753 / 1.755, 1001 2.196 / 2.119."""
    if weight.shape[0] % 16 == 0 and _skinny_ok(x, (weight,)) and fused_swiglu_enabled():
        return _skinny(x, [weight], True)
    if not (x.is_cuda and x.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16 and weight.dim() == 2
            and weight.shape[0] % 16 == 0 and x.shape[-1] % 8 == 0 and x.shape[-1] >= 64 and x.numel() > 0
            and weight.stride(-1) == 1 and weight.stride(0) % 8 == 0
            and not backend.transformed() and weight.data_ptr() % 16 == 0 and (x.data_ptr() % 16 == 0 or not x.is_contiguous())
            and fused_swiglu_enabled() and backend.use_cuda_kernel("gemm", x, weight)):
        return None
    g = getattr(weight, "_fsdp_group", None)
    if g is not None and getattr(g, "ag_pending", False):
        return None                                     # this GEMM carries the unit's fused all-gather: keep that path
    if not x.is_contiguous():
        x = x.contiguous()
    return backend.apply(_LinearSwiGLUFn, x, weight, torch.is_grad_enabled() and (x.requires_grad or weight.requires_grad))


def linear(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``x @ weightᵀ + bias``; bf16 CUDA inputs run the tcgen05 kernel for fwd, dgrad and wgrad.

    Without gradients, token counts beyond 64 that are no multiple of 8 stay with the library: the own GEMM's gain at such counts lies in
    the backward pass.  µs of one product in a graph, library / own: 1024x1024 at 65 tokens 5.0 / 9.8, 1001 5.2 / 11.0, 4001 9.1 / 11.8,
    16383 26.0 / 28.5; 5632x1024 at 257 6.8 / 11.2, 1001 12.6 / 16.2, 4001 37.1 / 34.9, 8191 69.5 / 68.8; 2048x2048 at 1001 9.3 / 15.7, 16383
    91.7 / 96.0; host 11 / 15.

    Functorch transforms, forward-mode differentiation and traces see the library's operator at every token count, and a backward pass
    that is itself recorded (``create_graph``) is made of differentiable operators.

    A bias is added to the fp32 sums, before the one rounding to bf16, on either route: added to a rounded product, a bias below half a
    unit in the last place is lost."""
    if bias is None and _skinny_ok(x, (weight,)):
        return _skinny(x, [weight], False)
    if (x.is_cuda and x.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16
            and x.shape[-1] % 8 == 0 and weight.shape[0] % 8 == 0 and x.shape[-1] >= 64 and x.numel() > 0
            and ((x.numel() // x.shape[-1]) % 8 == 0 or not backend.plain_call()) and not backend.transformed()
            and backend.use_cuda_kernel("gemm", x, weight)):
        if not x.is_contiguous():
            x = x.contiguous()
        return backend.apply(_LinearFn, x, weight, bias)
    g = getattr(weight, "_fsdp_group", None)
    if g is not None and getattr(g, "ag_pending", False):
        weight._fsdp_engine.finish_pending_gather(g)
    if weight.dtype != x.dtype:
        weight = weight.to(x.dtype)
        bias = bias.to(x.dtype) if bias is not None else None
    return torch.nn.functional.linear(x, weight, bias)


def widened_ok(x: torch.Tensor, weight: torch.Tensor) -> bool:
    """Whether :func:`linear_widened` pays: bf16 on the GPU, a feature count that is no multiple of 8, and enough tokens for the extra
    launches.  x_proj and dt_proj of one layer, forward + backward, ms, library on the unaligned operands / widened: d_model 1984
    0.110 / 0.107 at 1000 tokens, 0.163 / 0.123 at 2048, 0.706 / 0.380 at 16384; d_model 1088 0.080 / 0.086, 0.104 / 0.095,
    0.353 / 0.309."""
    g = getattr(weight, "_fsdp_group", None)
    return (x.is_cuda and x.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16
            and (x.shape[-1] % 8 != 0 or weight.shape[0] % 8 != 0) and x.shape[-1] >= 64 and x.numel() // x.shape[-1] >= 2048
            and not (g is not None and getattr(g, "ag_pending", False)))


def linear_widened(x: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
    """``x @ weightᵀ`` for feature counts that are no multiple of 8 (dt_rank = 124 at 1984 channels): both operands are widened
    with zeros to the next multiple of 8, so that every row of the product and of its two gradients starts on a 16-byte boundary
    (unaligned rows leave the library only its sm_80 kernels with element-wise loads: 4.6 ms of a step with five such layers at
    4 x 4096 tokens).
    The result is a view of the widened product's first columns."""
    k, n = -x.shape[-1] % 8, -weight.shape[0] % 8
    y = linear(torch.nn.functional.pad(x, (0, k)) if k else x, torch.nn.functional.pad(weight, (0, k, 0, n)))
    return y[..., :weight.shape[0]] if n else y


# ------------------------------------------------------------------------------------------ fused sibling projections
def _adjacent(ts) -> bool:
    """True when the tensors are dense 2-D row blocks stored back to back in one storage (views of one flat parameter buffer).
    Separate tensors can lie back to back too (the allocator cuts large ones from one segment), but no view spans them."""
    for a, b in zip(ts[:-1], ts[1:]):
        if not (a.is_contiguous() and b.is_contiguous() and a.dtype == b.dtype and a.shape[1] == b.shape[1]
                and a.data_ptr() + a.numel() * a.element_size() == b.data_ptr()
                and a.untyped_storage().data_ptr() == b.untyped_storage().data_ptr()):
            return False
    return True


def _cat_view(ts) -> torch.Tensor:
    rows = sum(t.shape[0] for t in ts)
    return ts[0].as_strided((rows, ts[0].shape[1]), (ts[0].shape[1], 1))


class _MultiLinearFn(torch.autograd.Function):
    """y = x @ [W₀; W₁; …]ᵀ for weights stored back to back: one forward GEMM, one dgrad GEMM (no partial-sum adds) and
    one wgrad GEMM that accumulates into the equally adjacent fp32 ``main_grad`` views."""

    @staticmethod
    def forward(ctx, x, *weights):
        w_cat = _cat_view([w.detach() for w in weights])
        x2 = x.reshape(-1, x.shape[-1])
        g = getattr(weights[0], "_fsdp_group", None)
        if g is not None and getattr(g, "ag_pending", False):
            eng = weights[0]._fsdp_engine
            if weights[0]._fsdp_first and x2.shape[0] % 8 == 0 and _cuda_ok(x2, w_cat, x2.shape[0], w_cat.shape[0], x2.shape[1]):
                g.ag_pending = False
                y = eng.symm.ag_gemm(x2, g, w_cat.shape[0])
            else:
                eng.finish_pending_gather(g)
                y = matmul_nt(x2, w_cat)
        else:
            y = matmul_nt(x2, w_cat)
        ctx.save_for_backward(x, w_cat)
        ctx.weights = weights
        return y.view(*x.shape[:-1], w_cat.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x, w_cat = ctx.saved_tensors
        x2, dy2 = x.reshape(-1, x.shape[-1]), dy.reshape(-1, dy.shape[-1])
        mgs = [getattr(w, "main_grad", None) for w in ctx.weights]
        if torch.is_grad_enabled() and all(m is None for m in mgs):          # create_graph: see _LinearFn
            return (dy @ torch.cat(ctx.weights), *(dy2.t() @ x2).split([w.shape[0] for w in ctx.weights]))
        if not dy2.is_contiguous():
            dy2 = dy2.contiguous()
        dx = matmul_nn(dy2, w_cat).view(*dy.shape[:-1], x2.shape[1]) if ctx.needs_input_grad[0] else None
        if all(m is not None for m in mgs) and _adjacent(mgs):
            matmul_tn_acc_(_cat_view(mgs), dy2, x2)
            return (dx,) + (None,) * len(ctx.weights)
        dw = matmul_tn(dy2, x2)
        outs, r = [], 0
        for w, m in zip(ctx.weights, mgs):
            piece = dw[r:r + w.shape[0]]
            r += w.shape[0]
            if m is not None:
                m.add_(piece.float())
                outs.append(None)
            else:
                outs.append(piece)
        return (dx,) + tuple(outs)


def plain_linear(l) -> bool:
    """True when a call of the layer ``l`` is the product with its weight and nothing else, so that a fused route may pass the
    module by: a ``Linear`` without bias or low-precision operands, hooks, or another ``forward`` than its own."""
    cls, d = type(l), l.__dict__
    return (cls.__name__ == "Linear" and cls.forward is getattr(cls, "plain_forward", None) and "forward" not in d
            and d["_parameters"].get("bias") is None and not l.mxfp8 and not l.nvfp4
            and not (d["_forward_hooks"] or d["_forward_pre_hooks"] or d["_backward_hooks"] or d["_backward_pre_hooks"])
            and l._compiled_call_impl is None and not _has_any_global_hook())


def linear_multi(x: torch.Tensor, layers, keep_fused: bool = False):
    """Outputs of several ``Linear`` layers that share the input ``x``.  When all are :func:`plain_linear` and their weights sit back to
    back in memory (consecutive views of the flat parameter buffer) the layers run as one GEMM and the outputs are column
    slices of its result; otherwise each layer is called on its own.  ``keep_fused``: return the one GEMM's result unsplit
    (a tensor instead of a list) when the layers did run as one GEMM."""
    if not all(plain_linear(l) for l in layers):
        return [l(x) for l in layers]
    ws = [l.weight for l in layers]
    if len(ws) <= 3 and _skinny_ok(x, ws):
        y = _skinny(x, ws, False)                       # the weights need not be neighbours here
        return y if keep_fused else list(y.split([w.shape[0] for w in ws], dim=-1))
    fusable = (x.is_cuda and x.dtype == torch.bfloat16 and not backend.transformed() and all(w.dtype == torch.bfloat16 for w in ws)
               and _adjacent(ws) and x.numel() > 0 and x.shape[-1] % 8 == 0 and x.shape[-1] >= 64
               and backend.use_cuda_kernel("gemm", x, ws[0]))
    if not fusable:
        return [l(x) for l in layers]
    y = backend.apply(_MultiLinearFn, x if x.is_contiguous() else x.contiguous(), *ws)
    if keep_fused:
        return y
    return list(y.split([w.shape[0] for w in ws], dim=-1))
