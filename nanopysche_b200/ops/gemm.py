"""GEMM ops: the tcgen05 bf16 GEMM (csrc/gemm_sm100.cu) on CUDA tensors, torch.matmul on CPU.

``gemm`` is the raw entry: ``C[M, N] (+)= alpha * sum_k A(m, k) * B(n, k)`` where each operand is
either K-major (``[rows, K]`` row-major, ``*_mn=False``) or MN-major (``[K, rows]`` row-major).
That single contraction covers forward (``x @ w.T``), dgrad (``dy @ w``: B MN-major) and wgrad
(``dy.T @ x``: both MN-major) without materialising a transpose.

``linear`` is the autograd function used by the model layers in place of ``nn.functional.linear``
(reference: model/attention.py:141-143,189; model/feed_forward.py:75). When the weight carries a
``main_grad`` buffer (the flat fp32 gradient arena of ``optim.arena``), the wgrad GEMM accumulates
straight into it from TMEM and autograd sees no weight gradient at all.
"""
from __future__ import annotations

import ctypes as C

import torch

from . import _lib


def _use_kernel(t: torch.Tensor) -> bool:
    return _lib.on(t)


def gemm_ref(a, b, *, a_mn=False, b_mn=False, out=None, out_dtype=None, accumulate=False, alpha=1.0):
    """PyTorch reference of ``gemm`` (also the CPU path)."""
    A = a.t() if a_mn else a
    B = b if b_mn else b.t()
    res = (A.float() @ B.float()) * alpha
    out_dtype = out_dtype or (out.dtype if out is not None else a.dtype)
    if out is not None:
        if accumulate:
            out.add_(res.to(out.dtype))
        else:
            out.copy_(res.to(out.dtype))
        return out
    return res.to(out_dtype)


def gemm(a: torch.Tensor, b: torch.Tensor, *, a_mn: bool = False, b_mn: bool = False,
         out: torch.Tensor | None = None, out_dtype: torch.dtype | None = None, accumulate: bool = False,
         alpha: float = 1.0, bn: int = 0, max_ctas: int = 0, bias: torch.Tensor | None = None,
         residual: torch.Tensor | None = None, mt: int = 0, split: int = 0, pair_bn: int = 0) -> torch.Tensor:
    """``out[M, N] (+)= alpha * A @ B^T (+ bias) (+ residual)`` in the operand layouts described in the module
    docstring. ``bias [N]`` (fp32) and ``residual [M, N]`` (dtype of ``out``) are added in the GEMM's epilogue."""
    if not _use_kernel(a):
        if bias is None and residual is None:
            return gemm_ref(a, b, a_mn=a_mn, b_mn=b_mn, out=out, out_dtype=out_dtype, accumulate=accumulate,
                            alpha=alpha)
        y = gemm_ref(a, b, a_mn=a_mn, b_mn=b_mn, out_dtype=torch.float32, alpha=alpha)
        if bias is not None:
            y = y + bias.float()
        if residual is not None:
            y = y + residual.float()
        if out is None:
            return y.to(out_dtype or a.dtype)
        out.copy_((y + out.float()) if accumulate else y)
        return out
    # requests; 0 = choose. mt 2: 256 x 256 tiles on pairs of CTAs, split 2 or 4: parts of K there (bn 128: one-CTA tiles),
    # pair_bn 128, 192 or 256: tiles of that many columns on pairs
    return _lib.host().gemm(a, b, a_mn, b_mn, out, out_dtype, accumulate, alpha, bn, max_ctas, bias, residual, mt, split, pair_bn)


def _gemm_args(a, b, a_mn, b_mn, out, out_dtype, accumulate, alpha):
    """Arguments of one product (checked) and its output tensor."""
    assert a.dtype == torch.bfloat16 and b.dtype == torch.bfloat16, "kernel path is bf16"
    assert a.dim() == 2 and b.dim() == 2 and a.stride(1) == 1 and b.stride(1) == 1
    M, K = (a.shape[1], a.shape[0]) if a_mn else (a.shape[0], a.shape[1])
    N, Kb = (b.shape[1], b.shape[0]) if b_mn else (b.shape[0], b.shape[1])
    assert K == Kb, f"contraction mismatch {K} vs {Kb}"
    if out is None:
        out = torch.empty((M, N), device=a.device, dtype=out_dtype or torch.bfloat16)
    assert out.shape == (M, N) and out.stride(1) == 1
    args = _lib.GemmArgs()
    args.A, args.B, args.C = a.data_ptr(), b.data_ptr(), out.data_ptr()
    args.lda, args.ldb, args.ldc = a.stride(0), b.stride(0), out.stride(0)
    args.a_rows, args.b_rows = a.shape[0], b.shape[0]
    args.M, args.N, args.K = M, N, K
    args.a_mn, args.b_mn = int(a_mn), int(b_mn)
    args.out_f32 = int(out.dtype == torch.float32)
    assert out.dtype in (torch.float32, torch.bfloat16)
    args.accumulate = int(accumulate)
    args.alpha = alpha
    return args, out


def gemm_swiglu(x: torch.Tensor, w_gate: torch.Tensor, w_up: torch.Tensor, *, save_gu: bool = True):
    """``h = silu(x @ w_gate.T) * (x @ w_up.T)`` in one kernel; optionally also returns ``[gate | up]``.

    The B tile of the GEMM is 128 gate rows + 128 up rows, so both pre-activations sit side by side in
    TMEM and the epilogue applies SwiGLU before anything reaches HBM.
    """
    M, K = x.shape
    F = w_gate.shape[0]
    if not _use_kernel(x):
        g = x.float() @ w_gate.float().t()
        u = x.float() @ w_up.float().t()
        h = (torch.nn.functional.silu(g) * u).to(x.dtype)
        return h, (torch.cat([g, u], dim=1).to(x.dtype) if save_gu else None)
    assert x.dtype == w_gate.dtype == w_up.dtype == torch.bfloat16, "kernel path is bf16"
    assert x.stride(1) == 1 and w_gate.stride(1) == 1 and w_gate.stride() == w_up.stride() and w_gate.shape == w_up.shape
    assert w_gate.shape == (F, K), f"contraction mismatch {K} vs {w_gate.shape[1]}"
    h = torch.empty((M, F), device=x.device, dtype=torch.bfloat16)
    gu = torch.empty((M, 2 * F), device=x.device, dtype=torch.bfloat16) if save_gu else None
    args = _lib.GemmArgs()
    args.A, args.B, args.B2, args.C = x.data_ptr(), w_gate.data_ptr(), w_up.data_ptr(), h.data_ptr()
    args.C2 = gu.data_ptr() if gu is not None else None
    args.lda, args.ldb, args.ldc, args.ldc2 = x.stride(0), w_gate.stride(0), F, 2 * F
    args.a_rows, args.b_rows = M, F
    args.M, args.N, args.K = M, F, K
    args.epilogue = 1
    args.alpha = 1.0
    _lib.check(_lib.lib().np_gemm_bf16(C.byref(args), C.c_void_p(_lib.stream())), "gemm_swiglu")
    return h, gu


def _glu_bwd_args(dy, w2, gu, round_dh):
    M, F = dy.shape[0], w2.shape[1]
    assert dy.dtype == w2.dtype == gu.dtype == torch.bfloat16, "kernel path is bf16"
    assert dy.shape[1] == w2.shape[0] and gu.shape == (M, 2 * F) and dy.stride(1) == w2.stride(1) == gu.stride(1) == 1
    out = torch.empty((M, 2 * F), device=dy.device, dtype=torch.bfloat16)
    args = _lib.GemmArgs()
    args.A, args.B, args.C, args.C2 = dy.data_ptr(), w2.data_ptr(), out.data_ptr(), gu.data_ptr()
    args.lda, args.ldb, args.ldc, args.ldc2 = dy.stride(0), w2.stride(0), 2 * F, gu.stride(0)
    args.a_rows, args.b_rows = M, w2.shape[0]
    args.M, args.N, args.K = M, F, dy.shape[1]
    args.b_mn, args.epilogue, args.alpha, args.round_acc = 1, 2, 1.0, int(round_dh)
    return args, out


def gemm_glu_bwd(dy: torch.Tensor, w2: torch.Tensor, gu: torch.Tensor, pair_bn: int = 0, round_dh: bool = False) -> torch.Tensor:
    """``[d gate | d up]`` of ``h = silu(gate) * up`` for ``dh = dy @ w2`` and ``gu = [gate | up]``, without forming ``dh``:
    the gradient of the activation is the epilogue of the GEMM (``dy [M, D]``, ``w2 [D, F]``, ``gu [M, 2F]``). ``round_dh``: the
    gradient of ``dh`` rounded to bf16, bit for bit what two products and a pass over ``dh`` give."""
    if not _use_kernel(dy):
        from .activation import glu_bwd

        dh = gemm_ref(dy, w2, b_mn=True)
        return glu_bwd(gu, dh.to(dy.dtype) if round_dh else dh)
    args, out = _glu_bwd_args(dy, w2, gu, round_dh)
    args.pair_bn = pair_bn
    _lib.check(_lib.lib().np_gemm_bf16(C.byref(args), C.c_void_p(_lib.stream())), "gemm_glu_bwd")
    return out


def gemm_dgrad_wgrad(dy: torch.Tensor, w: torch.Tensor, x: torch.Tensor, *, out: torch.Tensor | None = None,
                     accumulate: bool = False, gu: torch.Tensor | None = None, pair_bn: int = 0, mt: int = 0,
                     round_dh: bool = False):
    """``(dy @ w, dy.T @ x)`` for ``dy [M, N]``, ``w [N, K]``, ``x [M, K]``: the two gradients of a linear layer, in one launch
    where that is expected to be faster than two. The second goes to ``out`` (added with ``accumulate``), by default a new
    tensor in the dtype of ``w``. ``gu``: pre-activations ``[gate | up]`` with ``x = silu(gate) * up``; the first result is then
    ``[d gate | d up]`` (``gemm_glu_bwd``, with ``round_dh``). ``pair_bn`` and ``mt`` ask for one launch with tiles of that
    many columns, two launches."""
    if not _use_kernel(dy):
        dx = gemm(dy, w, b_mn=True) if gu is None else gemm_glu_bwd(dy, w, gu, round_dh=round_dh)
        return dx, gemm(dy, x, a_mn=True, b_mn=True, out=out, out_dtype=w.dtype if out is None else None, accumulate=accumulate)
    a0, dx = _gemm_args(dy, w, False, True, None, None, False, 1.0) if gu is None else _glu_bwd_args(dy, w, gu, round_dh)
    a1, dw = _gemm_args(dy, x, True, True, out, w.dtype, accumulate, 1.0)
    a0.pair_bn, a0.mt = pair_bn, mt
    rc = _lib.lib().np_gemm_bf16_two(C.byref(a0), C.byref(a1), C.c_void_p(_lib.stream()))
    if rc != 0:
        raise _lib.KernelError(f"gemm_bf16_two failed with code {rc}: dy={tuple(dy.shape)}/{dy.stride()} w={tuple(w.shape)}/"
                               f"{w.stride()} x={tuple(x.shape)}/{x.stride()} dw={tuple(dw.shape)}/{dw.stride()} {dw.dtype} "
                               f"ptrs={dy.data_ptr() % 256},{w.data_ptr() % 256},{x.data_ptr() % 256},{dw.data_ptr() % 256}")
    _lib.check(rc, "gemm_bf16_two")
    return dx, dw


# Zero-bubble pipeline schedules split a backward pass into B (input gradients, on the critical path between
# stages) and W (weight gradients, moved into what would be bubbles). While ``_DEFER`` is a list, every weight-gradient
# GEMM is queued there instead of run; ``run_deferred_wgrads`` executes a queue later. ``SPLIT_MODE`` makes ``linear``
# take its autograd function on every device (CPU included), so that all linear weight gradients are deferrable.
_DEFER: "list | None" = None
SPLIT_MODE = False


class defer_wgrad:
    """Context manager: weight-gradient GEMMs issued inside are appended to ``queue`` as ``(w, dy, x)``."""

    def __init__(self, queue: list):
        self.queue, self._prev = queue, None

    def __enter__(self):
        global _DEFER
        self._prev, _DEFER = _DEFER, self.queue
        return self.queue

    def __exit__(self, *exc):
        global _DEFER
        _DEFER = self._prev
        return False


def run_deferred_wgrads(queue: list) -> None:
    """The W step: run the queued weight-gradient GEMMs (into ``main_grad`` when the weight has one, else into
    ``.grad``) and release the saved activations."""
    with torch.no_grad():      # like the backward pass these GEMMs were taken out of: nothing here is differentiated
        while queue:
            w, dy2, x2 = queue.pop(0)
            g = _wgrad_into(w, dy2, x2)
            if g is not None:
                g = g.to(w.dtype)
                w.grad = g if w.grad is None else w.grad + g


def _deferred(w: torch.Tensor) -> bool:
    return _DEFER is not None and (w.is_leaf or hasattr(w, "main_grad"))


def _main_grad_done(w: torch.Tensor) -> None:
    """``w.main_grad`` has its gradient: the next one is added, and whoever waits for it is told."""
    w._main_grad_dirty = True
    for q in getattr(w, "_covers", None) or (w,):  # a fused view stands for several parameters
        q._main_grad_dirty = True
        cb = getattr(q, "_grad_ready_cb", None)      # the arena's overlapped gradient reduction (optim/arena.py)
        if cb is not None:
            cb(q)


def _wgrad_into(w: torch.Tensor, dy2: torch.Tensor, x2: torch.Tensor):
    """dW[N, K] = dy^T x, accumulated into ``w.main_grad`` when present; returns the autograd grad."""
    if _deferred(w):
        # a weight that is itself computed (two parameters concatenated for one GEMM) has no ``.grad`` to fill later:
        # its gradient has to go back through autograd now, so only leaves and arena views are deferred
        _DEFER.append((w, dy2, x2))
        return None
    mg = getattr(w, "main_grad", None)
    if mg is not None:
        first = not getattr(w, "_main_grad_dirty", False)
        gemm(dy2, x2, a_mn=True, b_mn=True, out=mg, accumulate=not first)
        _main_grad_done(w)
        return None
    return gemm(dy2, x2, a_mn=True, b_mn=True, out_dtype=w.dtype if w.is_cuda else None)


def _both_grads(w: torch.Tensor, dy2: torch.Tensor, x2: torch.Tensor, gu: torch.Tensor | None = None, round_dh: bool = False):
    """Input gradient (with ``gu``: the gradient of its pre-activations) and what ``_wgrad_into`` returns for ``w``."""
    if not _use_kernel(dy2) or _deferred(w):
        dx = gemm(dy2, w, b_mn=True) if gu is None else gemm_glu_bwd(dy2, w, gu, round_dh=round_dh)
        return dx, _wgrad_into(w, dy2, x2)
    mg = getattr(w, "main_grad", None)
    if mg is None:
        return gemm_dgrad_wgrad(dy2, w, x2, gu=gu, round_dh=round_dh)
    dx, _ = gemm_dgrad_wgrad(dy2, w, x2, out=mg, accumulate=getattr(w, "_main_grad_dirty", False), gu=gu, round_dh=round_dh)
    _main_grad_done(w)
    return dx, None


def _linear_grads(ctx, w: torch.Tensor, dy2: torch.Tensor, x2: torch.Tensor):
    """``(dx, dw)`` of ``x2 @ w.T`` as far as they are asked for (inputs 0 and 1 of the autograd function)."""
    want_dw = ctx.needs_input_grad[1] or hasattr(w, "main_grad")
    if ctx.needs_input_grad[0] and want_dw:
        return _both_grads(w, dy2, x2)
    return (gemm(dy2, w, b_mn=True) if ctx.needs_input_grad[0] else None), (_wgrad_into(w, dy2, x2) if want_dw else None)


class _Linear(torch.autograd.Function):
    """``x @ w.T`` off the kernel path with a weight gradient that can be deferred (on it: ``Linear`` in csrc/host.cpp)."""

    @staticmethod
    def forward(ctx, x, w):
        ctx.save_for_backward(x, w)
        x2 = x.reshape(-1, x.shape[-1])
        y = gemm(x2, w)
        return y.reshape(*x.shape[:-1], w.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x, w = ctx.saved_tensors
        dy2 = dy.reshape(-1, dy.shape[-1])
        if not dy2.is_contiguous():
            dy2 = dy2.contiguous()
        dx, dw = _linear_grads(ctx, w, dy2, x.reshape(-1, x.shape[-1]))
        return None if dx is None else dx.reshape(x.shape), dw


class _LinearBias(torch.autograd.Function):
    """``x @ w.T + bias`` with the bias added in the GEMM's epilogue."""

    @staticmethod
    def forward(ctx, x, w, bias):
        ctx.save_for_backward(x, w)
        ctx.bias_dtype = bias.dtype
        x2 = x.reshape(-1, x.shape[-1])
        y = gemm(x2, w, bias=bias.detach().float().contiguous())
        return y.reshape(*x.shape[:-1], w.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x, w = ctx.saved_tensors
        dy2 = dy.reshape(-1, dy.shape[-1])
        if not dy2.is_contiguous():
            dy2 = dy2.contiguous()
        dx, dw = _linear_grads(ctx, w, dy2, x.reshape(-1, x.shape[-1]))
        dx = None if dx is None else dx.reshape(x.shape)
        db = dy2.float().sum(0).to(ctx.bias_dtype) if ctx.needs_input_grad[2] else None
        return dx, dw, db


def linear(x: torch.Tensor, w: torch.Tensor, bias: torch.Tensor | None = None) -> torch.Tensor:
    """``x @ w.T (+ bias)``; tcgen05 kernels for bf16 CUDA tensors, ``F.linear`` otherwise."""
    if SPLIT_MODE and not (_lib.on(x) and x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16):
        # same math through the autograd function whose weight gradient can be deferred
        xx = x if x.dtype == w.dtype else x.to(w.dtype)
        return _Linear.apply(xx, w) if bias is None else _LinearBias.apply(xx, w, bias)
    if _lib.on(x) and x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16:
        rt = getattr(w, "_fsdp_rt", None)
        if rt is not None:  # row-sharded weight: all-gather inside the GEMM, reduce-scattered weight gradient
            from .fsdp_fused import sharded_linear

            y = sharded_linear(x, w, rt)
            return y if bias is None else y + bias
        rec = getattr(w, "_fp8_recipe", None)
        if rec is not None:  # weight tagged by fp8.training.apply_fp8: forward GEMM on e4m3 operands
            if rec == "mxfp8":
                from .gemm_mxfp8 import mx_linear, mx_linear_supported

                if mx_linear_supported(x, w):
                    return mx_linear(x, w, bias)
            else:
                from .gemm_fp8 import fp8_block_linear, fp8_block_linear_supported

                if fp8_block_linear_supported(x, w):
                    return fp8_block_linear(x, w, bias)
        if bias is not None:
            return _LinearBias.apply(x, w, bias)
        return _lib.host().linear(x, w)
    return torch.nn.functional.linear(x, w, bias)


class _SwiGLUFeedForward(torch.autograd.Function):
    """``(silu(x @ w1.T) * (x @ w3.T)) @ w2.T`` for a fused ``[w1; w3]`` weight: the activation in the epilogue of the
    gate|up GEMM (which also stores the pre-activations when a backward pass will need them), its gradient in the epilogue
    of the down projection's input-gradient GEMM."""

    @staticmethod
    def forward(ctx, x, w13, w2, save):
        F = w13.shape[0] // 2
        x2 = x.reshape(-1, x.shape[-1])
        h, gu = gemm_swiglu(x2, w13[:F], w13[F:], save_gu=save)
        if save:
            ctx.save_for_backward(x, w13, w2, h, gu)
        return gemm(h, w2).view(*x.shape[:-1], w2.shape[0])

    @staticmethod
    def backward(ctx, dy):
        dx, dw13, dw2 = _feed_forward_grads(ctx, dy)
        return None if dx is None else dx.view(dy.shape[:-1] + dx.shape[-1:]), dw13, dw2, None


def _feed_forward_grads(ctx, dy: torch.Tensor, round_dh: bool = False):
    """``(dx [rows, D], dw13, dw2)`` as far as they are asked for (inputs 0 to 2 of the autograd function, which saved ``x, w13,
    w2, h, gu``). ``round_dh``: as in ``gemm_glu_bwd``."""
    x, w13, w2, h, gu = ctx.saved_tensors
    dy2 = dy.reshape(-1, dy.shape[-1])
    if not dy2.is_contiguous():
        dy2 = dy2.contiguous()
    want_dw2 = ctx.needs_input_grad[2] or hasattr(w2, "main_grad")
    if not (ctx.needs_input_grad[0] or ctx.needs_input_grad[1] or hasattr(w13, "main_grad")):
        return None, None, _wgrad_into(w2, dy2, h) if want_dw2 else None
    if want_dw2:
        dgu, dw2 = _both_grads(w2, dy2, h, gu, round_dh)
    else:
        dgu, dw2 = gemm_glu_bwd(dy2, w2, gu, round_dh=round_dh), None
    return *_linear_grads(ctx, w13, dgu, x.reshape(-1, x.shape[-1])), dw2


def _plain_weight(w: torch.Tensor) -> bool:
    """A bf16 weight that the GEMMs read in place: not row-sharded, not tagged for fp8, 16-byte aligned rows."""
    return (w.dtype == torch.bfloat16 and w.dim() == 2 and w.stride(1) == 1 and w.stride(0) % 8 == 0 and
            w.data_ptr() % 16 == 0 and getattr(w, "_fsdp_rt", None) is None and getattr(w, "_fp8_recipe", None) is None)


def feed_forward_glu(x: torch.Tensor, w13: torch.Tensor, w2: torch.Tensor, act: str = "silu") -> torch.Tensor:
    """``(act(x @ w1.T) * (x @ w3.T)) @ w2.T`` for a fused ``[w1; w3]`` weight. SwiGLU of more rows than the few-row kernel
    takes runs with the activation and its gradient inside the GEMMs (4096 tokens, 2048 x 5632: the separate passes took 34
    and 46 us of the layer's 753); other activations, fp8 or sharded weights take GEMMs and the GLU kernels."""
    from .activation import glu

    if (act == "silu" and not SPLIT_MODE and _lib.on(x) and x.dtype == torch.bfloat16 and x.numel() > 64 * x.shape[-1] and
            w13.shape[0] % 16 == 0 and x.shape[-1] % 8 == 0 and w2.shape[0] % 8 == 0 and _plain_weight(w13) and
            _plain_weight(w2)):
        x2 = x if x.is_contiguous() and x.data_ptr() % 16 == 0 else x.clone(memory_format=torch.contiguous_format)
        save = torch.is_grad_enabled() and (x2.requires_grad or w13.requires_grad or w2.requires_grad)
        return _SwiGLUFeedForward.apply(x2, w13, w2, save)
    if (act == "silu" and not SPLIT_MODE and _lib.on(x) and x.dtype == torch.bfloat16 and x.numel() > 0 and
            getattr(w13, "_fp8_recipe", None) == getattr(w2, "_fp8_recipe", None) == "mxfp8" and
            all(w.is_contiguous() and getattr(w, "_fsdp_rt", None) is None for w in (w13, w2))):
        from .gemm_mxfp8 import _MXFeedForward, mx_linear_supported

        if mx_linear_supported(x, w13) and mx_linear_supported(x, w2):
            save = torch.is_grad_enabled() and (x.requires_grad or w13.requires_grad or w2.requires_grad)
            return _MXFeedForward.apply(x, w13, w2, save)
    return linear(glu(linear(x, w13), act), w2)
