r"""
Gate math: top-k selection with softmax over the selected logits.

Parity: the ``topk`` → ``softmax`` sequence of ``fmoe/gates/naive_gate.py:31-38`` (ATen ops
in the reference).  On a GPU one kernel reads each logits row once, keeps the k largest in
registers, writes ids and probabilities, and a second small kernel applies the softmax
Jacobian in backward and scatters the result into the dense logits gradient.

``linear_topk_softmax`` goes one step further for the plain linear gate
(``fmoe/gates/naive_gate.py:24-38``: ``nn.Linear`` → ``topk`` → ``softmax``): with at most 8
experts one kernel reads the token once, keeps its logits in registers and writes logits, ids
and probabilities, and the backward is three kernels (softmax Jacobian + ``dx``; partial
sums of ``dW`` and ``db``; their merge) instead of the six of the ATen sequence.
"""
import torch
from torch.autograd import Function, forward_ad

from . import grouped_gemm as gg
from . import native

MAX_FUSED_K = 8
MAX_FUSED_EXPERTS = 4096
MAX_SINGLE_PASS_EXPERTS = 8
# Up to here the one-block-per-token kernel is faster than the tensor-core product and the top-k after
# it, which take 11 us or more (64 experts, d 1024: 6.0 us for 64 tokens, 10.0 for 512, 15.8 for 1024; d
# 2048: 17.0 for 512, against 15.6).
MAX_FEW_TOKENS = 512
MAX_FEW_PRODUCTS = 1 << 25


def _topk_softmax_torch(logits, k):
    val, idx = torch.topk(logits, k=k, dim=-1, largest=True, sorted=True)
    return idx, torch.softmax(val, dim=-1)


class _TopkSoftmax(Function):
    @staticmethod
    def forward(ctx, logits, k, zero=None):
        idx, score = native.get().gate_topk_softmax(logits.contiguous(), int(k), zero)
        ctx.save_for_backward(idx, score)
        ctx.shape = logits.shape
        ctx.mark_non_differentiable(idx)
        return idx, score

    @staticmethod
    def backward(ctx, _grad_idx, grad_score):
        idx, score = ctx.saved_tensors
        grad_logits = native.get().gate_topk_softmax_bwd(
            grad_score.contiguous(), idx, score, int(ctx.shape[-1]))
        return grad_logits, None, None


def topk_softmax(logits, k):
    r"""``(idx int64 [B,k], prob [B,k])``: the k largest logits per row (descending) and their softmax."""
    if (logits.is_cuda and k <= MAX_FUSED_K and logits.shape[-1] <= MAX_FUSED_EXPERTS
            and logits.dtype in (torch.float32, torch.bfloat16, torch.float16)):
        return _TopkSoftmax.apply(logits, k)
    return _topk_softmax_torch(logits, k)


class _LinearTopkSoftmax(Function):
    r"""``logits = x W^T + b``, top-k ids and softmax of the selected logits as one op.  The native node of
    the same (``binding.cpp::GateLinearTopk``) takes all calls but those that are traced: a trace records
    a Python function, and nothing of a native one."""

    @staticmethod
    def forward(ctx, x, weight, bias, k):
        # (the kernels load 16 bytes at a time; saved are the inputs, which a gradient of the gradient goes
        # on to, and not copies made here: each where the other's gradient is wanted, as what is not saved
        # may be changed in place)
        logits, idx, prob = native.get().gate_linear_topk(gg.aligned(x, 16), gg.aligned(weight, 16), bias, int(k))
        need_dx, need_dw, need_db = ctx.needs_input_grad[:3]
        ctx.save_for_backward(x if need_dw or need_db else None, weight if need_dx else None, idx, prob)
        ctx.has_bias, ctx.tot = bias is not None, weight.shape[0]
        ctx.mark_non_differentiable(idx)
        ctx.set_materialize_grads(False)
        return logits, idx, prob

    @staticmethod
    def backward(ctx, grad_logits, _grad_idx, grad_prob):
        x, weight, idx, prob = ctx.saved_tensors
        if grad_logits is None and grad_prob is None:
            return None, None, None, None
        need_dx, need_dw, need_db = ctx.needs_input_grad[:3]
        if torch.is_grad_enabled() and prob.dtype == torch.float32:
            # a gradient of the gradient, as in the native node
            dl = grad_logits
            if grad_prob is not None:
                through = native.get().gate_topk_softmax_bwd(grad_prob.contiguous(), idx, prob, ctx.tot)
                dl = through if dl is None else dl + through
            return (dl.matmul(weight) if need_dx else None, dl.t().matmul(x) if need_dw else None,
                    dl.sum(0) if need_db else None, None)
        dx, dw, db, _dl = native.get().gate_linear_topk_bwd(
            None if grad_prob is None else grad_prob.contiguous(), idx, prob,
            None if grad_logits is None else grad_logits.contiguous(), gg.aligned(x, 16), gg.aligned(weight, 16),
            need_dx, need_db, ctx.tot)
        return dx if need_dx else None, dw if need_dw else None, db if need_db else None, None


def _plain(*tensors):
    r"""Whether these are plain tensors: a subclass may want to see the operations."""
    return all(t is None or type(t) in (torch.Tensor, torch.nn.Parameter) for t in tensors)


def _single_pass_type(x, weight, bias):
    r"""Whether the single-pass kernel takes these types: all 16 bits, or all 32 as plain tensors (a linear, top-k,
    softmax and their backward as operations, 8192 tokens, d 1024, 8 experts: 163 us, 87 in the kernels, whose
    logits are within 1.2 units of 2^-24 of 64 bits, weight gradients 2.3, against 5.5 and 4.9)."""
    if weight.dtype != x.dtype or (bias is not None and bias.dtype != x.dtype):
        return False
    if x.dtype in (torch.bfloat16, torch.float16):
        return True
    return x.dtype == torch.float32 and _plain(x, weight, bias)


def _wants_grad(*tensors):
    return torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in tensors)


def _no_tangent(*tensors):
    r"""Whether no forward-mode derivative passes through: the native calls would drop it."""
    return all(t is None or forward_ad.unpack_dual(t).tangent is None for t in tensors)


def _library_linear_better(tokens, d, experts, grads):
    r"""Whether a Switch layer in 16 bits is faster with the library's linear.  The library has tensor-core
    kernels for output rows of a multiple of 16 bytes (8 experts); with others it splits K, is slower and
    rounds twice.  Layers of 8 experts with the kernel / with the linear, us: without gradients d 512: 30.8 / 31.1 at 64
    tokens, 48.6 / 46.7 at 8192; d 1024: 34.9 / 34.5, 64.0 / 60.7; d 4096: 61.8 / 58.3, 150.9 / 135.0, and 4 us of host
    time; a step of d 512: 78.7 / 80.3, 138.3 / 151.3; d 1024: 90.4 / 88.4, 121.7 / 119.7 at 2048 tokens, 171.8 /
    181.5; d 2048: 112.8 / 104.9, 241.3 / 237.4.  (4 experts, d 2048, 64 tokens: 41.4 / 49.8, a step 103.9 / 114.3.)"""
    return experts % 8 == 0 and not (grads and (d <= 512 or (d <= 1024 and tokens >= 4096)))


def linear_logits(x, linear):
    r"""``linear(x)`` of a gate's ``nn.Linear`` in the single-pass kernel, or ``None`` where that does not
    take the call, somebody watches the module or the linear is faster.  It stands for three library products
    and a column sum (a Switch layer's step, 8192 tokens, d 1024, 2 experts: 216 us with those, 193 with this)."""
    from ..transformer import _hooked, _hooked_globally
    if type(linear) is not torch.nn.Linear:   # the user's own module (a quantised one, an adapter)
        return None
    w, b = linear.weight, linear.bias
    if (w.shape[0] <= MAX_SINGLE_PASS_EXPERTS and x.is_cuda and x.dim() == 2 and x.is_contiguous()
            and x.shape[0] > 0 and _single_pass_type(x, w, b) and not torch.is_autocast_enabled() and not traced()
            and not (x.element_size() == 2 and _library_linear_better(x.shape[0], x.shape[1], w.shape[0],
                                                                      _wants_grad(x, w, b)))
            and native.get().gate_fused_supported(w.shape[0], x.shape[1], 1)
            and _plain(x, w, b) and _no_tangent(x, w, b)
            and not _hooked(linear) and not _hooked_globally()):
        return native.get().gate_linear_topk_node(x, w.contiguous(), b, 1, None)[0]
    return None


def traced():
    r"""Whether ``torch.jit.trace`` watches."""
    return torch._C._get_tracing_state() is not None   # pylint: disable=protected-access


class _GateGemm(Function):
    r"""``logits = x W^T + b`` on the tcgen05 grouped-GEMM kernel (one group, whose row count goes
    with the launch: no offsets on the device), for any number of experts.  The expert dimension is
    padded to a multiple of 64 — the padding columns get a large negative bias, so a top-k over the
    padded logits never selects them; 64, 128 ... experts need no copies, others one launch — and the
    backward products ``dx = dl W`` and ``dW = dl^T x`` (with ``db`` from the same launch) run on the
    same kernel's input-gradient and weight-gradient modes."""

    @staticmethod
    def forward(ctx, x, weight, bias):
        tot, d = weight.shape
        pad = (-tot) % 64
        if pad == 0:   # nothing to pad: the parameters as they are
            wp = weight.contiguous().unsqueeze(0)
            bp = None if bias is None else bias.contiguous().unsqueeze(0)
        else:
            wp, bp = native.get().gate_pad(gg.aligned(weight, 16), None if bias is None else bias.contiguous(),
                                           tot + pad)
        logits = gg.forward(x, wp, None, bp)
        ctx.save_for_backward(x, wp)
        ctx.tot = tot
        ctx.has_bias = bias is not None
        return logits

    @staticmethod
    def backward(ctx, dl):
        x, wp = ctx.saved_tensors
        dl = dl.contiguous()
        dx = gg.dgrad(dl, wp, None) if ctx.needs_input_grad[0] else None
        dw = db = None
        if ctx.needs_input_grad[1] or (ctx.has_bias and ctx.needs_input_grad[2]):
            dwp, dbp = gg.wgrad(dl, x, None, 1, with_bias_grad=True)
            dw = dwp[0, :ctx.tot]
            db = dbp[0, :ctx.tot] if ctx.has_bias else None
        return dx, dw, db


def _gate_gemm_ok(x, weight, bias):
    return (x.is_cuda and x.dim() == 2 and x.dtype in (torch.bfloat16, torch.float16)
            and weight.dtype == x.dtype and (bias is None or bias.dtype == x.dtype)
            and x.shape[1] % 64 == 0 and x.shape[0] > 0 and not torch.is_autocast_enabled()
            and native.available()
            and native.get().grouped_gemm_supported(gg.MODE_NT, 0, weight.shape[0] + (-weight.shape[0]) % 64,
                                                    x.shape[1], 1))


def _few_tokens_ok(x, weight, bias, k):
    r"""A decoding step over 9 to 64 experts without gradients, which the kernel for few tokens takes in one
    launch instead of five."""
    return (x.is_cuda and x.dim() == 2 and 0 < x.shape[0] <= MAX_FEW_TOKENS
            and x.shape[0] * x.shape[1] * weight.shape[0] <= MAX_FEW_PRODUCTS
            and x.dtype in (torch.bfloat16, torch.float16) and weight.dtype == x.dtype
            and (bias is None or bias.dtype == x.dtype)
            and not _wants_grad(x, weight, bias)
            and not torch.is_autocast_enabled() and not traced() and _no_tangent(x, weight, bias)
            and native.get().gate_fused_supported(weight.shape[0], x.shape[1], k))


def linear_topk_softmax(x, weight, bias, k, zero=None):
    r"""``(logits [B,E], idx int64 [B,k], prob [B,k])`` of a linear gate over 2-D ``x``.

    Uses the single-pass kernel when the shape allows it (16 or 32 bits on a GPU, ``d_model`` a
    multiple of 8) and the expert count is small enough for its SIMT dot products to beat a GEMM
    (with one token per warp, 4096 tokens, ``d_model`` 1024: 30.6 vs 35.5 µs forward + backward at 2
    experts, 52 vs 37 µs at 16; up to 8 experts warps take several tokens, 17.5 µs at 2).  Above that the
    product runs on the tcgen05 grouped-GEMM kernel with a single group (:class:`_GateGemm`),
    followed by :func:`topk_softmax`, but for a few tokens without gradients (one launch); 64-bit inputs,
    32-bit ones with more than 8 experts, CPU tensors and odd ``d_model`` take the ``linear`` →
    :func:`topk_softmax` sequence of PyTorch ops.

    ``zero``: a one-element fp32 tensor on ``x``'s device that is set to 0 on the way, by the gate's
    kernel where there is one (a launch of its own took a fiftieth of a small decoding step).
    """
    if zero is not None and (not x.is_cuda or x.shape[0] == 0):
        zero.zero_()
        zero = None
    if (x.is_cuda and x.dim() == 2 and weight.shape[0] <= MAX_SINGLE_PASS_EXPERTS
            and _single_pass_type(x, weight, bias) and not torch.is_autocast_enabled()
            and native.get().gate_fused_supported(weight.shape[0], x.shape[1], k)):
        xc = x if x.is_contiguous() else x.contiguous()
        if traced():
            if zero is not None:
                zero.zero_()
            return _LinearTopkSoftmax.apply(xc, weight.contiguous(), bias, k)
        return tuple(native.get().gate_linear_topk_node(xc, weight.contiguous(), bias, int(k), zero))
    if _few_tokens_ok(x, weight, bias, k):
        x, weight = gg.aligned(x, 16), gg.aligned(weight, 16)
        bias = None if bias is None else bias.contiguous()
        return tuple(native.get().gate_linear_topk(x, weight, bias, int(k), True, zero))
    if _gate_gemm_ok(x, weight, bias) and k <= MAX_FUSED_K:
        # more experts: tensor-core product on this library's own kernel, then the top-k /
        # softmax kernel over the (padded) logits
        tot = weight.shape[0]
        padded = _GateGemm.apply(x if x.is_contiguous() else x.contiguous(), weight, bias)
        if zero is not None and traced():
            zero.zero_()
            zero = None
        idx, prob = _TopkSoftmax.apply(padded, k, zero)
        return padded[:, :tot], idx, prob
    if zero is not None:
        zero.zero_()
    logits = torch.nn.functional.linear(x, weight, bias)
    idx, prob = topk_softmax(logits, k)
    return logits, idx, prob


# ------------------------------------------------------------------ capacity-limited gates
def balance_native(logits):
    r"""Whether the balance-loss kernels take these logits (a non-empty CUDA matrix, 16 or 32 bits, at
    most 64 experts)."""
    return (logits.is_cuda and logits.dim() == 2 and logits.shape[0] > 0 and logits.stride(1) == 1
            and logits.dtype in (torch.float32, torch.bfloat16, torch.float16)
            and native.get().balance_supported(logits.shape[1]))


def prune_to_capacity(idx, cap, tot_expert):
    r"""``idx`` with the slots of every expert beyond its first ``cap`` (slot order) set to -1."""
    return native.get().prune_gate_scalar(idx.contiguous(), int(cap), int(tot_expert))


class _BalanceLoss(Function):
    r"""``reference(logits, ids)`` — GShard's loss — from two launches, its gradient from one.  Both
    round to the type of the logits where the PyTorch operations do (without autocast).
    ``reference`` lives as long as the loss, so it must not hold the gate that holds the loss."""

    @staticmethod
    def forward(ctx, logits, ids, scale, reference):
        loss, weight = native.get().balance_loss(logits, ids, False, float(scale))
        ctx.save_for_backward(logits, ids, weight)
        ctx.reference, ctx.scale = reference, float(scale)
        return loss

    @staticmethod
    def backward(ctx, grad):
        logits, ids, weight = ctx.saved_tensors
        if torch.is_grad_enabled():   # a gradient of the gradient is wanted
            with torch.enable_grad():
                (dl,) = torch.autograd.grad(ctx.reference(logits, ids), logits, grad, create_graph=True)
        else:
            dl = native.get().balance_bwd(logits, weight, grad.contiguous(), None, None, False, ctx.scale)
        return dl, None, None, None


def gshard_loss(logits, ids, scale, reference):
    return _BalanceLoss.apply(logits, ids.contiguous(), scale, reference)


class _SwitchRoute(Function):
    r"""Switch's choice, capacity limit and balance loss of one rank: ``(ids [n, 1], score [n, 1],
    loss)``.  ``reference(logits, chosen, kept)`` gives ``(score, loss)`` in PyTorch operations for
    the chosen experts and those of them that the capacity kept (-1 elsewhere).  It lives as long
    as the loss, so it must not hold the gate that holds the loss."""

    @staticmethod
    def forward(ctx, logits, cap, reference):
        nat = native.get()
        tot = logits.shape[1]
        win, score = nat.switch_top1(logits)
        kept = nat.prune_gate_scalar(win, cap, tot)
        loss, weight = nat.balance_loss(logits, kept, True, float(tot))
        # (`kept` is the caller's to change; a second derivative forms it again)
        ctx.save_for_backward(logits, win, weight)
        ctx.reference, ctx.cap = reference, cap
        ctx.mark_non_differentiable(kept)
        ctx.set_materialize_grads(False)
        return kept, score, loss

    @staticmethod
    def backward(ctx, _grad_kept, grad_score, grad_loss):
        logits, win, weight = ctx.saved_tensors
        if grad_score is None and grad_loss is None:
            return None, None, None
        if torch.is_grad_enabled():   # a gradient of the gradient is wanted
            kept = native.get().prune_gate_scalar(win, ctx.cap, logits.shape[1])
            with torch.enable_grad():
                outs, grads = [], []
                for out, grad in zip(ctx.reference(logits, win, kept), (grad_score, grad_loss)):
                    if grad is not None:
                        outs.append(out)
                        grads.append(grad)
                (dl,) = torch.autograd.grad(outs, logits, grads, create_graph=True)
        else:
            dl = native.get().balance_bwd(logits, weight, None if grad_loss is None else grad_loss.contiguous(),
                                          None if grad_score is None else win,
                                          None if grad_score is None else grad_score.contiguous(),
                                          True, float(logits.shape[1]))
        return dl, None, None


def switch_route(logits, cap, reference):
    return _SwitchRoute.apply(logits.contiguous(), int(min(cap, 2 ** 31 - 1)), reference)
