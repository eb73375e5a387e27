r"""
The fused device path of ``FMoETransformerMLP``.

One layer call is a fixed sequence of kernels with no host read in between:

    route (count + rank + offsets)  →  dispatch (rows to expert segments; peer-to-peer stores
    when the experts live on other GPUs)  →  grouped GEMM 1 (+bias, +activation, pre-activation
    kept)  →  grouped GEMM 2 (+bias)  →  combine (gate-weighted sum of the top-k rows)

It replaces ``_fmoe_general_global_forward`` of the reference (``fmoe/layers.py:26-78``:
``prepare_forward`` with two host syncs, ``MOEScatter``, a Python loop over experts with two
synchronising linears each, ``MOEGather``, ``bmm``).  Buffers are sized from host-known
quantities only (``B·k`` rows on one GPU, the configured receive capacity on several), so
autograd never needs a count on the host.  Backward mirrors forward: the combine backward
produces ``d score`` and the scaled output gradients in one pass, the activation derivative
is applied in the epilogue of the input-gradient GEMM, and the weight gradients reduce over
token rows on the tensor cores.
"""
import torch
from torch.autograd import Function

from . import grouped_gemm as gg
from . import native
from .gating import _no_tangent, _plain, traced
from .. import config
from ..transformer import activation_kind, plain_experts
from ..utils.profiling import check_routing, fused_range

_TC = (torch.bfloat16, torch.float16)


def supports(layer, x, idx, score=None):
    r"""Whether the fused kernels can run this call (else the general path is used).  Without ``score`` the
    question is whether they can with scores that fit the ids."""
    if not native.available() or idx.dim() != 2:
        return False
    if x.dtype == torch.float32:
        return _fp32_layer_ok(layer, x, idx, score)
    if x.dtype not in _TC:
        return False
    e = layer.experts
    if e.htoh4.weight.dtype != x.dtype or e.htoh4.bias is None or e.h4toh.bias is None:
        return False
    d, h = layer.d_model, layer.d_hidden
    if d % 64 != 0 or h % 64 != 0:
        return False
    if layer.world_size > 1 or _forced_ep():
        from ..parallel import symm
        return symm.fused_available(layer, x)
    return True


def _fp32_layer_ok(layer, x, idx, score):
    r"""Whether the fp32 layer on one GPU runs as :class:`_MoEMLP`.  The general path, which takes the
    rest, calls ``expert_fn`` and the expert modules: a call that somebody watches or does in another way
    stays there, and so does autocast, under which the weighted sum is formed in 16 bits."""
    e = layer.experts
    if (layer.world_size > 1 or _forced_ep() or not config.fused_enabled() or config.faster_schedule_enabled()
            or torch.is_autocast_enabled() or not layer._usual_expert_fn() or not plain_experts(e)):
        return False
    if any(t is None or t.dtype != torch.float32 or not t.is_cuda
           for t in (e.htoh4.weight, e.htoh4.bias, e.h4toh.weight, e.h4toh.bias)):
        return False
    if not _plain(x, score) or not _no_tangent(score):   # as in `rows_supported`
        return False
    # (as many choices as the layer was made for: the general path refuses others)
    return (idx.shape[1] == layer.top_k and _native_call_ok(layer, x, idx, score)
            and native.get().moe_mlp_supported_f32(layer.num_expert, layer.d_model, layer.d_hidden, idx.numel()))


def _forced_ep():
    if not config.force_ep_path():
        return False
    import torch.distributed as dist
    return dist.is_available() and dist.is_initialized()


def _rows_of_slots(idx, rank, offs):
    r"""``(row, kept)`` of every slot as PyTorch operations: for a gradient of the gradient."""
    kept = rank >= 0
    return torch.where(kept, offs[idx.clamp(0, offs.numel() - 2)] + rank, 0).long(), kept


def slot_scores(scores, dtype):
    r"""One score per slot for the kernels, which read them next to each other: ``reshape`` returns a strided
    view where it can (a column of a table, an expanded constant)."""
    return scores.reshape(-1).to(dtype).contiguous()


class _Dispatch(Function):
    r"""``xs[offs[e] + rank[s]] = x[s // k]`` for every kept slot ``s`` routed to expert ``e``;
    ``n_rows``: rows of ``xs`` where the caller knows how many slots are kept."""

    @staticmethod
    def forward(ctx, x, idx, rank, offs, k, n_rows=None):
        nat = native.get()
        xs = torch.empty(idx.numel() if n_rows is None else n_rows, x.shape[1], dtype=x.dtype, device=x.device)
        nat.scatter_rows(gg.aligned(x, 16), idx, rank, offs, None, k, xs, None)
        ctx.save_for_backward(idx, rank, offs)
        ctx.k = k
        ctx.n_tok = x.shape[0]
        return xs

    @staticmethod
    def backward(ctx, dxs):
        idx, rank, offs = ctx.saved_tensors
        if torch.is_grad_enabled():   # a gradient of the gradient is wanted
            if dxs.shape[0] == 0:
                return dxs.new_zeros(ctx.n_tok, dxs.shape[1]) + dxs.sum(), None, None, None, None, None
            row, kept = _rows_of_slots(idx, rank, offs)
            dx = torch.where(kept[:, None], dxs[row], 0).view(ctx.n_tok, ctx.k, -1).sum(1)
            return dx, None, None, None, None, None
        dx = torch.empty(ctx.n_tok, dxs.shape[1], dtype=dxs.dtype, device=dxs.device)
        native.get().gather_combine(gg.aligned(dxs, 16), idx, rank, offs, None, ctx.k, dx)
        return dx, None, None, None, None, None


class _Combine(Function):
    r"""``out[t] = Σ_j score[t, j] · ys[row(t, j)]``; dropped slots contribute nothing."""

    @staticmethod
    def forward(ctx, ys, score, idx, rank, offs, k):
        n_tok = idx.numel() // k
        out = torch.empty(n_tok, ys.shape[1], dtype=ys.dtype, device=ys.device)
        native.get().gather_combine(gg.aligned(ys, 16), idx, rank, offs, score, k, out)
        ctx.save_for_backward(ys, score, idx, rank, offs)
        ctx.k = k
        return out

    @staticmethod
    def backward(ctx, dout):
        ys, score, idx, rank, offs = ctx.saved_tensors
        if torch.is_grad_enabled():   # a gradient of the gradient is wanted (rows or scores may be constants)
            if ys.shape[0] == 0:
                return (dout[:0] * score[:1, None], torch.zeros_like(score) + ys.sum() + dout[:0].sum(),
                        None, None, None, None)
            row, kept = _rows_of_slots(idx, rank, offs)
            g = dout.repeat_interleave(ctx.k, 0)
            dys = torch.zeros_like(ys, memory_format=torch.contiguous_format).index_add(
                0, row, torch.where(kept[:, None], g * score[:, None], 0))
            return dys, torch.where(kept, (g * ys[row]).sum(1), 0), None, None, None, None
        dys = torch.empty_like(ys, memory_format=torch.contiguous_format)
        dscore = torch.empty_like(score)
        native.get().combine_bwd(gg.aligned(dout, 16), gg.aligned(ys, 16), idx, rank, offs, score, ctx.k, dys, dscore)
        return dys, dscore, None, None, None, None


def rows_supported(x, ids, scores):
    r"""Whether the kernels that move and combine rows take a call of the general path."""
    return (torch.is_tensor(x) and x.is_cuda and x.dim() == 2 and x.dtype in _TC + (torch.float32,)
            and x.shape[1] % 8 == 0 and x.shape[1] > 0
            and ids.is_cuda and ids.dtype == torch.int64 and ids.dim() in (1, 2)
            and ids.device == x.device and scores.device == x.device
            and ids.shape[0] == x.shape[0] and ids.numel() > 0 and ids.numel() < 2 ** 31
            and scores.numel() == ids.numel() and scores.is_floating_point()
            # (the operations keep a subclass for the experts, and a forward-mode derivative of the scores)
            and _plain(x, ids, scores) and _no_tangent(scores)
            and not torch.is_autocast_enabled())


def general_path(x, ids, scores, expert_fn, num_expert, own_rows=False):
    r"""The general path of one GPU around ``expert_fn(rows, counts)``: rows to their experts, the
    weighted sum of what comes back.  One read of the counts on the host, as the experts are called
    with Python slices.  With ``own_rows`` ``expert_fn`` is known to hold the rows by their segments
    only.  ``(out, rows, routing)``: ``out`` is ``None``, and ``routing`` what
    ``MOEGather`` needs, where ``expert_fn`` did not return rows that the kernels combine.

    8 experts of two ``nn.Linear`` with 2048 tokens, top-2, d 512: the zeroed tensors, copies and additions
    behind slices, and index operations and ``bmm`` around the experts, were 33 of 123 launches."""
    nat = native.get()
    k = ids.shape[1] if ids.dim() == 2 else 1
    idx = ids.contiguous().view(-1)
    counts, rank, offs, pos = nat.route_pos(idx, num_expert)
    counts = counts.cpu().long()
    n_rows = int(counts.sum())
    xs = _Dispatch.apply(x.contiguous(), idx, rank, offs, k, n_rows)
    if own_rows:
        xs.fmoe_own_rows = True   # a buffer that nobody else holds (see FMoE.expert_fn)
    ys = expert_fn(xs, counts)
    if (torch.is_tensor(ys) and ys.is_cuda and ys.dim() == 2 and ys.dtype in _TC + (torch.float32,)
            and ys.shape[0] == n_rows and ys.shape[1] % 8 == 0 and ys.shape[1] > 0 and ys.device == x.device):
        return _Combine.apply(ys.contiguous(), slot_scores(scores, ys.dtype), idx, rank, offs, k), ys, None
    return None, ys, (pos[:n_rows].long(), counts)


class _ExpertMLP(Function):
    r"""``h4toh(act(htoh4(xs)))`` over expert segments with a fused activation."""

    @staticmethod
    def forward(ctx, xs, w1, b1, w2, b2, offs, act):
        a, pre = gg.forward(xs, w1, offs, b1, act=act, want_pre=True)
        ys = gg.forward(a, w2, offs, b2)
        ctx.save_for_backward(xs, w1, w2, offs, pre, a)
        ctx.act = act
        return ys

    @staticmethod
    def backward(ctx, dys):
        xs, w1, w2, offs, pre, a = ctx.saved_tensors
        groups = w1.shape[0]
        dys = dys.contiguous()
        dw2, db2 = gg.wgrad(dys, a, offs, groups, with_bias_grad=True)
        da = gg.dgrad(dys, w2, offs, pre=pre, act=ctx.act)
        dw1, db1 = gg.wgrad(da, xs, offs, groups, with_bias_grad=True)
        dxs = gg.dgrad(da, w1, offs) if ctx.needs_input_grad[0] else None
        return dxs, dw1, db1, dw2, db2, None, None


class _GroupedLinear(Function):
    r"""One grouped linear over expert segments (used around activations that are not fused)."""

    @staticmethod
    def forward(ctx, xs, w, b, offs):
        ys = gg.forward(xs, w, offs, b)
        ctx.save_for_backward(xs, w, offs)
        return ys

    @staticmethod
    def backward(ctx, dys):
        xs, w, offs = ctx.saved_tensors
        dys = dys.contiguous()
        dw, db = gg.wgrad(dys, xs, offs, w.shape[0], with_bias_grad=True)
        dxs = gg.dgrad(dys, w, offs) if ctx.needs_input_grad[0] else None
        return dxs, dw, db, None


def expert_mlp(layer, xs, offs):
    r"""Both expert linears on rows already grouped by expert (``offs`` on the device)."""
    e = layer.experts
    act = activation_kind(e.activation)
    if act is not None:
        return _ExpertMLP.apply(xs, e.htoh4.weight, e.htoh4.bias, e.h4toh.weight, e.h4toh.bias,
                                offs, act)
    hid = _GroupedLinear.apply(xs, e.htoh4.weight, e.htoh4.bias, offs)
    hid = e.activation(hid)
    return _GroupedLinear.apply(hid.contiguous(), e.h4toh.weight, e.h4toh.bias, offs)


def expert_mlp_weights(xs, offs, w1, b1, w2, b2, activation):
    r"""Both expert linears with explicit weights ``[G, h, d]`` / ``[G, d, h]`` (``activation`` is
    the module between them)."""
    act = activation_kind(activation)
    if act is not None:
        return _ExpertMLP.apply(xs, w1, b1, w2, b2, offs, act)
    hid = _GroupedLinear.apply(xs, w1, b1, offs)
    hid = activation(hid)
    return _GroupedLinear.apply(hid.contiguous(), w2, b2, offs)


def moe_mlp_local(x, gate_idx, gate_score, w1, b1, w2, b2, activation):
    r"""The single-GPU fused MoE MLP over the ``G = w1.shape[0]`` experts given by explicit weights
    (``gate_idx`` in ``[0, G)`` or ``-1`` for slots that take no part).  Used for shadow
    experts, whose parameters arrive by broadcast and are not module parameters."""
    nat = native.get()
    k = gate_idx.shape[1]
    idx = gate_idx.contiguous().view(-1)
    score = slot_scores(gate_score, x.dtype)
    _counts, rank, offs = nat.route_offs(idx, w1.shape[0])
    xs = _Dispatch.apply(x.contiguous(), idx, rank, offs, k)
    ys = expert_mlp_weights(xs, offs, w1.contiguous(), b1.contiguous(), w2.contiguous(), b2.contiguous(),
                            activation)
    return _Combine.apply(ys, score, idx, rank, offs, k)


class _MoEMLP(Function):
    r"""The whole single-GPU layer behind the gate as one node: :class:`_Dispatch`,
    :class:`_ExpertMLP` and :class:`_Combine` with their launches issued by one native call per
    direction.  With ``keep`` false (nothing will be differentiated) the pre-activation is not
    written.  In fp32 ``xs`` and ``a`` are kept as the bf16 parts that the tensor cores multiply, 6
    bytes an element between forward and backward where fp32 has 4, and beside each GEMM its weights
    are held in parts too (6 bytes a weight, for the time of the launch).

    The native node of the same (``binding.cpp::MoEMLP``) takes all calls but traced ones: its backward
    runs without the interpreter (a small layer's step, 512 tokens, d 256, 4 experts: 429 us of host time
    with this class and the gate's, 262 with theirs)."""

    @staticmethod
    def forward(ctx, x, score, w1, b1, w2, b2, idx, act, keep):
        out, xs, pre, a, ys, rank, offs, score16, slots = native.get().moe_mlp_forward(
            x, idx, score, w1, b1, w2, b2, act, keep)
        if keep:
            ctx.save_for_backward(xs, pre, a, ys, rank, offs, score16, slots, w1, w2)
        ctx.act = act
        ctx.score_like = score.shape, score.dtype
        return out

    @staticmethod
    def backward(ctx, dout):
        xs, pre, a, ys, rank, offs, score16, slots, w1, w2 = ctx.saved_tensors
        need = ctx.needs_input_grad
        dx, dscore, dw1, db1, dw2, db2 = native.get().moe_mlp_backward(
            dout, xs, pre, a, ys, rank, offs, score16, slots, w1, w2, ctx.act,
            need[0], need[2] or need[3], need[4] or need[5])
        shape, dtype = ctx.score_like
        return (dx, dscore.to(dtype).view(shape) if need[1] else None, dw1, db1, dw2, db2, None, None, None)


def _native_call_ok(layer, x, gate_idx, gate_score):
    r"""What :class:`_MoEMLP` asks of a call in any type: an activation the GEMM epilogue knows, at
    least one row, an id and a score per slot beside it, and nobody who wants to look between the launches."""
    act = activation_kind(layer.experts.activation)
    return (act is not None and x.dim() == 2 and x.shape[0] > 0 and gate_idx.shape[1] > 0
            and gate_idx.shape[0] == x.shape[0] and gate_idx.dtype == torch.int64
            and gate_idx.device == x.device
            and (gate_score is None or (gate_score.numel() == gate_idx.numel() and gate_score.device == x.device
                                        and gate_score.is_floating_point()))
            and not config.nvtx_enabled() and not config.debug_bounds())


def _native_layer_ok(layer, x, gate_idx, gate_score):
    return (_native_call_ok(layer, x, gate_idx, gate_score)
            and (x.dtype == torch.float32   # `supports` has looked at the shapes
                 or native.get().moe_mlp_supported(layer.num_expert, layer.d_model, layer.d_hidden)))


def moe_mlp_forward(layer, x, gate_idx, gate_score):
    r"""``[B, d] → [B, d]`` for one ``FMoETransformerMLP`` call on the GPU."""
    if layer.world_size > 1 or _forced_ep():
        from ..parallel import symm
        return symm.moe_mlp_forward(layer, x, gate_idx, gate_score)
    nat = native.get()
    if _native_layer_ok(layer, x, gate_idx, gate_score):
        e = layer.experts
        args = (x, gate_score, e.htoh4.weight, e.htoh4.bias, e.h4toh.weight, e.h4toh.bias)
        keep = torch.is_grad_enabled() and any(t.requires_grad for t in args)
        run = _MoEMLP.apply if traced() else nat.moe_mlp
        return run(*args, gate_idx, gg.ACT_CODES[activation_kind(e.activation)], keep)
    k = gate_idx.shape[1]
    idx = gate_idx.contiguous().view(-1)
    score = slot_scores(gate_score, x.dtype)
    with fused_range("route"):
        counts, rank, offs = nat.route_offs(idx, layer.num_expert)
    if config.debug_bounds():
        check_routing(idx, rank, counts, layer.num_expert, offs, idx.numel())
    with fused_range("dispatch"):
        xs = _Dispatch.apply(x.contiguous(), idx, rank, offs, k)
    with fused_range("experts"):
        ys = expert_mlp(layer, xs, offs)
    with fused_range("combine"):
        return _Combine.apply(ys, score, idx, rank, offs, k)
