r"""GPU tier: whole layers against fp32 PyTorch oracles (the matrix of the reference's
``tests/test_numerical.py``: expert counts, top-k, dtypes; plus gates and pytree inputs)."""
import pytest
import torch
import torch.nn as nn

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _fp32_leaves(moe):
    e = moe.experts
    return [t.detach().float().requires_grad_(True)
            for t in (e.htoh4.weight, e.htoh4.bias, e.h4toh.weight, e.h4toh.bias)]


def _dense_reference(moe, x32, idx, score32, leaves=None):
    r"""fp32 evaluation of an FMoETransformerMLP with given routing (vectorised per expert)."""
    e = moe.experts
    w1, b1, w2, b2 = leaves if leaves is not None else _fp32_leaves(moe)
    out = torch.zeros_like(x32)
    for j in range(idx.shape[1]):
        for ex in range(w1.shape[0]):
            m = idx[:, j] == ex
            if m.any():
                h = e.activation(x32[m] @ w1[ex].t() + b1[ex])
                out[m] = out[m] + score32[m, j:j + 1] * (h @ w2[ex].t() + b2[ex])
    return out


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("num_expert,top_k,d,h,batch,act", [
    (4, 2, 64, 128, 300, nn.GELU()),
    (8, 3, 128, 256, 1000, nn.ReLU()),
    (2, 1, 256, 512, 64, nn.GELU(approximate="tanh")),
    (4, 2, 64, 128, 257, nn.Sequential(nn.ReLU(), nn.Dropout(0.0))),
])
def test_fused_mlp_forward_backward(dtype, num_expert, top_k, d, h, batch, act):
    from fastmoe_b200 import FMoETransformerMLP
    from fastmoe_b200.ops import fused, native
    torch.manual_seed(42)
    moe = FMoETransformerMLP(num_expert=num_expert, d_model=d, d_hidden=h, top_k=top_k,
                             activation=act).to(DEV).to(dtype)
    with torch.no_grad():
        moe.experts.htoh4.bias.normal_(0, 0.1)
        moe.experts.h4toh.bias.normal_(0, 0.1)
    x = torch.randn(batch, d, device=DEV, dtype=dtype, requires_grad=True)
    assert fused.supports(moe, x, torch.zeros(1, top_k, dtype=torch.long))
    y = moe(x)
    gy = torch.randn_like(y)
    y.backward(gy)
    got = {n: p.grad.float().clone() for n, p in moe.named_parameters()}
    gx = x.grad.float().clone()
    moe.zero_grad()

    # fp32 oracle with the same routing decisions
    x32 = x.detach().float().requires_grad_(True)
    logits = moe.gate.gate(x.detach()).float()
    gw = moe.gate.gate.weight.float().detach().requires_grad_(True)
    gb = moe.gate.gate.bias.float().detach().requires_grad_(True)
    logits32 = x32 @ gw.t() + gb
    _, idx = torch.topk(logits, top_k, dim=-1)
    score32 = torch.softmax(torch.gather(logits32, 1, idx), dim=-1)
    leaves = _fp32_leaves(moe)
    ref = _dense_reference(moe, x32, idx, score32, leaves)
    ref.backward(gy.float())
    w1g, b1g, w2g, b2g = [t.grad for t in leaves]
    tol = 6e-2 if dtype == torch.bfloat16 else 1e-2
    assert torch.allclose(y.float(), ref, atol=tol, rtol=tol), float((y.float() - ref).abs().max())
    assert torch.allclose(gx, x32.grad, atol=tol * 2, rtol=tol)
    scale = batch ** 0.5
    assert torch.allclose(got["experts.htoh4.weight"], w1g, atol=tol * scale, rtol=tol)
    assert torch.allclose(got["experts.h4toh.weight"], w2g, atol=tol * scale, rtol=tol)
    assert torch.allclose(got["experts.htoh4.bias"], b1g, atol=tol * scale, rtol=tol)
    assert torch.allclose(got["experts.h4toh.bias"], b2g, atol=tol * scale, rtol=tol)
    assert torch.allclose(got["gate.gate.weight"], gw.grad, atol=tol * scale, rtol=tol * 2)
    assert native.get().read_status(0) == 0


def test_fused_mlp_with_dropped_slots():
    r"""A gate that drops slots (-1): dropped slots contribute zero and receive zero gradient."""
    from fastmoe_b200 import FMoETransformerMLP
    from fastmoe_b200.gates import GShardGate
    torch.manual_seed(0)
    moe = FMoETransformerMLP(num_expert=4, d_model=64, d_hidden=128, top_k=2,
                             gate=GShardGate).to(DEV).to(torch.bfloat16)
    moe.gate.capacity = (0.3, 0.3)
    x = torch.randn(400, 64, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    seen = {}
    moe.gate_hook = lambda idx, score, _: seen.update(idx=idx.clone(), score=score.detach().clone())
    y = moe(x)
    y.float().sum().backward()
    idx = seen["idx"]
    assert (idx < 0).any()
    ref = _dense_reference(moe, x.detach().float(), idx, seen["score"].float().view(-1, 2))
    assert torch.allclose(y.float(), ref, atol=6e-2, rtol=6e-2)
    assert torch.isfinite(x.grad.float()).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_general_path_on_gpu(dtype):
    r"""Arbitrary experts + FMoELinear in fp32/fp64 on the device (reference-precision kernels)."""
    from fastmoe_b200 import FMoE, FMoETransformerMLP
    from oracle import LinearExpert, moe_bruteforce
    torch.manual_seed(3)
    d = 16
    moe = FMoE(num_expert=4, d_model=d, top_k=2, expert=LinearExpert).to(DEV).to(dtype)
    x = torch.randn(40, d, device=DEV, dtype=dtype, requires_grad=True)
    y = moe(x)
    val, idx = torch.topk(moe.gate.gate(x), 2, dim=-1)
    ref = moe_bruteforce(x, idx, torch.softmax(val, -1), moe.experts)
    assert torch.allclose(y, ref, atol=1e-4)
    y.sum().backward()

    mlp = FMoETransformerMLP(num_expert=4, d_model=16, d_hidden=32, top_k=2).to(DEV).to(dtype)
    x2 = torch.randn(64, 16, device=DEV, dtype=dtype, requires_grad=True)
    y2 = mlp(x2)
    cpu = FMoETransformerMLP(num_expert=4, d_model=16, d_hidden=32, top_k=2).to(dtype)
    cpu.load_state_dict(mlp.state_dict())
    y2c = cpu(x2.detach().cpu())
    assert torch.allclose(y2.cpu(), y2c, atol=1e-4)
    y2.sum().backward()
    assert torch.isfinite(x2.grad).all()


@pytest.mark.parametrize("gate_name", ["NaiveGate", "NoisyGate", "GShardGate", "SwitchGate",
                                       "DCGate", "ZeroGate", "SwipeGate"])
def test_gates_run_on_gpu(gate_name):
    from fastmoe_b200 import FMoETransformerMLP
    from fastmoe_b200 import gates
    torch.manual_seed(1)
    gate = getattr(gates, gate_name)
    top_k = 1 if gate_name == "SwitchGate" else 2
    moe = FMoETransformerMLP(num_expert=4, d_model=64, d_hidden=128, top_k=top_k,
                             gate=gate).to(DEV).to(torch.bfloat16)
    x = torch.randn(128, 64, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    y = moe(x)
    loss = y.float().pow(2).mean()
    if moe.gate.has_loss:
        loss = loss + moe.gate.get_loss().float().sum()
    loss.backward()
    assert torch.isfinite(y.float()).all() and torch.isfinite(x.grad.float()).all()


def test_smoke_entry():
    import __graft_entry__ as entry
    entry.smoke()


@pytest.mark.parametrize("case", ["plain", "strided", "scores_fp32", "frozen_weights", "frozen_input", "no_grad",
                                  "unaligned", "dropped"])
@pytest.mark.parametrize("act", [torch.nn.GELU(), torch.nn.Identity()])
def test_native_layer_call_equals_separate_launches(case, act, monkeypatch):
    r"""One native call per direction against the route / dispatch / experts / combine functions (taken
    when the bounds checks look between the launches): the same kernels, so the same bits."""
    from fastmoe_b200 import FMoETransformerMLP
    from fastmoe_b200.ops import fused
    torch.manual_seed(13)
    layer = FMoETransformerMLP(num_expert=5, d_model=128, d_hidden=192, top_k=2, activation=act).cuda().bfloat16()
    x = torch.randn(77, 128, device="cuda").bfloat16()
    score = torch.rand(77, 2, device="cuda").to(torch.float32 if case == "scores_fp32" else torch.bfloat16)
    idx = torch.randint(0, 5, (77, 2), device="cuda")
    if case == "strided":
        x = torch.randn(128, 77, device="cuda").bfloat16().t()
        score = torch.rand(2, 77, device="cuda").bfloat16().t()
        idx = torch.randint(0, 5, (2, 77), device="cuda").t()
    if case == "dropped":
        idx[::3, 1] = -1
        idx[5] = -1
    if case == "frozen_weights":
        layer.experts.requires_grad_(False)
    if case == "unaligned":
        for lin in (layer.experts.htoh4, layer.experts.h4toh):
            flat = torch.empty(lin.weight.numel() + 1, device="cuda", dtype=torch.bfloat16)
            flat[1:] = lin.weight.detach().view(-1)
            lin.weight = torch.nn.Parameter(flat[1:].view_as(lin.weight))
    gy = torch.randn(77, 128, device="cuda").bfloat16()

    def run():
        layer.zero_grad(set_to_none=True)
        xi = x.detach().requires_grad_(case != "frozen_input")
        si = score.detach().requires_grad_(True)
        if case == "no_grad":
            with torch.no_grad():
                return [fused.moe_mlp_forward(layer, xi, idx, si)]
        y = fused.moe_mlp_forward(layer, xi, idx, si)
        y.backward(gy)
        return [y, xi.grad, si.grad] + [p.grad for p in layer.experts.parameters()]

    got = run()
    monkeypatch.setenv("FMOE_DEBUG_BOUNDS", "1")
    want = run()
    assert len(got) == len(want)
    for a, b in zip(got, want):
        assert (a is None) == (b is None)
        if a is not None:
            assert a.dtype == b.dtype and torch.equal(a, b)


def _shifted(t):
    r"""The same values as a contiguous view that starts one element after an allocation."""
    flat = torch.empty(t.numel() + 1, device=t.device, dtype=t.dtype)
    flat[1:] = t.detach().reshape(-1)
    view = flat[1:].view_as(t)
    assert view.is_contiguous() and view.data_ptr() % 16 != 0
    return view


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("act", [nn.GELU(), nn.Tanh()])
@pytest.mark.parametrize("experts", [5, 12])
def test_rows_that_start_anywhere(dtype, act, experts, monkeypatch):
    r"""Input, output gradient and gate weight inside flat buffers, for a fused and for a user's
    activation, with the gate in one kernel (5 experts) and on the tensor cores (12), and with the
    bounds checks on (separate launches): the bits of aligned operands."""
    from fastmoe_b200 import FMoETransformerMLP
    torch.manual_seed(21)
    layer = FMoETransformerMLP(num_expert=experts, d_model=128, d_hidden=192, top_k=2, activation=act).to(DEV).to(dtype)
    x = torch.randn(77, 128, device=DEV).to(dtype)
    gy = torch.randn(77, 128, device=DEV).to(dtype)

    def run(x, gy):
        layer.zero_grad(set_to_none=True)
        xi = x.detach().requires_grad_(True)
        y = layer(xi)
        y.backward(gy)
        return [y, xi.grad] + [p.grad for p in layer.parameters()]

    want = run(x, gy)
    layer.gate.gate.weight = nn.Parameter(_shifted(layer.gate.gate.weight))
    for checks in ("0", "1"):
        monkeypatch.setenv("FMOE_DEBUG_BOUNDS", checks)
        for a, b in zip(run(_shifted(x), _shifted(gy)), want):
            assert torch.equal(a, b)


@pytest.mark.parametrize("experts", [5, 12])
@pytest.mark.parametrize("act", [nn.GELU(), nn.Tanh()])
def test_saved_tensors_that_come_back_elsewhere(experts, act, monkeypatch):
    r"""Hooks on saved tensors may return them at any address: the bits of a run without hooks."""
    from fastmoe_b200 import FMoETransformerMLP
    torch.manual_seed(28)
    layer = FMoETransformerMLP(num_expert=experts, d_model=128, d_hidden=192, top_k=2, activation=act).to(DEV).bfloat16()
    x = torch.randn(77, 128, device=DEV).bfloat16()
    gy = torch.randn(77, 128, device=DEV).bfloat16()

    def run(unpack):
        layer.zero_grad(set_to_none=True)
        xi = x.detach().requires_grad_(True)
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
            y = layer(xi)
        y.backward(gy)
        return [y, xi.grad] + [p.grad for p in layer.parameters()]

    for checks in ("0", "1"):
        monkeypatch.setenv("FMOE_DEBUG_BOUNDS", checks)
        want = run(lambda t: t)
        for a, b in zip(run(lambda t: _shifted(t) if t.dtype == torch.bfloat16 else t), want):
            assert torch.equal(a, b)


def test_native_calls_refuse_unaligned_rows():
    r"""The kernels with 16-byte accesses are not launched on rows that start elsewhere."""
    from fastmoe_b200.ops import native
    nat = native.get()
    rows = torch.zeros(8, 64, device=DEV, dtype=torch.bfloat16)
    bad = _shifted(rows)
    idx = torch.zeros(8, device=DEV, dtype=torch.int64)
    _counts, rank, offs = nat.route_offs(idx, 1)
    score = torch.ones(8, device=DEV, dtype=torch.bfloat16)
    w = torch.zeros(2, 64, device=DEV, dtype=torch.bfloat16)
    for call in (lambda: nat.scatter_rows(bad, idx, rank, offs, None, 1, rows, None),
                 lambda: nat.scatter_rows(rows, idx, rank, offs, None, 1, bad, None),
                 lambda: nat.gather_combine(bad, idx, rank, offs, None, 1, rows),
                 lambda: nat.combine_bwd(bad, rows, idx, rank, offs, score, 1, rows.clone(), score.clone()),
                 lambda: nat.colsum(bad, offs), lambda: nat.slot_dot(bad, rows, idx, 1, score),
                 lambda: nat.gate_linear_topk(bad, w, None, 1), lambda: nat.gate_linear_topk(rows, _shifted(w), None, 1)):
        with pytest.raises(RuntimeError, match="16-byte aligned"):
            call()


@pytest.mark.parametrize("shape", [(64, 128), (64, 72)])
def test_grouped_linear_of_unaligned_rows(shape):
    r"""``FMoELinear`` on the tensor cores and (72 columns) on the general kernels, whose bias gradient
    is a kernel of its own."""
    from fastmoe_b200 import FMoELinear
    torch.manual_seed(22)
    layer = FMoELinear(3, *shape).to(DEV).bfloat16()
    counts = torch.tensor([20, 0, 13])
    x = torch.randn(33, shape[0], device=DEV).bfloat16()
    gy = torch.randn(33, shape[1], device=DEV).bfloat16()
    got = []
    for a, g in ((x, gy), (_shifted(x), _shifted(gy))):
        layer.zero_grad(set_to_none=True)
        a = a.detach().requires_grad_(True)
        y = layer(a, counts)
        y.backward(g)
        got.append([y, a.grad, layer.weight.grad, layer.bias.grad])
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("act", [nn.GELU(), nn.Tanh()])
def test_no_rows_at_all(dtype, act):
    r"""Forward and backward of the layer without tokens and of ``FMoELinear`` without rows: empty
    outputs and input gradients, zero parameter gradients."""
    from fastmoe_b200 import FMoELinear, FMoETransformerMLP
    layer = FMoETransformerMLP(num_expert=4, d_model=64, d_hidden=128, top_k=2, activation=act).to(DEV).to(dtype)
    linear = FMoELinear(3, 64, 128).to(DEV).to(dtype)
    torch.full((4, 128, 64), float("nan"), device=DEV, dtype=dtype)   # stale bits for the allocator to hand out
    for module, args, width in ((layer, (), 64), (linear, (torch.zeros(3, dtype=torch.int64),), 128)):
        x = torch.empty(0, 64, device=DEV, dtype=dtype, requires_grad=True)
        y = module(x, *args)
        assert y.shape == (0, width)
        y.backward(torch.empty_like(y))
        assert x.grad.shape == (0, 64)
        for name, p in module.named_parameters():
            assert p.grad is not None and not p.grad.any(), name


def test_no_rows_leave_an_accumulated_gradient_alone():
    from fastmoe_b200.ops import grouped_gemm as gg
    out = torch.ones(2, 64, 32, device=DEV, dtype=torch.bfloat16)
    offs = torch.zeros(3, dtype=torch.int32, device=DEV)
    empty = [torch.empty(0, n, device=DEV, dtype=torch.bfloat16) for n in (64, 32)]
    assert (gg.wgrad(*empty, offs, 2, out=out, accumulate=True) == 1).all()
    assert not gg.wgrad(*empty, offs, 2, out=out).any()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_native_nodes_as_the_python_ones(monkeypatch, dtype):
    r"""The layer's and the gate's nodes of the native engine and those a trace records give the same bits:
    all gradients, single ones, and with a gradient at the gate's scores and logits."""
    from fastmoe_b200 import FMoETransformerMLP
    from fastmoe_b200.ops import fused, gating
    torch.manual_seed(0)
    moe = FMoETransformerMLP(num_expert=4, d_model=64, d_hidden=128, top_k=2).to(DEV).to(dtype)
    x0 = torch.randn(300, 64, device=DEV, dtype=dtype)
    gy = torch.randn_like(x0)

    def grads(wanted):
        x = x0.clone().requires_grad_(True)
        leaves = dict(moe.named_parameters(), x=x)
        ids, score, logits = moe.gate(x, return_all_scores=True)
        y = fused.moe_mlp_forward(moe, x, ids, score)
        loss = (y * gy).float().sum() + score.float().square().sum() + logits.float().square().sum() + moe.gate.get_loss().sum()
        return [y.detach()] + list(torch.autograd.grad(loss, [leaves[n] for n in wanted]))

    names = [n for n, _ in moe.named_parameters()] + ["x"]
    for wanted in [names] + [[n] for n in names]:
        native_ones = grads(wanted)
        with monkeypatch.context() as m:
            m.setattr(fused, "traced", lambda: True)
            m.setattr(gating, "traced", lambda: True)
            python_ones = grads(wanted)
        assert all(torch.equal(a, b) for a, b in zip(native_ones, python_ones))


def test_traced_layer_follows_its_input():
    from fastmoe_b200 import FMoETransformerMLP
    torch.manual_seed(0)
    for experts in (4, 16):
        moe = FMoETransformerMLP(num_expert=experts, d_model=64, d_hidden=64, top_k=2).to(DEV).bfloat16().eval()
        xs = [torch.randn(40, 64, device=DEV, dtype=torch.bfloat16) for _ in range(2)]
        with torch.no_grad():
            traced = torch.jit.trace(moe, xs[0], check_trace=False)
            want = moe(xs[1])
            if experts <= 8:
                assert torch.equal(traced(xs[1]), want)
            else:   # (traced, many experts keep the tensor-core gate: sums in another order)
                assert torch.allclose(traced(xs[1]).float(), want.float(), atol=2e-2, rtol=2e-2)


def test_native_nodes_refuse_what_the_python_ones_refuse():
    from torch.autograd import forward_ad
    from fastmoe_b200 import FMoETransformerMLP
    moe = FMoETransformerMLP(num_expert=4, d_model=64, d_hidden=64, top_k=2).to(DEV).bfloat16()
    x = torch.randn(16, 64, device=DEV, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError), forward_ad.dual_level():
        moe(forward_ad.make_dual(x, torch.ones_like(x)))
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: moe(t).float().sum())(x)
    with pytest.raises(RuntimeError):
        torch.func.vmap(moe)(x.view(2, 8, 64))


def test_gate_for_few_tokens_refuses_forward_mode():
    from torch.autograd import forward_ad
    from fastmoe_b200.gates import NaiveGate
    gate = NaiveGate(64, 16, 1, 2).to(DEV).bfloat16()
    x = torch.randn(16, 64, device=DEV, dtype=torch.bfloat16)
    with torch.no_grad(), forward_ad.dual_level(), pytest.raises(NotImplementedError):
        gate(forward_ad.make_dual(x, torch.ones_like(x)))


def test_switch_gate_linear_is_the_kernel_only_when_nobody_looks():
    from fastmoe_b200.gates import SwitchGate
    from fastmoe_b200.ops import gating
    gate = SwitchGate(64, 4, 1, switch_eps=0.0).to(DEV).bfloat16()
    x = torch.randn(32, 64, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    logits = gating.linear_logits(x, gate.gate)
    assert torch.allclose(logits.float(), gate.gate(x).float(), atol=2e-2)
    seen = []
    handle = gate.gate.register_forward_hook(lambda *_: seen.append(1))
    assert gating.linear_logits(x, gate.gate) is None
    gate(x)
    assert seen
    handle.remove()
    # a gradient of the gradient, as of the linear
    results = []
    for fused in (True, False):
        p = [t.detach().clone().requires_grad_(True) for t in (x, gate.gate.weight, gate.gate.bias)]
        linear = torch.nn.Linear(64, 4).to(DEV).bfloat16()
        linear.weight, linear.bias = torch.nn.Parameter(p[1]), torch.nn.Parameter(p[2])
        leaves = [p[0], linear.weight, linear.bias]
        out = gating.linear_logits(p[0], linear) if fused else linear(p[0])
        first = torch.autograd.grad(out.float().square().sum(), leaves, create_graph=True)
        second = torch.autograd.grad(sum(g.float().square().sum() for g in first), leaves)
        results.append([t.detach().float() for t in first + second])
    for a, b in zip(*results):
        assert float((a - b).norm()) <= 2e-2 * float(b.norm())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("what", ["one score per token", "scores on the host", "ids on the host"])
def test_layer_refuses_what_a_gate_should_not_return(dtype, what):
    from fastmoe_b200 import FMoETransformerMLP
    from fastmoe_b200.ops import native
    layer = FMoETransformerMLP(num_expert=4, d_model=64, d_hidden=64, top_k=2).to(DEV).to(dtype)
    x = torch.randn(64, 64, device=DEV, dtype=dtype)
    ids = torch.randint(0, 4, (64, 2), device=DEV)
    scores = torch.rand(64, 2, device=DEV, dtype=dtype)
    if what == "one score per token":
        scores = scores[:, :1]
    elif what == "scores on the host":
        scores = scores.cpu()
    else:
        ids = ids.cpu()
    layer.gate.forward = lambda _x: (ids, scores)
    with pytest.raises(RuntimeError):
        layer(x)
    e = layer.experts
    with pytest.raises(RuntimeError, match="do not fit"):
        native.get().moe_mlp(x, scores, e.htoh4.weight, e.htoh4.bias, e.h4toh.weight, e.h4toh.bias, ids, 2, False)
