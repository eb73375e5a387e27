r"""GPU tier: the gate's kernels at the sizes their launch rules choose by."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _native():
    from fastmoe_b200.ops import native
    return native.get()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens,d,experts,k", [(1, 8, 9, 1), (3, 264, 17, 8), (129, 256, 33, 4), (512, 1024, 64, 2), (5, 2048, 63, 3)])
def test_few_tokens_many_experts(dtype, tokens, d, experts, k):
    r"""Logits within one rounding and an fp32 sum of d terms of 64 bits; ids and probabilities those of
    the top-k kernel on the same logits, also with ties, infinities and NaN."""
    from fastmoe_b200.ops import gating
    torch.manual_seed(tokens + experts)
    x = torch.randn(tokens, d, device=DEV, dtype=dtype)
    w = (torch.randn(experts, d, device=DEV) / d ** 0.5).to(dtype)
    w[experts // 2] = w[0]            # a tie in every token
    b = torch.randn(experts, device=DEV).to(dtype) * 0
    if tokens > 2:
        x[0, 0], x[1, 0], x[2, 0] = float("nan"), float("inf"), 0
    with torch.no_grad():
        assert gating._few_tokens_ok(x, w, b, k)
        logits, idx, prob = gating.linear_topk_softmax(x, w, b, k)
    ref = x.double() @ w.double().t() + b.double()
    size = x.double().abs() @ w.double().abs().t()
    ok = torch.isfinite(ref)
    eps = torch.finfo(dtype).eps
    assert bool(((logits.double() - ref).abs() <= eps * ref.abs() + d * 2.0 ** -24 * size + 1e-7)[ok].all())
    i2, p2 = _native().gate_topk_softmax(logits, k)
    assert torch.equal(idx, i2) and torch.equal(prob.nan_to_num(7.0), p2.nan_to_num(7.0))
    chosen = idx.cpu()
    assert int(chosen.min()) >= 0 and int(chosen.max()) < experts
    assert all(len(set(row)) == k for row in chosen.tolist())   # NaN or not
    finite = ok.all(1)
    top = torch.topk(logits.float(), k, dim=1).values
    assert torch.equal(logits.float().cpu().gather(1, chosen)[finite.cpu()], top[finite].cpu())


def test_few_tokens_rule():
    from fastmoe_b200.ops import gating
    x = torch.randn(16, 64, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(16, 64, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    assert not gating._few_tokens_ok(x, w, None, 2)            # gradients are wanted
    with torch.no_grad():
        assert gating._few_tokens_ok(x, w, None, 2)
        assert not gating._few_tokens_ok(x.repeat(33, 1), w, None, 2)
        assert not gating._few_tokens_ok(x.float(), w.float(), None, 2)
        assert not gating._few_tokens_ok(x, w.repeat(5, 1), None, 2)   # more than 64 experts


@pytest.mark.parametrize("experts", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("tokens,d", [(2367, 264), (2369, 256), (4737, 64)])   # 1, 2 and 4 tokens per warp, odd ends
def test_gate_backward_of_several_tokens_per_warp(experts, tokens, d):
    r"""Against 64 bits: dl is exact to a few fp32 roundings; dx a sum of as many terms as experts and one
    rounding to bf16; dW and db fp32 sums over the tokens and one rounding."""
    nat = _native()
    torch.manual_seed(tokens + experts)
    k = min(2, experts)
    x = torch.randn(tokens, d, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(experts, d, device=DEV, dtype=torch.bfloat16)
    logits, idx, prob = nat.gate_linear_topk(x, w, None, k)
    dp, dlog = torch.randn_like(prob), torch.randn_like(logits)
    dlog[::3] = 0
    dx, dw, db, dl = nat.gate_linear_topk_bwd(dp, idx, prob, dlog, x, w, True, True)
    p, g = prob.double(), dp.double()
    sel = p * (g - (p * g).sum(1, keepdim=True))
    ref = dlog.double().scatter_add(1, idx, sel)
    assert bool(((dl.double() - ref).abs() <= 8 * 2.0 ** -24 * (dlog.double().abs() + 4 * g.abs().sum(1, keepdim=True))).all())
    dl = dl.double()
    eps = 2.0 ** -8
    for got, want, size, terms in [(dx, dl @ w.double(), dl.abs() @ w.double().abs(), experts),
                                   (dw, dl.t() @ x.double(), dl.abs().t() @ x.double().abs(), tokens),
                                   (db, dl.sum(0), dl.abs().sum(0), tokens)]:
        assert bool(((got.double() - want).abs() <= eps * want.abs() + terms * 2.0 ** -24 * size + 1e-30).all())


# 1, 2 and 4 tokens per warp, strips of 128 columns with a rest, fewer tokens than a block has warps
@pytest.mark.parametrize("experts,k,bias", [(1, 1, True), (2, 2, False), (3, 1, True), (4, 2, True), (5, 3, True), (8, 2, True)])
@pytest.mark.parametrize("tokens,d", [(3, 8), (257, 136), (2369, 264), (4737, 64), (4800, 1024)])
def test_fp32_gate(tokens, d, experts, k, bias):
    r"""The fp32 linear gate against 64 bits.  Every sum of n products is formed in fp32: its error is at most
    n 2^-24 times the sum of the magnitudes; the softmax's exponential has 2 units in the last place and an
    argument of at most 2^-24 |v| error, taken as 32 units of 2^-24."""
    from fastmoe_b200.ops import gating
    torch.manual_seed(tokens + experts)
    x = torch.randn(tokens, d, device=DEV, requires_grad=True)
    w = (torch.randn(experts, d, device=DEV) / d ** 0.5).requires_grad_(True)
    b = torch.randn(experts, device=DEV, requires_grad=True) if bias else None
    assert gating._single_pass_type(x, w, b)
    logits, idx, prob = gating.linear_topk_softmax(x, w, b, k)
    u = 2.0 ** -24
    x64, w64 = x.detach().double(), w.detach().double()
    b64 = b.detach().double() if bias else 0.0
    ref, size = x64 @ w64.t() + b64, x64.abs() @ w64.abs().t() + (b64.abs() if bias else 0.0)
    assert bool(((logits.double() - ref).abs() <= (d + 2) * u * size).all())
    val, chosen = torch.topk(logits.detach(), k, dim=1)
    assert torch.equal(idx, chosen)
    assert bool(((prob.double() - torch.softmax(val.double(), 1)).abs() <= 32 * u).all())
    gl, gp = torch.randn_like(logits), torch.randn_like(prob)
    torch.autograd.backward([logits, prob], [gl, gp])
    p, g = prob.detach().double(), gp.double()
    through = p * (g - (p * g).sum(1, keepdim=True))
    dl = gl.double().scatter_add(1, idx, through)
    dl_err = (8 + 2 * k) * u * gl.double().abs().scatter_add(1, idx, p * (g.abs() + (p * g).abs().sum(1, keepdim=True)))
    for got, want, bound in [
            (x.grad, dl @ w64, (experts + 1) * u * (dl.abs() @ w64.abs()) + dl_err @ w64.abs()),
            (w.grad, dl.t() @ x64, (tokens + 1) * u * (dl.abs().t() @ x64.abs()) + dl_err.t() @ x64.abs())] + (
            [(b.grad, dl.sum(0), (tokens + 1) * u * dl.abs().sum(0) + dl_err.sum(0))] if bias else []):
        assert bool(((got.double() - want).abs() <= bound).all())


def test_fp32_gate_gradient_of_the_gradient():
    from fastmoe_b200.ops import gating
    torch.manual_seed(0)
    x = torch.randn(40, 32, device=DEV, requires_grad=True)
    w = torch.randn(4, 32, device=DEV, requires_grad=True)
    second = []
    for logits in (gating.linear_topk_softmax(x, w, None, 2)[0], gating._LinearTopkSoftmax.apply(x, w, None, 2)[0],
                   torch.nn.functional.linear(x, w)):
        dx, = torch.autograd.grad(logits.square().sum(), x, create_graph=True)
        second.append(torch.autograd.grad(dx.square().sum(), w)[0])
    # sums of at most 40 * 32 terms in fp32
    for got in second[:2]:
        assert torch.allclose(got, second[2], rtol=1e-3, atol=1e-3 * float(second[2].abs().max()))


def test_gate_gradient_of_the_gradient_at_odd_addresses():
    r"""fp32 sums of at most 40 * 32 terms."""
    from fastmoe_b200.ops import gating
    torch.manual_seed(0)
    flat_x, flat_w = (torch.randn(n + 1, device=DEV, requires_grad=True) for n in (40 * 32, 4 * 32))
    second = []
    for gate in (lambda x, w: gating.linear_topk_softmax(x, w, None, 2)[0],
                 lambda x, w: gating._LinearTopkSoftmax.apply(x, w, None, 2)[0], torch.nn.functional.linear):
        x, w = flat_x[1:].view(40, 32), flat_w[1:].view(4, 32)
        assert x.data_ptr() % 16 == 4 and w.data_ptr() % 16 == 4
        dx, dw = torch.autograd.grad(gate(x, w).square().sum(), (x, w), create_graph=True)
        second.append(torch.autograd.grad(dx.square().sum() + dw.square().sum(), (flat_x, flat_w)))
    for got in second[:2]:
        for a, b in zip(got, second[2]):
            assert torch.allclose(a, b, rtol=1e-3, atol=1e-3 * float(b.abs().max()))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("frozen", ["weight", "weight and bias", "input"])
def test_gate_saves_what_its_gradients_need(dtype, frozen):
    r"""With a frozen gate the input may be changed in place afterwards, and the weight where the input
    needs no gradient, as around ``nn.Linear``; the other gradients are those of all together."""
    from fastmoe_b200.ops import gating
    torch.manual_seed(1)
    base = [torch.randn(100, 64, device=DEV, dtype=dtype), torch.randn(4, 64, device=DEV, dtype=dtype),
            torch.randn(4, device=DEV, dtype=dtype)]
    off = {"weight": (1,), "weight and bias": (1, 2), "input": (0,)}[frozen]
    for gate in (lambda *a: gating.linear_topk_softmax(*a, 2), lambda *a: gating._LinearTopkSoftmax.apply(*a, 2)):
        results = []
        for partly in (True, False):
            t = [b.clone().requires_grad_(not partly or i not in off) for i, b in enumerate(base)]
            x, w, b = (v * 1 for v in t)   # (not leaves, which nothing may change in place)
            logits, _idx, prob = gate(x, w, b)
            if partly and frozen == "weight and bias":
                x.add_(1.0)
            elif partly and frozen == "input":
                w.add_(1.0)
            torch.autograd.backward([logits, prob], [torch.ones_like(logits), logits.detach()[:, :2] + 1])
            results.append([v.grad for i, v in enumerate(t) if i not in off])
        for a, c in zip(*results):
            assert torch.equal(a, c)


def test_fp32_gate_keeps_subclasses_and_autocast_on_the_operations():
    from fastmoe_b200.ops import gating

    class Mine(torch.Tensor):
        pass
    x, w = torch.randn(16, 64, device=DEV), torch.randn(4, 64, device=DEV)
    assert gating._single_pass_type(x, w, None)
    assert not gating._single_pass_type(x, w.as_subclass(Mine), None)
    assert not gating._single_pass_type(x.bfloat16(), w, None)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert gating.linear_topk_softmax(x, w, None, 2)[0].dtype == torch.bfloat16
    with pytest.raises(RuntimeError):
        gating.linear_topk_softmax(x, w[:, :56], None, 2)   # widths that differ


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tot,d,bias", [(9, 64, True), (16, 1024, True), (63, 192, False), (65, 16384, True), (200, 4096, False)])
def test_padded_gate(dtype, tot, d, bias):
    torch.manual_seed(tot)
    w = torch.randn(tot, d, device=DEV, dtype=dtype)
    b = torch.randn(tot, device=DEV, dtype=dtype) if bias else None
    pad = -tot % 64
    wp, bp = _native().gate_pad(w, b, tot + pad)
    assert torch.equal(wp, torch.nn.functional.pad(w, (0, 0, 0, pad)).unsqueeze(0))
    want = torch.full((1, tot + pad), -30000.0, device=DEV, dtype=dtype)
    want[0, :tot] = b if bias else 0
    assert torch.equal(bp, want)


def test_padded_gate_of_views():
    from fastmoe_b200.ops import gating
    torch.manual_seed(0)
    flat = torch.randn(16 * 128 + 1, device=DEV).bfloat16()
    w = flat[1:].view(16, 128)                                       # an odd address
    b = torch.randn(32, device=DEV).bfloat16()[::2]
    x = torch.randn(600, 128, device=DEV).bfloat16()
    odd = gating._GateGemm.apply(x, w, b)
    strided = gating._GateGemm.apply(x, w.t().contiguous().t(), b.clone())
    plain = gating._GateGemm.apply(x, w.clone(), b.clone())
    assert torch.equal(odd, plain) and torch.equal(strided, plain)
