r"""GPU tier: the fp32 grouped GEMM on the tensor cores and the fp32 layer that is built on it."""
import pytest
import torch
import torch.nn as nn

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _native():
    from fastmoe_b200.ops import native
    return native.get()


def _offs(counts):
    from fastmoe_b200.ops import grouped_gemm as gg
    return gg.offsets_from_counts(counts, DEV)


def _bound(a_abs, terms):
    r"""What the sum of ``terms`` products may be off by, given the sum of their magnitudes: the parts of a
    product left out (2^-26); per K block of 64 four additions of the tensor cores that truncate
    (2^-23 each), one of fp32 for every block, and the small products' truncated sum, 2^-8 of it with five
    additions per 16 terms."""
    blocks = (terms + 63) // 64
    return a_abs * (2.0 ** -26 + 4 * 2.0 ** -23 + (blocks + 2) * 2.0 ** -24 + 5 * (terms / 16 + 1) * 2.0 ** -31)


@pytest.mark.parametrize("counts,k,n", [
    ([1, 0, 3], 16, 16),                      # the narrowest, a single row
    ([64, 63, 65, 0], 64, 128),               # edges of the 64-row blocks
    ([256, 255, 257, 128, 129], 72, 136),     # edges of the 256 x 128 tiles, ragged in every direction
    ([700], 520, 264),
    ([9, 0, 0, 1200, 31], 264, 1032),
    ([40] * 40, 128, 64),                     # more experts than a warp has lanes
    ([5000, 17], 64, 72),                     # one expert's rows shared among many pairs
    ([300, 200], 4096, 128),                  # a long sum whose tiles are cut
    ([2048] * 3 + [100], 256, 2048),          # several rounds and a cut rest
])
def test_split_gemm_against_64_bits(counts, k, n):
    nat = _native()
    torch.manual_seed(len(counts) * 1000 + k + n)
    rows, groups, tail = sum(counts), len(counts), 5
    offs = _offs(counts)
    x = torch.randn(rows + tail, k, device=DEV)
    dy = torch.randn(rows + tail, n, device=DEV)
    w = torch.randn(groups, n, k, device=DEV)
    b = torch.randn(groups, n, device=DEV)
    y = torch.full((rows + tail, n), float("nan"), device=DEV)
    dx = torch.full((rows + tail, k), float("nan"), device=DEV)
    dw = torch.full((groups, n, k), float("nan"), device=DEV)
    db = torch.full((groups, n), float("nan"), device=DEV)
    for _ in range(2):   # equal calls add in equal order
        nat.split_grouped_gemm(0, x, w, offs, y, b, None)
        nat.split_grouped_gemm(1, dy, w, offs, dx, None, None)
        nat.split_grouped_gemm(2, dy, x, offs, dw, None, db)
        again = [t.clone() for t in (y, dx, dw, db)] if _ == 0 else again
    assert all(torch.equal(p, q) for p, q in zip(again, (y, dx, dw, db)))
    assert not y[rows:].any() and not dx[rows:].any()   # rows past the last expert
    base = 0
    for e, c in enumerate(counts):
        s = slice(base, base + c)
        base += c
        X, D, W = x[s].double(), dy[s].double(), w[e].double()
        for got, ref, size, terms in [
                (y[s], X @ W.t() + b[e].double(), X.abs() @ W.abs().t() + b[e].abs().double(), k),
                (dx[s], D @ W, D.abs() @ W.abs(), n),
                (dw[e], D.t() @ X, D.abs().t() @ X.abs(), c)]:
            assert bool(((got.double() - ref).abs() <= _bound(size, terms)).all())
        # pieces of 256 rows, each a sum of 16 steps, 4 rows and 4 lanes; then the pieces
        assert bool(((db[e].double() - D.sum(0)).abs() <= D.abs().sum(0) * (24 + c / 256) * 2.0 ** -24).all())
    assert nat.read_status(0) == 0


def test_split_gemm_keeps_infinities_large_and_small_values():
    nat = _native()
    torch.manual_seed(0)
    counts, k, n = [70, 30], 128, 128
    offs = _offs(counts)
    x = torch.randn(100, k, device=DEV)
    w = torch.randn(2, n, k, device=DEV)
    x[3, 5] = float("inf")
    x[4, 6] = float("-inf")
    x[5, 7] = float("nan")
    x[6] = 0
    x[6, 0] = torch.finfo(torch.float32).max    # would round up to infinity in bf16
    w[:, :, 0] = 0.5
    x[7] *= 2.0 ** -100
    x[8] *= 2.0 ** 100
    y = torch.empty(100, n, device=DEV)
    nat.split_grouped_gemm(0, x, w, offs, y, None, None)
    ref = torch.cat([x[:70].double() @ w[0].double().t(), x[70:].double() @ w[1].double().t()])
    assert torch.equal(torch.isnan(y), torch.isnan(ref))
    inf = torch.isinf(ref)
    assert torch.equal(y[inf].double(), ref[inf]) and inf[3].all() and inf[4].all()
    ok = torch.isfinite(ref)
    size = torch.cat([x[:70].double().abs() @ w[0].double().abs().t(), x[70:].double().abs() @ w[1].double().abs().t()])
    assert bool(((y.double() - ref).abs()[ok] <= _bound(size, k)[ok]).all())


@pytest.mark.parametrize("exponent", [-100, -108, -112, -116, -120, -124, -127])
@pytest.mark.parametrize("which", ["rows", "weights"])
def test_split_gemm_of_values_near_the_end_of_the_range(exponent, which):
    r"""As for other values; besides, an operand is held to 2^-148, and a sum below 2^-126 is a multiple of 2^-149."""
    nat = _native()
    torch.manual_seed(exponent)
    counts, k, n = [70, 300], 128, 192
    offs = _offs(counts)
    x, dy = torch.randn(370, k, device=DEV), torch.randn(370, n, device=DEV)
    w = torch.randn(2, n, k, device=DEV)
    for t in (x, dy) if which == "rows" else (w,):
        t *= 2.0 ** exponent
    y, dx, dw, db = (torch.empty(*size, device=DEV) for size in ((370, n), (370, k), (2, n, k), (2, n)))
    nat.split_grouped_gemm(0, x, w, offs, y, None, None)
    nat.split_grouped_gemm(1, dy, w, offs, dx, None, None)
    nat.split_grouped_gemm(2, dy, x if which == "weights" else x * 2.0 ** -exponent, offs, dw, None, db)
    if which == "rows":
        x_of_dw = x * 2.0 ** -exponent
    base = 0
    for e, c in enumerate(counts):
        s = slice(base, base + c)
        base += c
        X, D, W = x[s].double(), dy[s].double(), w[e].double()
        V = x_of_dw[s].double() if which == "rows" else X
        for got, ref, size, small, terms in [
                (y[s], X @ W.t(), X.abs() @ W.abs().t(), (X if which == "weights" else W).abs().max(), k),
                (dx[s], D @ W, D.abs() @ W.abs(), (D if which == "weights" else W).abs().max(), n),
                (dw[e], D.t() @ V, D.abs().t() @ V.abs(), V.abs().max(), c)]:
            bound = _bound(size, terms) + terms * (2.0 ** -148 * small + 2.0 ** -149)
            assert bool(((got.double() - ref).abs() <= bound).all()), float(((got.double() - ref).abs() / bound).max())
        bound = D.abs().sum(0) * (24 + c / 256) * 2.0 ** -24 + c * 2.0 ** -148
        assert bool(((db[e].double() - D.sum(0)).abs() <= bound).all())


@pytest.mark.parametrize("act", [nn.GELU(), nn.ReLU(), nn.GELU(approximate="tanh"), nn.Identity(),
                                 nn.Sequential(nn.ReLU(), nn.Dropout(0.0))])
@pytest.mark.parametrize("experts,k,d,h,tokens", [(4, 2, 64, 136, 300), (3, 1, 40, 72, 65), (8, 3, 128, 512, 1000)])
def test_fp32_layer_as_the_general_path(monkeypatch, act, experts, k, d, h, tokens):
    r"""Outputs and gradients of the one-call layer against 64 bits: no further off than the general
    path, up to what the last bits of single sums make of it."""
    from fastmoe_b200 import FMoETransformerMLP
    from fastmoe_b200.ops import fused
    torch.manual_seed(experts + tokens)
    moe = FMoETransformerMLP(num_expert=experts, d_model=d, d_hidden=h, top_k=k, activation=act).to(DEV)
    x = torch.randn(tokens, d, device=DEV)
    gy = torch.randn(tokens, d, device=DEV)
    ids, score = moe.gate(x)
    ids = torch.where(torch.rand(ids.shape, device=DEV) < 0.1, -1, ids)   # dropped slots
    score = score.detach()

    def run(module, dtype):
        leaves = {n: p.detach().to(dtype).requires_grad_(True) for n, p in module.experts.named_parameters()}
        xs, sc = (t.detach().to(dtype, copy=True).requires_grad_(True) for t in (x, score))
        if dtype == torch.float64:
            rows = []
            for e in range(experts):
                hid = act(xs @ leaves["htoh4.weight"][e].t() + leaves["htoh4.bias"][e])
                rows.append(hid @ leaves["h4toh.weight"][e].t() + leaves["h4toh.bias"][e])
            picked = torch.stack(rows)[ids.clamp(min=0), torch.arange(tokens, device=DEV)[:, None]]
            y = (picked * (sc * (ids >= 0))[..., None]).sum(1)
            y.backward(gy.to(dtype))
            grads = [leaves[n].grad for n in sorted(leaves)]
        else:
            module.zero_grad()
            y = module._fused_forward(xs, ids, sc)
            if y is None:
                y = module._general_path(xs, ids, sc)
            y.backward(gy)
            grads = [p.grad for n, p in sorted(module.experts.named_parameters())]
        return [y.detach(), xs.grad, sc.grad] + grads

    assert fused.supports(moe, x, ids)
    new = run(moe, torch.float32)
    monkeypatch.setenv("FMOE_FUSED", "0")
    assert not fused.supports(moe, x, ids)
    old = run(moe, torch.float32)
    ref = run(moe, torch.float64)
    for a, b, r in zip(new, old, ref):
        far = lambda t: float((t.double() - r).norm() / r.norm().clamp(min=1e-30))
        assert far(a) <= 1.1 * far(b) + 2.0 ** -24, (far(a), far(b))


def test_fp32_calls_that_keep_the_general_path(monkeypatch):
    from fastmoe_b200 import FMoETransformerMLP
    from fastmoe_b200.ops import fused
    moe = FMoETransformerMLP(num_expert=2, d_model=64, d_hidden=64, top_k=2).to(DEV)
    x = torch.randn(128, 64, device=DEV)
    ids = torch.zeros(128, 2, dtype=torch.long, device=DEV)
    assert fused.supports(moe, x, ids)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert not fused.supports(moe, x, ids)
    for module in (moe.experts, moe.experts.htoh4, moe.experts.activation):
        seen = []
        handle = module.register_forward_hook(lambda *_: seen.append(1))
        assert not fused.supports(moe, x, ids)
        moe(x)
        handle.remove()
        assert seen
    monkeypatch.setenv("FMOE_FASTER_SCHEDULE_ENABLE", "1")
    assert not fused.supports(moe, x, ids)
    monkeypatch.undo()
    moe.experts.htoh4.register_parameter("bias", None)
    assert not fused.supports(moe, x, ids)


def test_fp32_layer_in_a_graph_and_on_two_streams():
    from fastmoe_b200 import FMoETransformerMLP
    from fastmoe_b200.utils.graph import GraphedStep
    torch.manual_seed(1)
    moe = FMoETransformerMLP(num_expert=4, d_model=128, d_hidden=512, top_k=2).to(DEV)
    xs = [torch.randn(700, 128, device=DEV) for _ in range(2)]

    def step(x):
        moe.zero_grad(set_to_none=True)
        y = moe(x)
        y.square().sum().backward()
        return y.detach(), [p.grad for p in moe.parameters()]

    graphed = GraphedStep(step, xs[0])
    for x in xs:
        got = [t.clone() for t in [graphed(x)[0]] + graphed(x)[1]]
        y, grads = step(x)
        assert all(torch.equal(a, b) for a, b in zip(got, [y] + grads))
    streams = [torch.cuda.Stream() for _ in xs]
    torch.cuda.synchronize()
    with torch.no_grad():
        want = [moe(x) for x in xs]
        torch.cuda.synchronize()
        for _ in range(5):
            outs = []
            for s, x in zip(streams, xs):
                with torch.cuda.stream(s):
                    outs.append(moe(x))
            torch.cuda.synchronize()
            assert all(torch.equal(a, b) for a, b in zip(outs, want))


@pytest.mark.parametrize("act", [nn.GELU(), nn.GELU(approximate="tanh"), nn.ReLU(), nn.Identity()])
@pytest.mark.parametrize("constant", ["nothing", "scores", "experts", "input"])
def test_fp32_layer_gradient_of_the_gradient(act, constant):
    r"""Second and third derivatives against 64 bits; dropped slots, an expert without rows.  fp32 sums of at
    most 2 * 64 * 96 terms, several of them one after the other."""
    from fastmoe_b200 import FMoETransformerMLP
    from fastmoe_b200.ops import fused
    torch.manual_seed(4)
    moe = FMoETransformerMLP(num_expert=4, d_model=64, d_hidden=96, activation=act, top_k=2).to(DEV)
    nn.init.normal_(moe.experts.htoh4.bias)
    nn.init.normal_(moe.experts.h4toh.bias)
    base = [torch.randn(64, 64, device=DEV), torch.rand(64, 2, device=DEV)]
    base += [p.detach() for p in moe.experts.parameters()]
    ids = torch.randint(-1, 3, (64, 2), device=DEV)
    off = {"nothing": (), "scores": (1,), "experts": (2, 3, 4, 5), "input": (0,)}[constant]
    names = [n for n, _ in moe.experts.named_parameters()]

    def layer(x, score, *params):
        p = dict(zip(names, params))
        if x.dtype == torch.float32:
            from fastmoe_b200.ops import grouped_gemm as gg, native
            from fastmoe_b200.transformer import activation_kind
            return native.get().moe_mlp(x, score, p["htoh4.weight"], p["htoh4.bias"], p["h4toh.weight"],
                                        p["h4toh.bias"], ids, gg.ACT_CODES[activation_kind(act)], True)
        rows = torch.stack([act(x @ p["htoh4.weight"][e].t() + p["htoh4.bias"][e]) @ p["h4toh.weight"][e].t()
                            + p["h4toh.bias"][e] for e in range(4)])
        picked = rows[ids.clamp(min=0), torch.arange(64, device=DEV)[:, None]]
        return (picked * (score * (ids >= 0))[..., None]).sum(1)

    assert fused.supports(moe, base[0], ids, base[1])
    results = []
    for dtype in (torch.float32, torch.float64):
        t = [b.to(dtype, copy=True).requires_grad_(i not in off) for i, b in enumerate(base)]
        wanted = [v for i, v in enumerate(t) if i not in off]
        y = layer(*t)
        first = torch.autograd.grad((y.sin() * 0.5).sum(), wanted, create_graph=True)
        second = torch.autograd.grad(sum(g.square().sum() for g in first), wanted, create_graph=True, allow_unused=True)
        third = torch.autograd.grad(sum(g.square().sum() for g in second if g is not None), wanted, allow_unused=True)
        results.append([torch.zeros(()) if g is None else g.detach().double().cpu() for g in first + second + third])
    for got, want in zip(*results):
        assert float((got - want).norm()) <= 2e-5 * float(want.norm()) + 1e-12, (got.shape,)


def test_fp32_layer_input_changed_in_place_afterwards():
    r"""The backward does not read the input: with a frozen gate it may be changed, as it may around the general
    path; a gradient of the gradient does, and notices."""
    from fastmoe_b200 import FMoETransformerMLP
    torch.manual_seed(5)
    moe = FMoETransformerMLP(num_expert=4, d_model=64, d_hidden=96, top_k=2).to(DEV)
    moe.gate.requires_grad_(False)
    leaf = torch.randn(64, 64, device=DEV, requires_grad=True)
    want, = torch.autograd.grad((leaf * 1 + moe(leaf * 1)).sum(), leaf)
    x = leaf * 1
    x += moe(x)
    got, = torch.autograd.grad(x.sum(), leaf)
    assert torch.allclose(got, want, rtol=0, atol=1e-6)   # (sums of three terms in another order)
    x = leaf * 1
    x += moe(x)
    with pytest.raises(RuntimeError, match="inplace operation"):
        torch.autograd.grad(x.square().sum(), leaf, create_graph=True)


def test_fp32_layer_under_checkpointing_and_offloading():
    from torch.utils.checkpoint import checkpoint
    from fastmoe_b200 import FMoETransformerMLP
    torch.manual_seed(6)
    moe = FMoETransformerMLP(num_expert=4, d_model=64, d_hidden=96, top_k=2).to(DEV)
    x = torch.randn(64, 64, device=DEV, requires_grad=True)

    def offloaded(t):
        with torch.autograd.graph.save_on_cpu():
            return moe(t)
    results = []
    for run in (moe, lambda t: checkpoint(moe, t, use_reentrant=False), offloaded):
        moe.zero_grad(set_to_none=True)
        grads = torch.autograd.grad(run(x).square().sum(), [x] + list(moe.parameters()))
        first, = torch.autograd.grad(run(x).square().sum(), x, create_graph=True)
        twice = torch.autograd.grad(first.square().sum(), x)
        results.append(grads + twice)
    for other in results[1:]:
        for a, b in zip(other, results[0]):
            assert torch.allclose(a, b, rtol=1e-5, atol=1e-5 * float(b.abs().max()))
