r"""GPU tier: the general path's row kernels against its PyTorch operations (``FMOE_FUSED=0``)."""
import pytest
import torch
import torch.nn as nn

pytestmark = pytest.mark.gpu

DEV = "cuda"


class _Expert(nn.Module):
    def __init__(self, d, out, kind):
        super().__init__()
        self.fc, self.kind = nn.Linear(d, out), kind

    def forward(self, x, _count):
        if self.kind == "inplace":
            x = x.mul_(2.0)
        elif self.kind == "doubled":
            x = x * 2.0
        y = torch.tanh(self.fc(x))
        if self.kind == "dict":
            return {"y": y, "s": y.sum(1, keepdim=True)}
        return y.unsqueeze(1).expand(-1, 2, -1) if self.kind == "3d" else y


def _layer(experts, d, out, k, kind, dtype):
    from fastmoe_b200 import FMoE
    torch.manual_seed(0)
    return FMoE(num_expert=experts, d_model=d, top_k=k, expert=lambda width: _Expert(width, out, kind)).to(DEV).to(dtype)


def _run(layer, x, ids, scores, gy):
    layer.zero_grad()
    x, scores = x.detach().clone().requires_grad_(True), scores.detach().clone().requires_grad_(True)
    out = layer._general_path(x, ids, scores)
    out.backward(gy)
    return [out.detach(), x.grad, scores.grad] + [p.grad for p in layer.experts.parameters()]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens,d,out,experts,k,kind", [
    (1, 8, 8, 1, 1, "plain"),           # the smallest
    (257, 64, 40, 5, 3, "plain"),       # another width behind the experts
    (300, 1032, 264, 4, 6, "inplace"),  # more than four choices, rows of more than one step per warp
    (64, 16, 24, 3, 2, "odd"),
])
def test_rows_as_the_operations(monkeypatch, dtype, tokens, d, out, experts, k, kind):
    r"""Up to the rounding of 16-bit sums, which the operations round after every addition and the kernels
    once: k + 1 of them, relative to the magnitudes that are summed."""
    layer = _layer(experts, d, out, k, kind, dtype)
    torch.manual_seed(1)
    x = torch.randn(tokens, d, device=DEV, dtype=dtype)
    ids = torch.randint(-1, experts, (tokens, k), device=DEV)
    if kind == "odd":
        ids[::7] = experts + 5   # names no expert: dropped, as by the operations
        ids[1::7] = -1
    scores = torch.rand(tokens, k, device=DEV, dtype=dtype)
    gy = torch.randn(tokens, out, device=DEV, dtype=dtype)
    got = _run(layer, x, ids, scores, gy)
    monkeypatch.setenv("FMOE_FUSED", "0")
    if kind == "inplace":   # slices of one buffer share a version counter: autograd refuses them
        for e in layer.experts:
            e.kind = "doubled"
    ref = _run(layer, x, ids, scores, gy)
    eps = torch.finfo(dtype).eps
    for a, b in zip(got, ref):
        assert a.shape == b.shape and a.dtype == b.dtype
        scale = float(b.float().abs().max()) + 1e-6
        assert float((a.float() - b.float()).abs().max()) <= (k + 2) * 8 * eps * scale


def test_general_path_of_other_outputs_and_no_rows(monkeypatch):
    from fastmoe_b200 import FMoE
    layer = _layer(3, 16, 24, 2, "3d", torch.float32)
    x = torch.randn(50, 16, device=DEV)
    ids = torch.randint(-1, 3, (50, 2), device=DEV)
    scores = torch.rand(50, 2, device=DEV)
    for kind in ("dict", "plain"):
        layer = _layer(3, 16, 24, 2, kind, torch.float32)
        for chosen in (ids, torch.full_like(ids, -1)):
            got = layer._general_path(x, chosen, scores)
            with monkeypatch.context() as m:
                m.setenv("FMOE_FUSED", "0")
                ref = layer._general_path(x, chosen, scores)
            for a, b in zip(got.values() if kind == "dict" else [got], ref.values() if kind == "dict" else [ref]):
                assert torch.allclose(a, b, rtol=1e-6, atol=1e-6)
    # a fused expert module whose rows come in another type than the input
    class Wide(FMoE):
        def expert_fn(self, inp, fwd_expert_count):
            return inp.double()
    wide = Wide(num_expert=3, d_model=16, top_k=2, expert=lambda d: nn.Linear(d, d)).to(DEV)
    out = wide._general_path(x, ids, scores)
    assert out.dtype == torch.float64
    ref = (x[:, None].double() * (scores * (ids >= 0))[..., None].double()).sum(1)
    assert torch.allclose(out, ref)


def test_gradient_of_the_gradient(monkeypatch):
    layer = _layer(3, 16, 16, 2, "plain", torch.float32)
    torch.manual_seed(2)
    x0 = torch.randn(40, 16, device=DEV)
    ids = torch.randint(-1, 3, (40, 2), device=DEV)
    s0 = torch.rand(40, 2, device=DEV)
    results = []
    for fused in ("1", "0"):
        monkeypatch.setenv("FMOE_FUSED", fused)
        x, s = x0.clone().requires_grad_(True), s0.clone().requires_grad_(True)
        out = layer._general_path(x, ids, s)
        gx, gs = torch.autograd.grad(out.square().sum(), (x, s), create_graph=True)
        layer.zero_grad()
        (gx.square().sum() + gs.square().sum()).backward()
        results.append([x.grad, s.grad] + [p.grad.clone() for p in layer.experts.parameters()])
    for a, b in zip(*results):
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("constant", ["scores", "rows"])
def test_gradient_of_the_gradient_beside_constants(monkeypatch, constant):
    layer = _layer(3, 16, 16, 2, "plain", torch.float32)
    torch.manual_seed(2)
    x0, s0 = torch.randn(40, 16, device=DEV), torch.rand(40, 2, device=DEV)
    ids = torch.randint(-1, 3, (40, 2), device=DEV)
    layer.experts.requires_grad_(constant != "rows")
    results = []
    for fused in ("1", "0"):
        monkeypatch.setenv("FMOE_FUSED", fused)
        x, s = x0.clone().requires_grad_(constant != "rows"), s0.clone().requires_grad_(constant != "scores")
        leaf = s if constant == "rows" else x
        first, = torch.autograd.grad(layer._general_path(x, ids, s).square().sum(), leaf, create_graph=True)
        results.append((first.detach(),) + torch.autograd.grad(first.square().sum(), leaf))
    for a, b in zip(*results):
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("groups", [1, 79, 80, 255, 959, 960, 3000])   # parameters of 80 and 960 values, the copy
def test_offsets_of_host_counts(groups):
    from fastmoe_b200.ops import grouped_gemm as gg
    counts = torch.randint(0, 50, (groups,), generator=torch.Generator().manual_seed(groups))
    want = torch.cat([torch.zeros(1, dtype=torch.int64), counts.cumsum(0)]).int()
    for given in (counts, counts.int(), counts.tolist(), torch.stack([counts, counts], 1)[:, 0]):
        offs = gg.offsets_from_counts(given, "cuda")
        assert offs.is_cuda and offs.dtype == torch.int32 and torch.equal(offs.cpu(), want)
    kept = counts.clone()
    offs = gg.offsets_from_counts(kept, torch.device("cuda", 0))
    kept.zero_()   # the call has taken what it needs
    assert torch.equal(offs.cpu(), want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("kind", ["column", "one value"])
def test_scores_need_not_lie_next_to_each_other(dtype, kind):
    from fastmoe_b200 import FMoETransformerMLP
    general = _layer(3, 64, 64, 1, "plain", dtype)
    between = FMoETransformerMLP(3, 64, 64, nn.Tanh(), top_k=1).to(DEV).to(dtype)   # no fused activation
    torch.manual_seed(3)
    x = torch.randn(50, 64, device=DEV, dtype=dtype)
    ids = torch.randint(-1, 3, (50, 1), device=DEV)
    table = torch.rand(*((50, 5) if kind == "column" else (1, 1)), device=DEV, dtype=dtype)
    for run in [general._general_path] + ([between._fused_forward] if dtype != torch.float32 else []):
        results = []
        for apart in (True, False):
            leaf = table.clone().requires_grad_(True)
            scores = leaf[:, :1] if kind == "column" else leaf.expand(50, 1)
            out = run(x, ids, scores if apart else scores.contiguous())
            out.sum().backward()
            results.append((out.detach(), leaf.grad))
        for a, b in zip(*results):
            assert torch.equal(a, b)


def test_row_kernels_refuse_slot_tables_that_do_not_fit():
    from fastmoe_b200.ops import native
    nat = native.get()
    rows, out = torch.zeros(8, 64, device=DEV), torch.zeros(4, 64, device=DEV)
    idx = torch.zeros(8, device=DEV, dtype=torch.int64)
    _counts, rank, offs = nat.route_offs(idx, 1)
    score = torch.ones(8, 2, device=DEV)
    for bad in (score[:, 0], score[:4, 0].contiguous(), score[:, 0].contiguous().double(), torch.ones(8)):
        with pytest.raises(RuntimeError):
            nat.gather_combine(rows, idx, rank, offs, bad, 2, out)
        with pytest.raises(RuntimeError):
            nat.combine_bwd(out, rows, idx, rank, offs, bad, 2, rows.clone(), torch.ones(8, device=DEV))
    for k, table in ((1, idx), (2, idx[:4]), (2, idx.cpu())):
        with pytest.raises(RuntimeError):
            nat.gather_combine(rows, table, rank, offs, None, k, out)
        with pytest.raises(RuntimeError):
            nat.scatter_rows(out, table, rank, offs, None, k, rows, None)
