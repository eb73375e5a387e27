r"""The glue around the general path's row kernels, with a stand-in for the kernels that runs on the CPU
and, as they do, reads its operands through their pointers."""
import pytest
import torch
import torch.nn as nn
from torch.autograd import forward_ad

from fastmoe_b200 import FMoE
from fastmoe_b200.ops import fused, native, torch_impl


def _flat(t, n):
    r"""What a kernel sees at ``t.data_ptr()``: ``n`` values in a row (an error where the storage is shorter)."""
    return torch.as_strided(t, (n,), (1,))


class _Kernels:
    @staticmethod
    def route_pos(idx, tot):
        counts = torch_impl.expert_count(idx, tot).to(torch.int32)
        rank = torch_impl.slot_rank(idx, tot).reshape(-1).to(torch.int32)
        offs = torch.zeros(tot + 1, dtype=torch.int32)
        offs[1:] = counts.cumsum(0)
        pos = torch_impl.assign_pos(idx, tot).to(torch.int32)
        return counts, rank, offs, pos

    @staticmethod
    def _rows(idx, rank, offs):
        kept = rank >= 0
        return kept, (offs[idx.clamp(min=0)] + rank)[kept].long()

    def scatter_rows(self, src, idx, rank, offs, _scale, k, dst, _row_slot):
        kept, row = self._rows(idx, rank, offs)
        dst[row] = src.repeat_interleave(k, 0)[kept]

    def gather_combine(self, rows, idx, rank, offs, weight, k, out):
        kept, row = self._rows(idx, rank, offs)
        slots = torch.zeros(idx.numel(), rows.shape[1], dtype=rows.dtype)
        slots[kept] = rows[row]
        if weight is not None:
            slots = slots * _flat(weight, idx.numel())[:, None]
        out.copy_(slots.view(out.shape[0], k, -1).sum(1))

    def combine_bwd(self, dout, rows, idx, rank, offs, weight, k, drows, dscore):
        kept, row = self._rows(idx, rank, offs)
        g = dout.repeat_interleave(k, 0)
        drows[row] = (g * _flat(weight, idx.numel())[:, None])[kept]
        ds = _flat(dscore, idx.numel())
        ds.zero_()
        ds[kept] = (g[kept] * rows[row]).sum(1)

    @staticmethod
    def moe_mlp_supported_f32(*_sizes):
        return True

    @staticmethod
    def moe_mlp(*_args):
        raise AssertionError("the layer's kernels were launched")


@pytest.fixture(autouse=True)
def kernels(monkeypatch):
    monkeypatch.setattr(native, "get", _Kernels)
    monkeypatch.setattr(native, "available", lambda: True)


class _Expert(nn.Module):
    def __init__(self, d):
        super().__init__()
        self.fc = nn.Linear(d, d)

    def forward(self, x, _count):
        return torch.tanh(self.fc(x))


def _layer(experts=3, d=16, k=2, cls=FMoE, expert=_Expert):
    torch.manual_seed(0)
    return cls(num_expert=experts, d_model=d, top_k=k, expert=expert).double()


def _general(layer, x, ids, scores):
    return fused.general_path(x, ids, scores, layer.expert_fn, layer.num_expert)[0]


@pytest.fixture(autouse=True)
def any_type(monkeypatch):
    monkeypatch.setattr(fused, "_TC", (torch.float64,))
    monkeypatch.setattr(torch.Tensor, "is_cuda", True, raising=False)


@pytest.mark.parametrize("kind", ["column", "one value"])
def test_scores_need_not_lie_next_to_each_other(kind):
    layer = _layer(k=1)
    torch.manual_seed(1)
    x, ids = torch.randn(10, 16, dtype=torch.float64), torch.randint(0, 3, (10, 1))
    table = torch.rand(10, 5, dtype=torch.float64) if kind == "column" else torch.rand(1, 1, dtype=torch.float64)
    results = []
    for apart in (True, False):
        leaf = table.clone().requires_grad_(True)
        scores = leaf[:, :1] if kind == "column" else leaf.expand(10, 1)
        assert scores.reshape(-1).is_contiguous() is False
        out = _general(layer, x, ids, scores if apart else scores.contiguous())
        out.square().sum().backward()
        results.append((out.detach(), leaf.grad))
    for a, b in zip(*results):
        assert torch.equal(a, b)


@pytest.mark.parametrize("what", ["fits", "one score per token", "more choices than the layer's", "scores elsewhere",
                                  "ids elsewhere"])
def test_fp32_layer_looks_at_what_the_gate_returned(what):
    from fastmoe_b200 import FMoETransformerMLP
    layer = FMoETransformerMLP(num_expert=3, d_model=16, d_hidden=16, top_k=2)
    x, ids, scores = torch.randn(10, 16), torch.randint(0, 3, (10, 2)), torch.rand(10, 2)
    if what == "one score per token":
        scores = scores[:, :1]
    elif what == "more choices than the layer's":
        ids, scores = ids.repeat(1, 2), scores.repeat(1, 2)
    elif what == "scores elsewhere":
        scores = scores.to("meta")
    elif what == "ids elsewhere":
        ids = ids.to("meta")
    if what == "fits":
        with pytest.raises(AssertionError, match="kernels were launched"):
            layer._fused_forward(x, ids, scores)
    else:
        assert layer._fused_forward(x, ids, scores) is None


@pytest.mark.parametrize("constant", ["neither", "scores", "rows"])
@pytest.mark.parametrize("dropped", ["some", "all"])
def test_gradient_of_the_gradient(constant, dropped, monkeypatch):
    r"""In 64 bits against the path of PyTorch operations."""
    layer = _layer()
    torch.manual_seed(2)
    x0, s0 = torch.randn(10, 16, dtype=torch.float64), torch.rand(10, 2, dtype=torch.float64)
    ids = torch.randint(-1, 3, (10, 2)) if dropped == "some" else torch.full((10, 2), -1)
    if constant == "rows":
        layer.experts.requires_grad_(False)

    def operations(*args):
        with monkeypatch.context() as m:
            m.setenv("FMOE_FUSED", "0")
            return layer._general_path(*args)
    results = []
    for run in (lambda *args: _general(layer, *args), operations):
        x, s = x0.clone().requires_grad_(constant != "rows"), s0.clone().requires_grad_(constant != "scores")
        wanted = [t for t in (x, s) if t.requires_grad]
        params = [p for p in layer.parameters() if p.requires_grad and p.dim() == 2]
        first = torch.autograd.grad(run(x, ids, s).square().sum(), wanted, create_graph=True, allow_unused=True)
        total = sum(g.square().sum() for g in first if g is not None)
        second = torch.autograd.grad(total, wanted + params, allow_unused=True)
        results.append([torch.zeros(()).double() if g is None else g.detach() for g in list(first) + list(second)])
    for a, b in zip(*results):
        assert float((a - b).abs().max()) <= 1e-9 * (1 + float(b.abs().max()))


@pytest.mark.parametrize("how", ["subclass", "instance"])
def test_fp32_layer_calls_another_expert_fn(how):
    from fastmoe_b200 import FMoETransformerMLP

    class Doubled(FMoETransformerMLP):
        def expert_fn(self, inp, fwd_expert_count):
            return super().expert_fn(inp, fwd_expert_count) * 2
    layer = (Doubled if how == "subclass" else FMoETransformerMLP)(num_expert=3, d_model=16, d_hidden=16, top_k=2)
    if how == "instance":
        layer.expert_fn = lambda inp, count: layer.experts(inp, count) * 2
    assert layer._fused_forward(torch.randn(10, 16), torch.randint(0, 3, (10, 2)), torch.rand(10, 2)) is None


class _InPlace(_Expert):
    def forward(self, x, _count):
        return torch.tanh(self.fc(x.mul_(2.0)))


def test_rows_that_another_expert_fn_saves_are_watched():
    r"""Experts that write to their rows, and an ``expert_fn`` that has used the rows before: autograd
    has to notice, as it does with slices."""
    class Shared(FMoE):
        def expert_fn(self, inp, fwd_expert_count):
            return self.shared(inp) + super().expert_fn(inp, fwd_expert_count)
    layer = _layer(cls=Shared, expert=_InPlace)
    layer.shared = nn.Linear(16, 16).double()
    torch.manual_seed(4)
    x, ids, scores = torch.randn(10, 16).double(), torch.randint(0, 3, (10, 2)), torch.rand(10, 2).double()
    out = layer._general_path(x.requires_grad_(True), ids, scores)
    with pytest.raises(RuntimeError, match="inplace operation"):
        out.sum().backward()
    # nobody else holds the rows of the usual one: its experts may write to them
    plain = _layer(expert=_InPlace)
    results = []
    for module, rows in ((plain, x), (_layer(), x * 2.0)):
        module.load_state_dict(plain.state_dict())
        module.zero_grad()
        module._general_path(rows, ids, scores).sum().backward()
        results.append([p.grad for p in module.experts.parameters()])
    assert all(torch.allclose(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("path", ["custom experts", "fp32 layer"])
def test_subclasses_and_tangents_of_scores_keep_the_operations(path, monkeypatch):
    from fastmoe_b200 import FMoETransformerMLP

    class Mine(torch.Tensor):
        pass
    dtype = torch.float64 if path == "custom experts" else torch.float32
    torch.manual_seed(5)
    x, ids, scores = torch.randn(10, 16, dtype=dtype), torch.randint(0, 3, (10, 2)), torch.rand(10, 2, dtype=dtype)
    if path == "custom experts":
        layer = _layer()
        taken = lambda x, scores: fused.rows_supported(x, ids, scores)
    else:
        layer = FMoETransformerMLP(num_expert=3, d_model=16, d_hidden=16, top_k=2)
        taken = lambda x, scores: fused.supports(layer, x, ids, scores)
    assert taken(x, scores)
    assert not taken(x.as_subclass(Mine), scores)
    assert not taken(x, scores.as_subclass(Mine))
    monkeypatch.delattr(torch.Tensor, "is_cuda")
    with torch.no_grad(), forward_ad.dual_level():   # the derivative is that of a sum linear in the scores
        out = layer._general_path(x, ids, forward_ad.make_dual(scores, scores))
        assert torch.allclose(*forward_ad.unpack_dual(out))
    monkeypatch.setattr(torch.Tensor, "is_cuda", True, raising=False)
    with torch.no_grad(), forward_ad.dual_level():
        assert not taken(x, forward_ad.make_dual(scores, scores))
