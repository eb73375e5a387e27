r"""Which calls of the gates go to which kernels, on the CPU with stand-ins."""
import pytest
import torch
from torch.autograd import forward_ad

from fastmoe_b200.ops import gating, native


class _Kernels:
    @staticmethod
    def gate_fused_supported(_tot, _d, _k):
        return True

    @staticmethod
    def gate_linear_topk_node(*_args):
        return ["kernel"]


@pytest.fixture
def kernels(monkeypatch):
    monkeypatch.setattr(native, "get", _Kernels)
    monkeypatch.setattr(torch.Tensor, "is_cuda", True, raising=False)


def test_few_tokens_with_a_tangent_are_left_to_the_others(kernels):
    r"""The native call is no autograd function: it would return scores without the tangent."""
    x, w, b = torch.randn(4, 64).bfloat16(), torch.randn(16, 64).bfloat16(), torch.randn(16).bfloat16()
    with torch.no_grad(), forward_ad.dual_level():
        assert gating._few_tokens_ok(x, w, b, 2)
        dual = lambda t: forward_ad.make_dual(t, torch.ones_like(t))
        assert not gating._few_tokens_ok(dual(x), w, b, 2)
        assert not gating._few_tokens_ok(x, dual(w), b, 2)
        assert not gating._few_tokens_ok(x, w, dual(b), 2)


def test_switch_gate_calls_whatever_module_is_its_linear():
    from fastmoe_b200.gates import SwitchGate

    class Quantised(torch.nn.Module):   # as PyTorch's dynamically quantised linear, whose weight is a method
        def __init__(self, linear):
            super().__init__()
            self.held = linear

        def weight(self):
            return self.held.weight

        def forward(self, x):
            return self.held(x)
    torch.manual_seed(0)
    gate, x = SwitchGate(16, 4, 1).eval(), torch.randn(6, 16)
    want = gate(x)
    for module in (torch.nn.Sequential(gate.gate), Quantised(gate.gate)):
        gate.gate = module
        assert all(torch.equal(a, b) for a, b in zip(gate(x), want))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("what", ["input", "weight", "neither"])
def test_switch_gate_leaves_tensor_subclasses_to_the_linear(kernels, dtype, what):
    class Mine(torch.Tensor):
        pass
    linear, x = torch.nn.Linear(64, 4).to(dtype), torch.randn(6, 64).to(dtype)
    if what == "input":
        x = x.as_subclass(Mine)
    elif what == "weight":
        linear.weight = torch.nn.Parameter(linear.weight.detach().as_subclass(Mine))
        assert type(linear.weight) is not torch.nn.Parameter
    assert gating.linear_logits(x, linear) == (None if what != "neither" else "kernel")


@pytest.mark.parametrize("default", [torch.float32, torch.float64])
def test_naive_gate_under_function_transforms(default):
    from fastmoe_b200.gates import NaiveGate
    torch.manual_seed(0)
    gate, x = NaiveGate(16, 4, 1, 2).to(default), torch.randn(6, 16, dtype=default)
    params = {n: p.detach() for n, p in gate.named_parameters()}

    def loss(params, x):
        return torch.func.functional_call(gate, params, (x,))[1].square().sum()
    before = torch.get_default_dtype()
    torch.set_default_dtype(default)
    try:
        grad = torch.func.grad(loss)(params, x)
        each = torch.func.vmap(torch.func.grad(loss), (None, 0))(params, x[:, None])
        torch.func.jvp(lambda t: loss(params, t), (x,), (torch.ones_like(x),))
        gate(x)[1].square().sum().backward()
    finally:
        torch.set_default_dtype(before)
    for n, p in gate.named_parameters():
        assert torch.allclose(grad[n], p.grad, atol=1e-6) and torch.allclose(each[n].sum(0), p.grad, atol=1e-6)
    held = gate.get_loss()
    assert held.dtype == default and held.requires_grad and held.is_leaf and float(held.detach()) == 0
    with torch.inference_mode():
        gate(x)


@pytest.mark.parametrize("how", ["subclass", "instance"])
def test_naive_gate_with_another_choice(how):
    from fastmoe_b200.gates import NaiveGate

    class Worst(NaiveGate):
        def _choose(self, inp):
            logits, idx, score = super()._choose(inp)
            return logits, idx.flip(1), score
    torch.manual_seed(0)
    plain, x = NaiveGate(16, 4, 1, 2), torch.randn(6, 16)
    gate = Worst(16, 4, 1, 2) if how == "subclass" else NaiveGate(16, 4, 1, 2)
    gate.load_state_dict(plain.state_dict())
    if how == "instance":
        def choose(inp):
            logits, idx, score = NaiveGate._choose(gate, inp)
            return logits, idx.flip(1), score
        gate._choose = choose
    assert torch.equal(gate(x)[0], plain(x)[0].flip(1)) and float(gate.get_loss().detach()) == 0


@pytest.mark.parametrize("dtype,experts,tokens,d,grads,kernel", [
    (torch.bfloat16, 8, 64, 512, False, False), (torch.float16, 8, 8192, 4096, False, False),
    (torch.bfloat16, 8, 64, 512, True, True), (torch.bfloat16, 8, 4095, 1024, True, False),
    (torch.float16, 8, 4096, 1024, True, True), (torch.bfloat16, 8, 8192, 2048, True, False),
    (torch.bfloat16, 7, 64, 4096, False, True), (torch.bfloat16, 2, 1, 256, True, True),
    (torch.float32, 8, 64, 512, False, True)])
def test_switch_gate_linear_goes_where_it_is_faster(kernels, dtype, experts, tokens, d, grads, kernel):
    linear, x = torch.nn.Linear(d, experts).to(dtype), torch.zeros(tokens, d, dtype=dtype)
    with torch.set_grad_enabled(grads):
        assert gating.linear_logits(x, linear) == ("kernel" if kernel else None)
