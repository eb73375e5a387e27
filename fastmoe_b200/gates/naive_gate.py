r"""Plain learned top-k gate (parity: ``fmoe/gates/naive_gate.py:11-45``)."""
import torch
import torch.nn as nn

from .base_gate import BaseGate
from ..ops import gating


class NaiveGate(BaseGate):
    r"""``Linear(d_model → tot_expert)``, top-k of the logits, softmax over the k selected logits.

    State-dict keys: ``gate.weight [tot_expert, d_model]``, ``gate.bias [tot_expert]``.
    On a GPU with 16- or 32-bit parameters and at most 8 experts the linear layer, the top-k and the
    softmax are one kernel (three in backward); otherwise the top-k + softmax are.
    """

    def __init__(self, d_model, num_expert, world_size, top_k=2, gate_bias=True):
        super().__init__(num_expert, world_size)
        self.gate = nn.Linear(d_model, self.tot_expert, bias=gate_bias)
        self.top_k = top_k

    def _choose(self, inp, zero=None):
        linear = self.gate
        return gating.linear_topk_softmax(
            inp if inp.dim() == 2 else inp.reshape(-1, inp.shape[-1]), linear.weight, linear.bias, self.top_k, zero)

    def forward(self, inp, return_all_scores=False):
        # The reference installs a zero "dummy" loss so that callers can always add it.
        # (made a leaf at once: transforms of torch.func do not let it become one later)
        loss = torch.empty(1, device=inp.device, requires_grad=True)
        zero = loss.detach()
        if zero.dtype == torch.float32 and type(self)._choose is NaiveGate._choose and "_choose" not in vars(self):
            logits, idx, score = self._choose(inp, zero)
        else:
            logits, idx, score = self._choose(inp)
            zero.zero_()
        self.set_loss(loss)
        if return_all_scores:
            return idx, score, logits.view(*inp.shape[:-1], self.tot_expert)
        return idx, score
