"""Layers over no rows at all: nothing to compute, and gradients of parameters that are zero and not what lay in their memory."""

import pytest
import torch

from rbf_attention_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("columns", [8, 264, 512])
def test_parameter_gradients_of_an_empty_batch_are_zero(columns):
    for fill in (float("nan"), 7.0):
        torch.full((1 << 16,), fill, device="cuda")             # freed at once: what the next allocations find
        up, down = (torch.nn.Linear(columns, columns, device="cuda", dtype=torch.bfloat16) for _ in range(2))
        x = torch.empty(0, columns, device="cuda", dtype=torch.bfloat16, requires_grad=True)
        out = ops.linear(down, ops.linear_gelu(up, x))
        grads = torch.autograd.grad(out, [x, *up.parameters(), *down.parameters()], torch.ones_like(out))
        torch.full((columns,), fill, device="cuda")
        _, sums = torch.ops.rbf_attn_b200.gelu_bwd(x.detach(), x.detach(), True)
        for g in (*grads, sums, torch.ops.rbf_attn_b200.column_sums(x.detach())):
            assert not g.count_nonzero()
    if columns % 256 == 0:
        stat = torch.empty(0, device="cuda")
        w = torch.ones(columns, device="cuda", dtype=torch.bfloat16)
        for g in torch.ops.rbf_attn_b200.layer_norm_bwd(x.detach(), x.detach(), w, stat, stat):
            assert not g.count_nonzero()
