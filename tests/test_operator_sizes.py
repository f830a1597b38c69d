"""Operator calls whose tensors do not have the sizes that the kernels walk: refused on the host, before any pointer is taken."""

import pytest
import torch

from rbf_attention_b200 import _lib, ops
from rbf_attention_b200.attention import CustomCausalAttention

DEV = "cuda:0"


def _zeros(*shape, dtype=torch.bfloat16):
    return torch.zeros(shape, dtype=dtype, device=DEV)


@pytest.mark.gpu
@pytest.mark.parametrize("heads,width", [(16, 1032), (12, 776), (9, 1160)])
@pytest.mark.parametrize("kind", ["rbf_triton", "rbf_non_softmax"])
def test_a_width_that_the_heads_do_not_divide_is_refused(kind, heads, width):
    """Head dims of 64 or 128 and a remainder of whole 16-byte chunks."""
    with torch.device(DEV):
        block = CustomCausalAttention(heads, width, max_seq_len=32, attention_type=kind, num_registers=2)
    block = block.to(torch.bfloat16)
    x = _zeros(2, 20, width)
    with torch.no_grad(), pytest.raises(RuntimeError):
        block(x)
    with pytest.raises(RuntimeError):
        block(x.requires_grad_(True))


@pytest.mark.gpu
@pytest.mark.parametrize("rest", [1, 2, 8, 24, -1])
@pytest.mark.parametrize("heads", [1, 2, 16])
def test_the_block_takes_three_times_its_heads_columns(heads, rest):
    pw, table = _zeros(heads, 32), _zeros(20, 64, dtype=torch.float32)
    qkv = _zeros(2, 20, 3 * heads * 64 + rest)
    for call in (_lib.host().block_fwd, torch.ops.rbf_attn_b200.susie_block_fwd, ops.susie_block_attention):
        with pytest.raises((RuntimeError, ValueError)):
            call(qkv, pw, None, table, heads, True)
