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


def _block_backward(softmax):
    B, S, H, D = 2, 20, 3, 64
    lse = _zeros(*((B, H, S) if softmax else (0,)), dtype=torch.float32)
    return dict(qkv=_zeros(B, S, 3 * H * D), qk=_zeros(2, B, S, H, D), out=_zeros(B, S, H * D), lse=lse,
                dout=_zeros(B, S, H * D), table=_zeros(S, D, dtype=torch.float32), num_registers=2, softmax=softmax)


@pytest.mark.gpu
@pytest.mark.parametrize("softmax", [True, False])
def test_the_blocks_backward_takes_tensors_of_one_size(softmax):
    op = torch.ops.rbf_attn_b200.susie_block_bwd
    good = _block_backward(softmax)
    dqkv, d_pw, d_rp = op(**good)
    assert dqkv.shape == good["qkv"].shape and d_pw.shape == (3, 32) and d_rp.shape == (3, 2, 64)
    lse = good["lse"]
    bad = [{name: good[name][:, :-1]} for name in ("qkv", "out", "dout", "qk")] + [{name: good[name][:1]} for name in
           ("qkv", "out", "dout", "qk")] + [{name: good[name][..., :-8]} for name in ("qkv", "out", "dout")]
    bad += [{"qk": good["qk"][0]}, {"qk": good["qk"][..., :32]}, {"qk": good["qk"].half()}, {"out": good["out"].float()},
            {"table": good["table"][:17]}, {"num_registers": 21}, {"num_registers": -1}, {"qkv": good["qkv"].float()},
            {"dout": good["dout"].cpu()}, {"out": good["out"].cpu()}, {"qkv": good["qkv"].cpu()}]
    if softmax:
        bad += [{"lse": lse[:, :, :-1]}, {"lse": lse[:0]}, {"lse": lse.double()}, {"lse": lse.cpu()}]
    for change in bad:
        with pytest.raises((RuntimeError, ValueError)):
            op(**{**good, **change})
    op(**{**good, "dout": good["dout"].float(), "qkv": good["qkv"].view(40, -1), "table": good["table"][:18]})
    ops.check_device_status()


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(4, 0), (0,), (2, 3, 0), ()])
def test_gradients_over_no_columns_are_refused(shape):
    x, w, stat = _zeros(*shape), _zeros(0), _zeros(4, dtype=torch.float32)
    op = torch.ops.rbf_attn_b200
    for call in (lambda: op.gelu_bwd(x, x, True), lambda: op.gelu_bwd(x, x, False), lambda: op.layer_norm_bwd(x, x, w, stat, stat),
                 lambda: op.layer_norm_bwd_add(x, x, x, w, stat, stat)):
        with pytest.raises(ValueError, match="no columns"):
            call()
