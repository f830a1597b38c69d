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


def _refused(call, good, bad):
    call(**good)
    for change in bad:
        with pytest.raises((RuntimeError, ValueError)):
            call(**{**good, **change})
    ops.check_device_status()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_attention_gradients_take_an_output_and_statistics_of_q(dtype):
    t, lse = _zeros(2, 3, 70, 64, dtype=dtype), _zeros(2, 3, 70, dtype=torch.float32)
    good = dict(q=t, k=t, v=t, out=t, L=lse, dout=t, is_causal=True, sm_scale=0.125)
    outs = [{"out": o} for o in (t[:, :, :-1], t[:1], t[..., :32], t[0], t.cpu())]
    _refused(torch.ops.rbf_attn_v5.scaled_bwd, good, outs + [{"L": x} for x in (lse[:, :, :-1], lse[:1], lse.half(), lse.cpu())])
    wide = torch.zeros(2, 3, 140, device=DEV)[:, :, ::2]
    torch.ops.rbf_attn_v5.scaled_bwd(**{**good, "L": wide, "out": t.half()})
    good = {name: good[name] for name in ("q", "k", "v", "out", "dout", "is_causal", "sm_scale")}
    _refused(torch.ops.rbf_attn_v5.non_softmax_bwd_with_out, good, outs)


@pytest.mark.gpu
def test_statistics_in_any_layout_give_the_same_gradients():
    g = torch.Generator(device=DEV).manual_seed(0)
    q, k, v, do = ((torch.randn(2, 3, 70, 64, generator=g, device=DEV) * 0.5).half() for _ in range(4))
    out, lse = torch.ops.rbf_attn_v5.scaled_fwd(q, k, v, True)
    strided = torch.stack((lse, -lse), -1)[..., 0]
    want = torch.ops.rbf_attn_v5.scaled_bwd(q, k, v, out, lse, do, True, 0.125)
    for a, b in zip(torch.ops.rbf_attn_v5.scaled_bwd(q, k, v, out, strided, do, True, 0.125), want):
        assert (a.double() - b.double()).norm() <= 1e-3 * b.double().norm()         # the order of dQ's fp32 additions


@pytest.mark.gpu
def test_the_block_takes_positions_of_its_heads():
    good = dict(qkv=_zeros(2, 20, 3 * 2 * 64), pos_weight=_zeros(2, 32), reg_pos_emb=_zeros(2, 4, 64),
                table=_zeros(16, 64, dtype=torch.float32), num_heads=2, softmax=True)
    _refused(torch.ops.rbf_attn_b200.susie_block_fwd, good,
             [{"pos_weight": _zeros(1, 32)}, {"pos_weight": _zeros(2, 16)}, {"pos_weight": good["pos_weight"].cpu()},
              {"reg_pos_emb": _zeros(1, 4, 64)}, {"reg_pos_emb": _zeros(2, 4, 32)}, {"reg_pos_emb": good["reg_pos_emb"].cpu()},
              {"table": good["table"][:15]}, {"table": good["table"][:, :32]}])


@pytest.mark.gpu
def test_layer_norms_take_parameters_and_gradients_of_their_columns():
    x, w, stat = _zeros(6, 512), _zeros(512), _zeros(6, dtype=torch.float32)
    params = [{name: t} for name in ("weight", "bias") for t in (w[:256], _zeros(1024), w.cpu(), w.float())]
    op = torch.ops.rbf_attn_b200
    _refused(op.layer_norm_fwd, dict(x=x, weight=w, bias=w, eps=1e-5), params)
    _refused(op.add_layer_norm_fwd, dict(x=x, residual=x, weight=w, bias=w, eps=1e-5), params + [{"residual": x[:5]}])
    bad = [{"dy": x[:5]}, {"dy": x[:, :256]}, {"dy": x.cpu()}, {"weight": w[:256]}, {"weight": w.float()}, {"weight": w.cpu()},
           {"x": x.float()}]
    bad += [{name: t} for name in ("mean", "rstd") for t in (stat[:5], stat.half(), stat.cpu())]
    good = dict(x=x, dy=x, weight=w, mean=stat, rstd=stat)
    _refused(op.layer_norm_bwd, good, bad)
    _refused(op.layer_norm_bwd_add, dict(good, dres=x), bad + [{"dres": x[:5]}, {"dres": x.cpu()}])


@pytest.mark.gpu
def test_exclusive_self_attention_takes_one_shape():
    t = _zeros(2, 3, 50, 64)
    bad = [{"v": t[:, :, :-1]}, {"v": t[:1]}, {"v": t.half()}, {"v": t.cpu()}]
    _refused(torch.ops.rbf_attn_b200.xsa_fwd, dict(o=t, v=t), bad)
    _refused(torch.ops.rbf_attn_b200.xsa_bwd, dict(g=t, o=t, v=t), bad + [{"g": t[:, :, :-1]}, {"g": t.cpu()}])


def test_the_extensions_rules_are_the_ones_python_uses(built_library):
    with pytest.raises(TypeError, match="k must be a tensor"):
        ops._validate("k", None)
    with pytest.raises(ValueError, match="q must have shape"):
        ops._validate("q", torch.zeros(3, 64))
    with pytest.raises(RuntimeError, match="q must be a CUDA tensor"):
        ops._validate("q", torch.zeros(1, 2, 3, 64))
    dense = torch.zeros(2, 3, 40, 64, dtype=torch.bfloat16)
    heads_last = dense.permute(0, 2, 1, 3)
    assert ops._tma_ready(dense) is dense and ops._tma_ready(heads_last) is heads_last
    for t in (dense[..., 1:], dense[..., ::2], dense[:, :, :1].expand(2, 3, 40, 64), torch.zeros(2, 3, 40, 36).half()[..., :33]):
        ready = ops._tma_ready(t)
        assert ready.is_contiguous() and ready.shape == t.shape and ready is not t
    with pytest.raises(ValueError, match="at most 128"):
        _lib.host().narrow_f32([torch.zeros(1, 1, 4, 136)], 1)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_head_dims_above_128_are_refused_before_anything_runs(dtype):
    t = _zeros(1, 2, 16, 136, dtype=dtype)
    mon = ops._monitor(t.device)
    ops.check_device_status()
    for call in (lambda: ops._forward(t, t, t, True, True), lambda: ops._backward(t, t, t, t, t[..., 0].float(), t, True, 0.1, True)):
        with pytest.raises(ValueError, match="at most 128"):
            call()
    assert len(mon.free) == mon.SLOTS
