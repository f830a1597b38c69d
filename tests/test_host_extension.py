"""The extension that prepares and enqueues operator calls (csrc/host.cpp): arguments that it refuses, and views that it has
to copy or pad before the kernels can read them, against the same values laid out densely."""

import pytest
import torch

from rbf_attention_b200 import _lib, ops


def test_bad_arguments_raise(built_library):
    host = _lib.host()
    q = torch.zeros(1, 2, 3, 64)
    with pytest.raises(TypeError, match="expected 5 arguments, got 3"):
        host.attention_fwd(q, q, q)
    with pytest.raises(TypeError, match="q must be a tensor"):
        host.attention_fwd(1, q, q, True, True)
    with pytest.raises(ValueError, match="must have shape"):
        host.attention_fwd(q[0], q, q, True, True)
    with pytest.raises(RuntimeError, match="no CPU path"):
        host.attention_bwd(q, q, q, None, None, q, True, 0.125, True)
    with pytest.raises(RuntimeError, match="no CPU path"):
        host.block_fwd(q[0], q, None, q, 2, True)
    with pytest.raises(ValueError):
        host.column_sums(q)
    with pytest.raises(ValueError):
        host.gelu_fwd(q)
    with pytest.raises(ValueError, match="256, 512, 768 or 1024 columns"):
        host.layer_norm_fwd(q, None, q, q, 1e-5)
    assert host.narrow_f32([q], 1) is None          # not on a GPU: left to PyTorch
    with pytest.raises(TypeError):
        host.narrow_f32([1], 1)
    with pytest.raises(ValueError):
        host.widen_f16([])


def _view(kind, shape, dtype, seed):
    """The values of one tensor in a layout of its own; NaN where the kernels must not read."""
    B, H, N, D = shape
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = (torch.randn(shape, generator=g, device="cuda") * 0.7).to(dtype)
    if kind == "heads last":
        return x.permute(0, 2, 1, 3).contiguous().permute(0, 2, 1, 3)
    if kind == "columns apart":
        buf = torch.full((B, H, N, 2 * D), float("nan"), dtype=dtype, device="cuda")
        return buf[..., ::2].copy_(x)
    if kind == "wide rows":
        buf = torch.full((B, H, N, D + 5), float("nan"), dtype=dtype, device="cuda")
        return buf[..., :D].copy_(x)
    if kind == "one head for all":
        return x[:, :1].expand(B, H, N, D)
    if kind == "overlapping rows":
        return x[:, :, :1].expand(B, H, N, D)
    return x


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,D", [(torch.bfloat16, 64), (torch.float16, 128), (torch.bfloat16, 40), (torch.float16, 36),
                                     (torch.float32, 64), (torch.float32, 100)])
@pytest.mark.parametrize("kind", ["dense", "heads last", "columns apart", "wide rows", "one head for all",
                                  "overlapping rows"])
def test_any_view_gives_what_its_values_give(kind, dtype, D):
    shape = (2, 3, 137, D)
    q, k, v, do = (_view(kind, shape, dtype, i) for i in range(4))
    for softmax in (True, False):
        want = ops._forward(*(t.contiguous() for t in (q, k, v)), True, softmax)
        out, lse = ops._forward(q, k, v, True, softmax)
        assert torch.equal(out, want[0]) and (lse is None or torch.equal(lse, want[1]))
        args = (True, D ** -0.5, softmax)
        dense = ops._backward(*(t.contiguous() for t in (q, k, v)), out, lse, do.contiguous(), *args)
        grads = ops._backward(q, k, v, out, lse, do, *args)
        ops.check_device_status()
        for a, b in zip(grads, dense):
            assert a.shape == shape and a.dtype == dtype and not a.isnan().any()
            assert (a.double() - b.double()).norm() <= 1e-3 * b.double().norm()     # the order of dQ's fp32 additions


@pytest.mark.gpu
def test_a_refused_call_takes_no_status_slot():
    q = torch.zeros(1, 2, 64, 64, device="cuda", dtype=torch.bfloat16)
    mon = ops._monitor(q.device)
    ops.check_device_status()
    for _ in range(2 * mon.SLOTS):
        with pytest.raises(ValueError):
            ops._forward(q, q[:, :1], q, True, True)
    assert len(mon.free) == mon.SLOTS
