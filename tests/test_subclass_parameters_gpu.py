"""Parameters that are wrappers without storage of their own (sharded, quantised): whatever is computed from one goes through
the registered operators, which the wrapper sees, and not to a kernel by its address."""

import pytest
import torch

from rbf_attention_b200 import ops

pytestmark = pytest.mark.gpu


class Wrapped(torch.Tensor):
    seen = []

    @staticmethod
    def __new__(cls, inner):
        return torch.Tensor._make_wrapper_subclass(cls, inner.shape, strides=inner.stride(), dtype=inner.dtype,
                                                   device=inner.device, requires_grad=inner.requires_grad)

    def __init__(self, inner):
        self.inner = inner

    @classmethod
    def __torch_dispatch__(cls, func, types, args=(), kwargs=None):
        cls.seen.append(str(func))
        unwrap = lambda t: t.inner if isinstance(t, cls) else t
        out = func(*(unwrap(a) for a in args), **{k: unwrap(v) for k, v in (kwargs or {}).items()})
        return cls(out) if isinstance(out, torch.Tensor) and func is not torch.ops.aten.detach.default else out


@pytest.mark.parametrize("which", ["weight", "bias"])
def test_linear_gelu_with_a_wrapped_parameter(which):
    torch.manual_seed(0)
    x = torch.randn(40, 64, device="cuda", dtype=torch.bfloat16)
    plain = torch.nn.Linear(64, 128, device="cuda", dtype=torch.bfloat16).requires_grad_(False)
    want = ops.linear_gelu(plain, x)

    class Holder:                       # what linear_gelu reads of a module
        weight, bias, out_features = plain.weight.data, plain.bias.data, 128

    holder = Holder()
    setattr(holder, which, Wrapped(getattr(holder, which)))
    Wrapped.seen.clear()
    with torch.no_grad():
        got = ops.linear_gelu(holder, x)
    assert any("gelu_fwd" in name for name in Wrapped.seen)
    assert isinstance(got, Wrapped) and torch.equal(got.inner, want)
