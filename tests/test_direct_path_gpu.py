"""The short way of eager calls (ops._direct) against the registered operators: same results, and whatever has to see an
operator still sees it."""

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from rbf_attention_b200 import lm, ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


class _Seen(TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.names = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.names.append(str(func))
        return func(*args, **(kwargs or {}))


def _randn(*shape, dtype=torch.bfloat16, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(shape, generator=g, device=DEV) * 0.5).to(dtype)


def _attention(fn):
    q, k, v = (_randn(2, 3, 200, 64, seed=i).requires_grad_(True) for i in range(3))
    return lambda: (fn(q, k, v, True), (q, k, v))


def _block():
    qkv, pw = _randn(2, 150, 3 * 2 * 64).requires_grad_(True), _randn(2, 32, seed=1).requires_grad_(True)
    reg, table = _randn(2, 4, 64, seed=2).requires_grad_(True), _randn(146, 64, seed=3).float()
    return lambda: (ops.susie_block_attention(qkv, pw, reg, table, 2), (qkv, pw, reg))


def _norms():
    x, r = (_randn(64, 512, seed=i).requires_grad_(True) for i in range(2))
    w, b = (_randn(512, seed=i).requires_grad_(True) for i in (2, 3))

    def run():
        s, y = ops.add_layer_norm(ops.layer_norm(x, w, b), r, w, b)
        return s * 2 + y, (x, r, w, b)
    return run


def _mlp():
    up, down = torch.nn.Linear(64, 128), torch.nn.Linear(128, 64)
    up, down = up.to(DEV, torch.bfloat16), down.to(DEV, torch.bfloat16)
    x = _randn(40, 64).requires_grad_(True)
    return lambda: (ops.linear(down, ops.linear_gelu(up, x)), (x, up.weight, up.bias, down.weight, down.bias))


def _loss():
    logits = _randn(40, 512).requires_grad_(True)
    targets = torch.arange(40, device=DEV)
    return lambda: (lm.cross_entropy(logits, targets) * 3.0, (logits,))


CASES = {"softmax": (lambda: _attention(ops.run_triton_rbf), "rbf_attn_v5.scaled_fwd"),
         "non_softmax": (lambda: _attention(ops.run_triton_non_softmax_rbf), "rbf_attn_v5.non_softmax_fwd"),
         "block": (_block, "rbf_attn_b200.susie_block_fwd"), "norms": (_norms, "rbf_attn_b200.add_layer_norm_fwd"),
         "mlp": (_mlp, "rbf_attn_b200.gelu_fwd"), "loss": (_loss, "rbf_attn_b200.cross_entropy_fwd")}


def _grads(run):
    out, inputs = run()
    return [out.detach()] + list(torch.autograd.grad(out, inputs, torch.ones_like(out)))


@pytest.mark.parametrize("name", sorted(CASES))
def test_direct_calls_equal_the_operators(name, monkeypatch):
    make, op = CASES[name]
    torch.manual_seed(0)
    run = make()
    direct = _grads(run)
    with torch.no_grad():
        assert torch.equal(run()[0], direct[0])
    seen = _Seen()
    with seen:
        through_mode = _grads(run)
    assert any(op in n for n in seen.names), "a dispatch mode sees the operator"
    monkeypatch.setattr(ops, "_direct", lambda *t: False)
    registered = _grads(run)
    for got in (through_mode, registered):
        for a, b in zip(direct, got):
            # equal but for the fp32 additions of dQ, whose order varies from run to run (and its bf16 rounding)
            assert a.dtype == b.dtype and a.shape == b.shape
            assert (a.float() - b.float()).norm() <= 1e-3 * b.float().norm() + 1e-12


@pytest.mark.parametrize("name", sorted(CASES))
def test_direct_calls_keep_autograds_rules(name):
    """Saved tensors go through the hooks."""
    torch.manual_seed(0)
    run = CASES[name][0]()
    want = _grads(run)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.shape) or t.clone(), lambda t: t):
        out, inputs = run()
    got = torch.autograd.grad(out, inputs, torch.ones_like(out))
    assert packed
    for a, b in zip(got, want[1:]):
        assert (a.float() - b.float()).norm() <= 1e-3 * b.float().norm() + 1e-12


@pytest.mark.parametrize("loss", ["linear", "quadratic"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_second_order_gradients_are_refused(name, loss):
    """A gradient taken with ``create_graph`` equals the plain one and refuses to be differentiated, as the registered
    backward operators do (test_second_order_cpu.py has the cases of the graph alone)."""
    torch.manual_seed(0)
    run = CASES[name][0]()
    reduce = (lambda t: t.float().sum()) if loss == "linear" else (lambda t: t.float().square().sum())
    out, inputs = run()
    (want,) = torch.autograd.grad(reduce(out), inputs[:1])
    out, inputs = run()
    (got,) = torch.autograd.grad(reduce(out), inputs[:1], create_graph=True)
    assert not want.requires_grad and got.requires_grad
    assert (got.float() - want.float()).norm() <= 1e-3 * want.float().norm() + 1e-12
    with pytest.raises(RuntimeError, match="Trying to backward through"):
        got.float().square().sum().backward()


def test_what_is_not_a_plain_cuda_tensor_takes_the_operator():
    x = torch.zeros(2)
    assert not ops._direct(x)
    y = torch.zeros(2, device=DEV)
    assert ops._direct(y, None, torch.nn.Parameter(y))
    with torch.device("cuda"):
        assert not ops._direct(y)
    assert not ops._direct(y.as_subclass(type("Sub", (torch.Tensor,), {})))
    assert torch.func.vmap(lambda t: torch.tensor(ops._direct(y)) + t.sum() * 0)(y).tolist() == [0.0, 0.0]
    with pytest.raises(Exception):
        ops.run_triton_rbf(x, x, x, True)
