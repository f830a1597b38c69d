"""Second-order gradients are not implemented and have to be refused, by the registered operators and by the calls that go
around them (``ops._direct``), also where the loss is linear in the output: a gradient returned as a constant would make a
penalty on it add nothing. CPU only: closed forms stand in for the kernels, what is tested is the graph around them."""

import pytest
import torch

from rbf_attention_b200 import ops


def _attention_fwd(q, k, v, causal):
    p = torch.softmax(q @ k.transpose(-1, -2), -1)
    return p @ v, p.sum(-1)


def _attention_bwd(q, k, v, out, lse, dout, causal, scale):
    return q * dout, k * dout, v * dout


def _norm_fwd(x, weight, bias, eps):
    mean, rstd = x.mean(-1), (x.var(-1, unbiased=False) + eps).rsqrt()
    return (x - mean[:, None]) * rstd[:, None] * weight + bias, mean, rstd


def _norm_bwd(x, dy, weight, mean, rstd):
    return x * dy * weight, (x * dy).sum(0), dy.sum(0)


def _block_fwd(qkv, pos_weight, reg_pos_emb, table, heads, softmax):
    q, k, v = (t.contiguous() for t in qkv.chunk(3, -1))
    return (q + pos_weight.sum()) * k * v, q.sum(-1), torch.stack((q, k))


def _block_bwd(qkv, qk, out, lse, dout, table, registers, softmax):
    return qkv * dout.repeat(1, 1, 3), dout.sum() * torch.ones(2, 2), dout.sum() * torch.ones(2, 1, 4)


def _gelu_bwd(h, dy, with_bias):
    return h * dy, (h * dy).sum(0) if with_bias else h.new_empty(0)


def _scale(x, factor):
    x.detach().mul_(factor)


def _loss_fwd(logits, targets, ignore_index):
    p = torch.softmax(logits, -1)
    grad = (p - torch.nn.functional.one_hot(targets, logits.shape[1])) / len(targets)
    return -p.gather(1, targets[:, None]).log().mean(), grad


# operator -> (implementation that a direct call runs, closed form)
STANDINS = {
    "rbf_attn_v5::scaled_fwd": (None, _attention_fwd),
    "rbf_attn_v5::scaled_bwd": (None, _attention_bwd),
    "rbf_attn_v5::non_softmax_fwd": (None, lambda *a: _attention_fwd(*a)[0]),
    "rbf_attn_v5::non_softmax_bwd_with_out": (None, lambda q, k, v, o, do, c, s: _attention_bwd(q, k, v, o, None, do, c, s)),
    "rbf_attn_b200::susie_block_fwd": ("_susie_block_fwd", _block_fwd),
    "rbf_attn_b200::susie_block_bwd": ("_susie_block_bwd", _block_bwd),
    "rbf_attn_b200::layer_norm_fwd": ("_layer_norm_fwd", _norm_fwd),
    "rbf_attn_b200::layer_norm_bwd": ("_layer_norm_bwd", _norm_bwd),
    "rbf_attn_b200::add_layer_norm_fwd": ("_add_layer_norm_fwd", lambda x, r, w, b, e: (x + r, *_norm_fwd(x + r, w, b, e))),
    "rbf_attn_b200::layer_norm_bwd_add": ("_layer_norm_bwd_add",
                                          lambda x, dy, dr, w, m, r: (_norm_bwd(x, dy, w, m, r)[0] + dr, (x * dy).sum(0), dy.sum(0))),
    "rbf_attn_b200::gelu_fwd": ("_gelu_fwd", torch.nn.functional.gelu),
    "rbf_attn_b200::gelu_bwd": ("_gelu_bwd", _gelu_bwd),
    "rbf_attn_b200::column_sums": ("_column_sums", lambda x: x.sum(0)),
    "rbf_attn_b200::cross_entropy_fwd": ("_cross_entropy_fwd", _loss_fwd),
    "rbf_attn_b200::scale_unless_one_": ("_scale_unless_one", _scale),
}


@pytest.fixture(params=["direct", "operators"])
def standins(request, monkeypatch):
    libraries = {ns: torch.library.Library(ns, "IMPL") for ns in ("rbf_attn_v5", "rbf_attn_b200")}
    for op, (name, fn) in STANDINS.items():
        namespace, _, op_name = op.partition("::")
        libraries[namespace].impl(op_name, fn, "CPU")
        if name is not None:
            monkeypatch.setattr(ops, name, fn)
    monkeypatch.setattr(ops, "_forward", lambda q, k, v, causal, softmax: _attention_fwd(q, k, v, causal))
    monkeypatch.setattr(ops, "_backward", lambda q, k, v, o, lse, do, c, s, softmax: _attention_bwd(q, k, v, o, lse, do, c, s))
    monkeypatch.setattr(ops, "_direct", lambda *tensors: request.param == "direct")
    yield request.param
    for library in libraries.values():
        library._destroy()


def _leaf(*shape):
    return torch.randn(shape, requires_grad=True)


def _attention(fn):
    q, k, v = (_leaf(1, 2, 5, 4) for _ in range(3))
    return fn(q, k, v, True), (q, k, v)


def _block():
    qkv, pw, reg = _leaf(1, 5, 12), _leaf(2, 2), _leaf(2, 1, 4)
    return ops.susie_block_attention(qkv, pw, reg, torch.zeros(4, 4), 2), (qkv, pw, reg)


def _norm():
    x, w, b = _leaf(5, 8), _leaf(8), _leaf(8)
    return ops.layer_norm(x, w, b), (x, w)


def _add_norm():
    x, r, w, b = _leaf(5, 8), _leaf(5, 8), _leaf(8), _leaf(8)
    s, y = ops.add_layer_norm(x, r, w, b)
    return s * 2 + y, (x, r, w)


def _gelu():
    x, w, b = _leaf(5, 8), _leaf(16, 8), _leaf(16)
    return ops._LinearGelu.apply(x, w, b), (x, w, b)


def _loss():
    logits, factor = _leaf(5, 8), _leaf()
    return ops.cross_entropy(logits, torch.arange(5)) * factor, (logits,)


CASES = {"softmax": lambda: _attention(ops.run_triton_rbf), "non_softmax": lambda: _attention(ops.run_triton_non_softmax_rbf),
         "block": _block, "norm": _norm, "add_norm": _add_norm, "gelu": _gelu, "loss": _loss}
LOSSES = {"linear": lambda out: out.sum(), "quadratic": lambda out: out.square().sum()}


@pytest.mark.parametrize("loss", sorted(LOSSES))
@pytest.mark.parametrize("name", sorted(CASES))
def test_second_order_gradients_are_refused(name, loss, standins):
    torch.manual_seed(0)
    out, inputs = CASES[name]()
    want = torch.autograd.grad(LOSSES[loss](out), inputs)
    assert not any(g.requires_grad for g in want)
    for i in range(len(inputs)):
        torch.manual_seed(0)
        out, inputs = CASES[name]()
        got = torch.autograd.grad(LOSSES[loss](out), inputs, create_graph=True)     # the gradient itself stays available
        assert torch.equal(got[i], want[i])
        with pytest.raises(RuntimeError, match="Trying to backward through"):
            got[i].square().sum().backward()


def test_a_factor_on_the_loss_does_not_lose_its_second_derivative(standins):
    logits, factor = _leaf(5, 8), _leaf()
    (g,) = torch.autograd.grad(ops.cross_entropy(logits, torch.arange(5)) * factor, (logits,), create_graph=True)
    with pytest.raises(RuntimeError, match="Trying to backward through"):
        torch.autograd.grad(g.square().sum(), (factor,))


def test_values_that_are_not_read_again_may_change_before_the_backward(standins):
    """What PyTorch's own loss and linear layer allow: scaling the loss in place, updating a bias."""
    logits = _leaf(5, 8)
    loss = ops.cross_entropy(logits, torch.arange(5))
    loss /= 2
    loss.backward()
    assert torch.allclose(logits.grad, _loss_fwd(logits.detach(), torch.arange(5), -100)[1] / 2)
    out, (x, w, b) = _gelu()
    with torch.no_grad():
        b.add_(1.0)
    out.sum().backward()


@pytest.mark.parametrize("loss", sorted(LOSSES))
def test_linear_second_order_is_exact_or_refused(loss, standins):
    """The two products of ``linear``'s backward are PyTorch's and differentiable, its bias sum is not."""
    x, w, b = _leaf(5, 8), _leaf(16, 8), _leaf(16)

    def penalty(fn, i):
        g = torch.autograd.grad(LOSSES[loss](fn(x, w, b)), (x, w, b), create_graph=True)[i]
        return torch.autograd.grad(g.square().sum(), (x, w, b), allow_unused=True)

    for i in (0, 1):
        for got, want in zip(penalty(ops._LinearBiasSum.apply, i), penalty(torch.nn.functional.linear, i)):
            assert (got is None) == (want is None)
            assert got is None or torch.allclose(got, want, rtol=1e-4, atol=1e-4 * float(want.norm()))
    with pytest.raises(RuntimeError):       # quadratic: refused; linear: a constant, as with F.linear
        penalty(ops._LinearBiasSum.apply, 2)
