"""Every path whose kernels overlap their launches: captured into a CUDA graph and replayed on other values, and enqueued from
two streams at once, against the same calls by themselves."""

import pytest
import torch

from rbf_attention_b200 import lm, ops
from rbf_attention_b200.attention import CustomCausalAttention

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _randn(*shape, dtype=torch.bfloat16, std=0.5):
    return (torch.randn(shape, device=DEV) * std).to(dtype)


def _operator(dtype, D, softmax, causal):
    fn = ops.run_triton_rbf if softmax else ops.run_triton_non_softmax_rbf
    return [_randn(2, 5, 333, D, dtype=dtype) for _ in range(3)], lambda q, k, v: fn(q, k, v, causal)


def _block():
    with torch.device(DEV):
        block = CustomCausalAttention(4, 256, max_seq_len=300, attention_type="rbf_triton", num_registers=3)
    block = block.to(DEV, torch.float16).requires_grad_(False)
    return [_randn(2, 300, 256, dtype=torch.float16), *(p.detach() for p in block.parameters())], \
        lambda x, *params: torch.func.functional_call(block, dict(zip(dict(block.named_parameters()), params)), (x,))[0]


def _norms():
    def run(x, r, w, b):
        s, y = ops.add_layer_norm(ops.layer_norm(x, w, b), r, w, b)
        return s * 2 + y
    return [_randn(700, 512), _randn(700, 512), _randn(512), _randn(512)], run


def _mlp():
    class Layer:
        out_features = 512

        def __init__(self, weight, bias):
            self.weight, self.bias = weight, bias
    return [_randn(700, 256), _randn(512, 256, std=0.06), _randn(512), _randn(512, 512, std=0.04), _randn(512)], \
        lambda x, w1, b1, w2, b2: ops.linear(Layer(w2, b2), ops.linear_gelu(Layer(w1, b1), x))


CASES = {
    "softmax D64": lambda: _operator(torch.bfloat16, 64, True, True),
    "softmax D128 full": lambda: _operator(torch.float16, 128, True, False),
    "non-softmax D64": lambda: _operator(torch.float16, 64, False, True),
    "non-softmax D80": lambda: _operator(torch.bfloat16, 80, False, True),
    "fp32 D64": lambda: _operator(torch.float32, 64, True, True),
    "fp32 D128": lambda: _operator(torch.float32, 128, True, True),
    "block": _block, "norms": _norms, "mlp": _mlp,
    "loss": lambda: ([_randn(300, 1000, std=2.0)], lambda x: lm.cross_entropy(x, torch.arange(300, device=DEV))),
}


class _Pass:
    """Forward and backward with inputs that can be written to."""

    def __init__(self, name, seed):
        torch.manual_seed(seed)
        inputs, self.fn = CASES[name]()
        self.inputs = [t.clone().requires_grad_(True) for t in inputs]
        self.dout = torch.randn_like(self.fn(*self.inputs))

    def refill(self, seed):
        torch.manual_seed(seed)
        with torch.no_grad():
            for t in (*self.inputs, self.dout):
                t.copy_(torch.randn_like(t) * t.std().clamp(min=0.02) if t.numel() > 1 else torch.randn_like(t))

    def run(self):
        out = self.fn(*self.inputs)
        return [out.detach(), *torch.autograd.grad(out, self.inputs, self.dout)]


def _close(got, want):
    for a, b in zip(got, want):
        # equal but for the fp32 additions of dQ, whose order varies from run to run, and their 16-bit roundings on the way on
        assert a.dtype == b.dtype and not a.isnan().any()
        assert (a.double() - b.double()).norm() <= 2e-3 * b.double().norm() + 1e-12


@pytest.mark.parametrize("name", sorted(CASES))
def test_a_captured_pass_replays_on_other_values(name):
    case = _Pass(name, 1)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            case.run()
    torch.cuda.current_stream().wait_stream(side)
    ops.check_device_status()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = case.run()
    for seed in (2, 3, 4):
        case.refill(seed)
        want = [t.clone() for t in case.run()]
        for t in got:
            t.fill_(7)
        for _ in range(3):                  # the graph's workspaces are used again without anything in between
            graph.replay()
        torch.cuda.synchronize()
        _close(got, want)
    ops.check_device_status()
    del graph


@pytest.mark.parametrize("name", sorted(CASES))
def test_two_streams_at_once(name):
    cases = [_Pass(name, seed) for seed in (1, 2)]
    want = [[t.clone() for t in case.run()] for case in cases]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in cases]
    got = [[], []]
    for _ in range(8):
        for case, stream, results in zip(cases, streams, got):
            with torch.cuda.stream(stream):
                results.append(case.run())
    torch.cuda.synchronize()
    ops.check_device_status()
    for results, reference in zip(got, want):
        for result in results:
            _close(result, reference)
