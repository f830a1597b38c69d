"""The forward at the edges of its tiles: items of one and more key tiles, with one or two query tiles, an odd number of
them, and rows whose maximum rises from key tile to key tile (the accumulated output is rescaled under the products in
flight). Against the fp32 oracle with the tolerances of the 16-bit operands (2^-9 and 2^-11 relative rounding of P and of the
result over sums of independent terms)."""

import pytest
import torch

from oracle import rbf_oracle as oracle
from rbf_attention_b200 import ops

pytestmark = pytest.mark.gpu
REL_L2 = {torch.bfloat16: 6e-3, torch.float16: 1e-3}


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("N", [127, 128, 129, 256, 257, 385, 640])
def test_forward_at_tile_edges(N, D, dtype):
    for softmax in (True, False):
        q, k, v, do = oracle.make_inputs(2, 3, N, D, seed=N, dtype=dtype, std=1.0 if softmax else 0.5)
        if softmax:                     # nearer keys come later: 2^8 is passed several times over the first keys
            k = (k.float() * torch.linspace(2.5, 0.8, N)[None, None, :, None]).to(dtype)
        for causal in (True, False):
            ref = oracle.torch_forward_backward(q, k, v, do, causal, softmax, dtype=torch.float32)[0]
            out, lse = ops._forward(q.to("cuda"), k.to("cuda"), v.to("cuda"), causal, softmax)
            again, _ = ops._forward(q.to("cuda"), k.to("cuda"), v.to("cuda"), causal, softmax)
            ops.check_device_status()
            rep = oracle.error_report(out.cpu().float(), ref)
            assert rep["rel_l2"] <= REL_L2[dtype], (softmax, causal, rep)
            assert torch.equal(out, again)
            if softmax:
                qf, kf = q.double(), k.double()
                scores = (2 * qf @ kf.mT - kf.square().sum(-1)[:, :, None]) / D ** 0.5
                if causal:
                    scores = scores.masked_fill(torch.ones(N, N, dtype=torch.bool).triu(1), float("-inf"))
                want = torch.logsumexp(scores, -1) / torch.tensor(2.0).double().log()
                assert (lse.cpu().double() - want).abs().max() <= 1e-3


@pytest.mark.parametrize("N", [64, 65, 127, 129, 300])
def test_fp32_forward_posts_its_status_word(N):
    """The word comes from the last block of the kernel itself, also on a workspace of an earlier call."""
    for seed in range(3):
        q, k, v, do = oracle.make_inputs(2, 3, N, 64, seed=seed, dtype=torch.float32)
        ref = oracle.torch_forward_backward(q, k, v, do, True, True, dtype=torch.float32)[0]
        out, _ = ops._forward(q.to("cuda"), k.to("cuda"), v.to("cuda"), True, True)
        ops.check_device_status()
        assert oracle.error_report(out.cpu(), ref)["rel_l2"] <= 6e-3


@pytest.mark.parametrize("rows", [1, 63, 64, 65, 64 * 8 + 1, 64 * 13 + 5, 70000])
def test_column_sums_over_few_and_many_bands(rows):
    """One fp32 sum per column over the bands' partial sums: the second kernel starts while the first one runs."""
    g = torch.Generator().manual_seed(rows)
    x = torch.randn(rows, 264, generator=g).to(torch.bfloat16)
    got = ops._column_sums(x.to("cuda")).cpu().double()
    want = x.double().sum(0)
    # sums of `rows` terms in any order: the error of an fp32 sum is at most its depth (well below 2^10) times 2^-24 of sum |x|
    assert ((got - want).abs() <= 2.0 ** -14 * x.double().abs().sum(0)).all()


@pytest.mark.parametrize("D,causal,dtype", [(128, False, torch.float16), (128, True, torch.bfloat16), (64, False, torch.float16)])
def test_forward_repeats_bitwise_under_load(D, causal, dtype):
    """Warps of a query tile drift apart by up to a key tile; what one of them has arrived for must not be counted for another,
    and a wait for a product must not be content with an earlier one. 2, 16 heads x 3333 rows: three rounds of CTAs."""
    q, k, v, _ = oracle.make_inputs(2, 16, 3333, D, seed=3, dtype=dtype)
    k = (k.float() * torch.linspace(1.5, 0.9, 3333)[None, None, :, None]).to(dtype)
    q, k, v = (t.to("cuda") for t in (q, k, v))
    first, lse = ops._forward(q, k, v, causal, True)
    for _ in range(40):
        out, again = ops._forward(q, k, v, causal, True)
        assert torch.equal(out, first) and torch.equal(again, lse)
    ops.check_device_status()
    ref = oracle.torch_forward_backward(q[1:, 15:].cpu(), k[1:, 15:].cpu(), v[1:, 15:].cpu(), v[1:, 15:].cpu(), causal, True,
                                        dtype=torch.float32)[0]
    assert oracle.error_report(first[1:, 15:].cpu().float(), ref)["rel_l2"] <= REL_L2[dtype]
