"""GELU, cross entropy and the pre-passes at the edges of their grids: a thread's second chunk missing, grids below, at and above
what is resident, rows that are brought into L2 ahead, rows that do not count among them, ragged lengths."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n", [8, 2048, 2056, 4096, 4104, 148 * 6 * 4096, 148 * 6 * 4096 + 2056])
def test_gelu_forward_chunks(n, dtype):
    """Within one rounding step of the erf form in fp64 (2^-8 / 2^-11 relative, 3e-7 absolute for the approximation of the
    normal distribution function), every element written, none beyond."""
    from rbf_attention_b200 import ops

    g = torch.Generator(device=DEV).manual_seed(n)
    h = (torch.randn(n, generator=g, device=DEV) * 2).to(dtype)
    want = F.gelu(h.double())
    rel = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert ((ops.gelu_fwd(h).double() - want).abs() <= rel * want.abs() + 3e-7).all()


@pytest.mark.parametrize("rows, cols", [(1, 256), (7, 256), (64, 2048), (65, 264), (4097, 512), (6001, 2048), (700, 40960)])
def test_gelu_backward_bands(rows, cols):
    """dh within one rounding step of fp64; the bias gradient within fp32 summation error (2^-23 times the rows a lane
    adds, at most 1e-5) of the sum of the stored dh."""
    from rbf_attention_b200 import ops

    g = torch.Generator(device=DEV).manual_seed(rows)
    h = (torch.randn((rows, cols), generator=g, device=DEV) * 2).bfloat16()
    dy = torch.randn((rows, cols), generator=g, device=DEV).bfloat16()
    x = h.double().requires_grad_(True)
    F.gelu(x).backward(dy.double())
    dh, db = ops.gelu_bwd(h, dy, True)
    assert ((dh.double() - x.grad).abs() <= 2.0 ** -8 * x.grad.abs() + 3e-7 * dy.double().abs()).all()
    assert ((db.double() - dh.double().sum(0)).abs() <= 1e-5 * dh.double().abs().sum(0) + 1e-6).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows, cols", [(1, 64), (295, 1000), (296, 1000), (297, 1000), (900, 4104), (640, 28920), (610, 57864)])
def test_cross_entropy_rows_brought_in_ahead(rows, cols, dtype):
    """Loss and gradient against fp64 with every third row ignored (the block's next row may or may not count), rows of
    odd widths for the staged, the re-read and (1000 columns of a wider tensor) the strided case. Gradients within one
    rounding step of the dtype (fp32: the exponential's 2^-21) of softmax / count, plus what a loss sum error of 1e-6 gives."""
    from rbf_attention_b200 import ops

    g = torch.Generator(device=DEV).manual_seed(rows + cols)
    x = (torch.randn((rows, cols + 24), generator=g, device=DEV) * 3).to(dtype)[:, :cols]
    t = torch.randint(0, cols, (rows,), generator=g, device=DEV)
    t[1::3] = -100
    ref_in = x.double().requires_grad_(True)
    ref = F.cross_entropy(ref_in, t, ignore_index=-100)
    ref.backward()
    a = x.detach().requires_grad_(True)
    loss = ops.cross_entropy(a, t)
    loss.backward()
    assert abs(loss.item() - ref.item()) <= 2e-6 * abs(ref.item()) + 1e-6
    rel = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -18}[dtype]
    tiny = 6e-8 if dtype == torch.float16 else 2e-6 / rows          # fp16 subnormals: spacing 2^-24
    err = (a.grad.double() - ref_in.grad).abs()
    assert (err <= rel * ref_in.grad.abs() + tiny).all()
    assert (a.grad[1::3] == 0).all()


@pytest.mark.parametrize("softmax", [True, False])
@pytest.mark.parametrize("D", [64, 72, 128])
@pytest.mark.parametrize("N", [1, 31, 33, 63, 65, 97, 129])
def test_row_statistics_at_ragged_lengths(N, D, softmax):
    """The pre-passes' rows that fill part of a batch, a warp's group or a block: outputs and gradients against the fp32 oracle
    (2^-11 relative rounding of operands, P, dS and results over sums of independent terms), on a workspace that a longer call
    has left behind."""
    from oracle import rbf_oracle as oracle
    from rbf_attention_b200 import ops

    for n in (2 * N + 200, N):
        q, k, v, do = oracle.make_inputs(2, 3, n, D, seed=n, dtype=torch.float16, std=1.0 if softmax else 0.3)
        ref = oracle.torch_forward_backward(q, k, v, do, True, softmax, dtype=torch.float32)
        qd, kd, vd, dod = (x.to(DEV) for x in (q, k, v, do))
        out, lse = ops._forward(qd, kd, vd, True, softmax)
        grads = ops._backward(qd, kd, vd, out, lse, dod, True, D ** -0.5, softmax)
        ops.check_device_status()
        for got, want in zip((out, *grads[:3]), (ref[0], *ref[-3:])):
            rep = oracle.error_report(got.cpu().float(), want)
            # a single key: dq and dk are exactly zero, their error that of dP and delta, two fp32 sums of up to 128 products
            # in different orders: 2^-24 * 128 * 4 * 4 times 2 D^-0.5 |k| <= 2 * 0.125 * 5
            assert rep["rel_l2"] <= 3e-3 or n == 1 and rep["max_abs"] <= 1.6e-4, rep


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B, H, N", [(1, 1, 700), (5, 20, 300), (2, 85, 129), (3, 67, 64), (1, 38, 900)])
def test_backward_items_in_groups_of_heads(B, H, N, D):
    """Every (key tile, head) item is worked on once, whatever the number of heads leaves for the first group (few heads, one
    group, a short first group, one key tile): gradients of each head by itself against the fp32 oracle."""
    from oracle import rbf_oracle as oracle
    from rbf_attention_b200 import ops

    q, k, v, do = oracle.make_inputs(B, H, N, D, seed=N, dtype=torch.float16, std=1.0)
    qd, kd, vd, dod = (x.to(DEV) for x in (q, k, v, do))
    for causal in (True, False):
        ref = oracle.torch_forward_backward(q, k, v, do, causal, True, dtype=torch.float32)[-3:]
        out, lse = ops._forward(qd, kd, vd, causal, True)
        grads = ops._backward(qd, kd, vd, out, lse, dod, causal, D ** -0.5, True)
        ops.check_device_status()
        for got, want in zip(grads[:3], ref):
            err = (got.cpu().float() - want).flatten(2).norm(dim=2) / want.flatten(2).norm(dim=2)
            assert err.max().item() <= 3e-3       # 2^-11 relative rounding of operands, P, dS and results
