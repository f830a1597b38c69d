"""What a user of this package has it do, as measurable cases: the attention operators, the attention block and the
language model around it, through their public entry points, forward alone and forward + backward.

``listed()`` are fixed cases, ``draw(rng)`` gives another one of the same ranges. ``prepare(case, seed)`` builds what a
program holds before the call, ``run(state)`` is one pass, ``work(case)`` its unavoidable bytes and operations,
``tolerance(case)`` how far another correct implementation of the same precision may be off."""

from __future__ import annotations

import math

import torch

from rbf_attention_b200 import lm
from rbf_attention_b200.attention import CustomCausalAttention
from rbf_attention_b200.ops import run_triton_non_softmax_rbf, run_triton_rbf

DEVICE = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}
VOCAB = 50257          # the language model of the training benchmark: 8 layers of width 512, 8 heads of 64, 4 registers
D_MODEL, HEADS, LAYERS, REGISTERS, MAX_SEQ = 512, 8, 8, 4, 1024


def _op(name, B, H, N, D, dtype, causal=True, softmax=True, train=True, key_sigma=0.0):
    return {"name": name, "kind": "op", "B": B, "H": H, "N": N, "D": D, "dtype": dtype, "causal": causal,
            "softmax": softmax, "train": train, "key_sigma": key_sigma}


def listed():
    return [
        # scoring a few short prompts: the smallest call, one forward whose launches outweigh its arithmetic
        _op("op_forward_256", 2, 4, 256, 64, "bf16", train=False),
        # one attention layer of a small training step (the shortest size of the operator's usual benchmark sweep)
        _op("op_train_1k_fp16", 4, 8, 1024, 64, "fp16"),
        # an encoder's unmasked attention over sequences that fill no whole number of tiles
        _op("op_train_1000_full", 4, 12, 1000, 64, "bf16", causal=False),
        # float32 training as debugging and parity runs do it
        _op("op_train_1k_fp32", 2, 8, 1024, 64, "fp32"),
        # a head dim between the two that the kernels are built for
        _op("op_train_1500_d80", 2, 12, 1500, 80, "fp16"),
        # the headline benchmark: a training step's attention over 4096 tokens, a few keys of outlying norm
        _op("op_train_4k", 8, 16, 4096, 64, "bf16", key_sigma=0.5),
        # the variant without a softmax denominator at its benchmark size
        _op("op_train_8k_no_softmax", 4, 16, 8192, 64, "bf16", softmax=False),
        # evaluation with wide heads, unmasked, an odd length
        _op("op_forward_3333_d128_full", 2, 16, 3333, 128, "fp16", causal=False, train=False),
        # long-context training with wide heads: the largest attention call
        _op("op_train_16k_d128", 2, 32, 16384, 128, "bf16"),
        # the attention block (projections, positions, registers) in a training step: the layer benchmark
        {"name": "block_train_4k_fp16", "kind": "block", "B": 4, "N": 4100, "heads": 8, "head_dim": 64, "dtype": "fp16",
         "registers": 4, "softmax": True, "train": True},
        # the language model reading a batch of prompts: logits for every position
        {"name": "lm_prefill_777", "kind": "lm", "B": 4, "T": 777, "train": False},
        # the training step of the language-model benchmark: forward, loss, backward (the largest case of all)
        {"name": "lm_train_64x1024", "kind": "lm", "B": 64, "T": 1024, "train": True},
    ]


def _log_int(rng, low, high):
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def _op_flops(B, H, N, D, causal, train):
    """2 products forward, 5 backward, half of them under the causal mask."""
    return (14.0 if train else 4.0) * B * H * float(N) * N * D * (0.5 if causal else 1.0)


def draw(rng):
    kind = rng.choice(["op"] * 8 + ["block"] * 2 + ["lm"] * 2)
    train = rng.random() < 0.7
    if kind == "lm":
        return {"kind": "lm", "B": _log_int(rng, 1, 48), "T": _log_int(rng, 64, MAX_SEQ), "train": train}
    if kind == "block":
        return {"kind": "block", "B": rng.randint(1, 6), "N": _log_int(rng, 100, 6000), "heads": rng.choice([4, 8, 16]),
                "head_dim": rng.choice([64, 64, 128]), "dtype": rng.choice(["bf16", "fp16"]),
                "registers": rng.choice([0, 4]), "softmax": rng.random() < 0.75, "train": train}
    case = _op("", 1, 1, 1, rng.choice([64] * 6 + [128] * 3 + [32, 48, 80]),
               rng.choice(["bf16"] * 5 + ["fp16"] * 3 + ["fp32"]), causal=rng.random() < 0.7,
               softmax=rng.random() < 0.75, train=train)
    del case["name"]
    if case["dtype"] == "fp32":
        case["D"] = 64
    case["key_sigma"] = rng.choice([0.0, 0.5])
    case["N"] = _log_int(rng, 100, 16384 if case["dtype"] != "fp32" else 4096)
    # batch x heads within what the largest listed calls cost
    most = _op_flops(2, 32, 16384, 128, True, True) / (16 if case["dtype"] == "fp32" else 3)
    pairs = most / _op_flops(1, 1, case["N"], case["D"], case["causal"], train)
    case["H"] = rng.choice([h for h in (1, 4, 8, 12, 16, 32) if h <= max(1, pairs)])
    case["B"] = _log_int(rng, 1, max(1, min(16, int(pairs / case["H"]))))
    return case


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _prepare_op(case, seed):
    g, dtype = _generator(seed), DTYPES[case["dtype"]]
    shape = (case["B"], case["H"], case["N"], case["D"])

    def normal(std=1.0):
        return torch.randn(shape, generator=g, device=DEVICE) * std

    # without a denominator the distances have to stay where the exponential does not vanish
    std = 1.0 if case["softmax"] else 0.5
    q, k, v, dout = normal(std), normal(std), normal(std), normal()
    if case["key_sigma"] > 0 and case["softmax"]:
        k = k * torch.exp(torch.randn(shape[:3] + (1,), generator=g, device=DEVICE) * case["key_sigma"])
    q, k, v, dout = (t.to(dtype) for t in (q, k, v, dout))
    if case["train"]:
        for t in (q, k, v):
            t.requires_grad_(True)
    return {"case": case, "q": q, "k": k, "v": v, "dout": dout}


def _run_op(s):
    case = s["case"]
    attention = run_triton_rbf if case["softmax"] else run_triton_non_softmax_rbf
    out = attention(s["q"], s["k"], s["v"], case["causal"])
    if not case["train"]:
        return out
    return (out.detach(),) + torch.autograd.grad(out, (s["q"], s["k"], s["v"]), s["dout"])


def _prepare_block(case, seed):
    g, dtype = _generator(seed), DTYPES[case["dtype"]]
    width = case["heads"] * case["head_dim"]
    torch.manual_seed(seed)
    with torch.device(DEVICE):
        block = CustomCausalAttention(case["heads"], width, max_seq_len=case["N"],
                                      attention_type="rbf_triton" if case["softmax"] else "rbf_non_softmax",
                                      num_registers=case["registers"])
    block = block.to(DEVICE, dtype)
    x = torch.randn((case["B"], case["N"], width), generator=g, device=DEVICE).to(dtype)
    dy = torch.randn((case["B"], case["N"], width), generator=g, device=DEVICE).to(dtype)
    return {"case": case, "block": block, "params": list(block.parameters()), "x": x.requires_grad_(case["train"]), "dy": dy}


def _run_block(s):
    if not s["case"]["train"]:
        with torch.no_grad():
            return s["block"](s["x"])[0]
    y, _ = s["block"](s["x"])
    return (y.detach(),) + torch.autograd.grad(y, [s["x"]] + s["params"], s["dy"])


def _prepare_lm(case, seed):
    torch.manual_seed(seed)
    with torch.device(DEVICE):
        model = lm.CausalLM(VOCAB, d_model=D_MODEL, num_layers=LAYERS, num_heads=HEADS, max_seq_len=MAX_SEQ,
                            pos_emb_type="rope", num_registers=REGISTERS, attention_type="rbf_triton")
    model = model.to(DEVICE, torch.bfloat16)
    ids = lm.zipf_token_ids(case["B"], case["T"] + 1, VOCAB, seed=seed).to(DEVICE)
    # gradients leave in buckets, one per block and one for the rest, as data-parallel training sends them
    buckets = [list(block.parameters()) for block in model.blocks]
    in_blocks = {id(p) for bucket in buckets for p in bucket}
    buckets.append([p for p in model.parameters() if id(p) not in in_blocks])
    return {"case": case, "model": model, "buckets": buckets, "tokens": ids[:, :-1].contiguous(),
            "targets": ids[:, 1:].contiguous()}


def _run_lm(s):
    if not s["case"]["train"]:
        with torch.no_grad():
            return s["model"](s["tokens"])[0]
    logits, _ = s["model"](s["tokens"], padded_logits=True)
    loss = lm.cross_entropy(logits, s["targets"])
    del logits
    loss.backward()
    out = [loss.detach()]
    for bucket in s["buckets"]:
        out.append(torch.cat([p.grad.reshape(-1) for p in bucket]))
        for p in bucket:
            p.grad = None
    return out


def prepare(case, seed):
    return {"op": _prepare_op, "block": _prepare_block, "lm": _prepare_lm}[case["kind"]](case, seed)


def run(state):
    return {"op": _run_op, "block": _run_block, "lm": _run_lm}[state["case"]["kind"]](state)


def work(case):
    if case["kind"] == "op":
        tensor = case["B"] * case["H"] * case["N"] * case["D"] * BYTES[case["dtype"]]
        # forward: q, k, v in, o out; backward: dO in, dq, dk, dv out
        return {"bytes": float((8 if case["train"] else 4) * tensor),
                "flops": _op_flops(case["B"], case["H"], case["N"], case["D"], case["causal"], case["train"])}
    if case["kind"] == "block":
        width = case["heads"] * case["head_dim"]
        rows = case["B"] * case["N"]
        weights = 4 * width * width
        flops = 2.0 * rows * weights * (3 if case["train"] else 1)
        flops += _op_flops(case["B"], case["heads"], case["N"], case["head_dim"], True, case["train"])
        moved = 2 * rows * width + weights           # x and the weights in, y out
        if case["train"]:
            moved += 2 * rows * width + weights      # dy in, dx and the weights' gradients out
        return {"bytes": 2.0 * moved, "flops": flops}
    rows = case["B"] * (case["T"] + REGISTERS)
    text_rows = case["B"] * case["T"]
    block_weights = 12 * D_MODEL * D_MODEL * LAYERS
    head_weights = D_MODEL * VOCAB
    flops = 2.0 * (rows * block_weights + text_rows * head_weights) * (3 if case["train"] else 1)
    flops += LAYERS * _op_flops(case["B"], HEADS, case["T"] + REGISTERS, D_MODEL // HEADS, True, case["train"])
    weights = block_weights + 2 * head_weights       # projections, embedding and vocabulary projection
    # a training step needs its weights and leaves as many gradients, a prompt its logits; ids are 8 bytes
    moved = 2 * weights if case["train"] else weights - head_weights + text_rows * VOCAB
    return {"bytes": 2.0 * moved + 8.0 * text_rows * (2 if case["train"] else 1), "flops": flops}


def tolerance(case):
    # four times what a pass is off the same mathematics in 64 bits (operators) or in fp32 (block): bf16 operands with
    # fp32 sums 2.7e-3, fp16 3.5e-4; float32 tensors run on 11-bit operands whose kind differs between forward (TF32)
    # and backward (fp16), 2.8e-3. In the block a bias gradient is a small difference of large sums: fp16 2e-3, bf16
    # 3.6e-2, whose fourfold is cut to the 3e-2 that eight bf16 layers of the language model also get.
    if case["kind"] == "op":
        return {"rel": {"bf16": 1.1e-2, "fp16": 1.4e-3, "fp32": 1.1e-2}[case["dtype"]]}
    if case["kind"] == "block":
        return {"rel": 3e-2 if case["dtype"] == "bf16" else 8e-3}
    return {"rel": 3e-2}
