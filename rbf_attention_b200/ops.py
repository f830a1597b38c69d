"""Operator boundary: the four ``rbf_attn_v5`` custom operators of the reference, with the same
schemas, fake kernels and autograd formulas, implemented by calls into ``librbf_b200.so``.

Reference counterparts (paths inside the reference project):
  rbf_attn_v5::scaled_fwd / scaled_bwd            rbf_attention.py:651-842
  rbf_attn_v5::non_softmax_fwd / non_softmax_bwd  rbf_attention.py:1355-1511
  run_triton_rbf / run_triton_non_softmax_rbf     rbf_attention.py:848-853
"""

from __future__ import annotations

import collections
import ctypes
import math
import os
import threading
import time

import torch
from torch.autograd import forward_ad

from . import _lib

_DTYPE_CODE = {torch.bfloat16: 0, torch.float16: 1}

_PLAIN_TYPES = (torch.Tensor, torch.nn.Parameter)


def _direct(*tensors) -> bool:
    """Whether a call may run its implementation right here instead of going through the registered operator: plain
    CUDA tensors in eager mode, with nothing active that has to see the operator (tracing or compilation, dispatch and
    function modes, functorch transforms, forward-mode differentiation). The operator layer - schema, fake kernels,
    dispatch keys, aliasing checks - costs 70 to 100 us of host time per call, more than the device time of a training
    step's attention below about 1500 tokens (B4 H8 D64: 76 us of kernels in a pass of 280 us); where the question is
    open the operator is used."""
    if torch.compiler.is_compiling() or torch._C._len_torch_dispatch_stack() or torch._C._len_torch_function_stack():
        return False
    if (torch._C._functorch.peek_interpreter_stack() is not None or torch._C._get_tracing_state() is not None
            or forward_ad._current_level >= 0):
        return False
    for t in tensors:
        if t is not None and not (type(t) in _PLAIN_TYPES and t.is_cuda):
            return False
    return True


def _direct_backward(*tensors) -> bool:
    """``_direct`` for a backward formula. Under ``create_graph`` (the only time a backward runs with grad mode on) the
    registered operator computes the gradient: it has no autograd formula, so what it returns is linked to its inputs and
    refuses to be differentiated, while a direct call's result would be a constant and a penalty on it would silently add
    nothing."""
    return not torch.is_grad_enabled() and _direct(*tensors)


class _FirstOrderOnly(torch.autograd.Function):
    """``grad`` itself, linked to the ``origins`` that it was computed from and refusing to be differentiated: for gradients
    formed under ``create_graph`` from saved tensors that carry no graph of their own."""

    @staticmethod
    def forward(ctx, what, grad, *origins):
        ctx.what = what
        return grad.view_as(grad)

    @staticmethod
    def backward(ctx, *_grads):
        raise RuntimeError(f"Trying to backward through the gradient of {ctx.what}, which has no second-order formula")


def _needs_grad(*tensors) -> bool:
    return torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in tensors)


def _validate(name: str, t: torch.Tensor, like: torch.Tensor | None = None) -> None:
    """(B, H, N, D) on a GPU and, if given, with the shape, dtype and device of ``like``."""
    _lib.host().validate(name, t, like)


def _tma_ready(t: torch.Tensor) -> torch.Tensor:
    """Returns ``t`` if the TMA engine can address it in place, else a contiguous copy. The reference assumes
    ``stride(-1) == 1`` without checking (rbf_attention.py:111-138)."""
    return _lib.host().tma_ready(t)


def _device_index(device: torch.device) -> int:
    return device.index if device.index is not None else torch._C._cuda_getDevice()


def _stream_ptr(device: torch.device) -> int:
    """Raw handle of the current stream of ``device`` (the binding's own call: building a ``torch.cuda.Stream`` object
    for it costs 10 us, a tenth of what a whole operator call takes on the host)."""
    return torch._C._cuda_getCurrentRawStream(_device_index(device))


class _OnDevice:
    """``torch.cuda.device(device)`` that does nothing when ``device`` is already the current one."""

    __slots__ = ("index", "prev")

    def __init__(self, device: torch.device):
        self.index = _device_index(device)
        self.prev = -1

    def __enter__(self):
        cur = torch._C._cuda_getDevice()
        if cur != self.index:
            self.prev = cur
            torch._C._cuda_setDevice(self.index)
        return self

    def __exit__(self, *exc):
        if self.prev >= 0:
            torch._C._cuda_setDevice(self.prev)
        return False


# States of a status entry: its slot is taken but its call has not returned yet; the call's kernels are enqueued and will
# post; the call was left by an exception and may or may not post.
_RESERVED, _ENQUEUED, _ABANDONED = range(3)


class _StatusEntry:
    __slots__ = ("slot", "what", "state")

    def __init__(self, slot, what):
        self.slot, self.what, self.state = slot, what, _RESERVED


class _StatusMonitor:
    """Surfaces device-side wait timeouts of the operator path without synchronising.

    Every kernel bounds its waits; one that runs out leaves a non-zero status word at the start of the call's
    workspace and the kernels return with incomplete results. Each call's last kernel stores the word into a ring of
    pinned host slots (a store through the mapped host address: a copy would queue on the copy engine behind the
    caller's own device-to-host transfers and hold the launch stream up for their duration); a slot holds -1 until its
    word has arrived, so no event is needed to see that it has. Later calls look at the slots that have been written and
    raise ``RuntimeError`` for a non-zero one. A timeout is therefore reported by a later operator call or by
    ``check_device_status()``, not by the call that suffered it. ``RBF_B200_SYNC_STATUS=1`` makes every call
    synchronise and check its own status (for debugging). Nothing is recorded while a CUDA graph is being captured.
    """

    SLOTS = 256
    _NOT_YET = -1          # slot value until the posting kernel has run (no status word is 0xffffffff: sites end at 250)

    def __init__(self, device):
        self.device = device
        self.index = _device_index(device)
        self.capturing = _lib.host().capturing
        self.host = torch.zeros(self.SLOTS, dtype=torch.int32).pin_memory()
        self.slots = memoryview(self.host.numpy())      # same memory: reading a slot costs 0.05 us instead of 3
        self.base = self.host.data_ptr()
        mapped = ctypes.c_void_p()
        with _OnDevice(device):
            _lib.check(_lib.load().rbf_b200_map_status_slots(self.base, ctypes.byref(mapped)), "rbf_b200_map_status_slots")
        self.mapped = mapped.value              # the ring's address on the device
        self.lock = threading.RLock()           # forward and backward run on different threads
        self.free = collections.deque(range(self.SLOTS))
        self.pending: dict = {}                 # slot -> entry, in the order of their reservation

    def _reserve(self, what) -> _StatusEntry:
        deadline = None
        while True:
            with self.lock:
                if not self.free:
                    self.poll()
                if self.free:
                    slot = self.free.popleft()
                    self.slots[slot] = self._NOT_YET
                    entry = self.pending[slot] = _StatusEntry(slot, what)
                    return entry
            # The ring is full: the oldest word belongs to a call SLOTS calls ago and arrives without any help from this
            # thread. (A device-wide synchronisation here would also drain the caller's copy streams: only when it is late.)
            now = time.monotonic()
            if deadline is None:
                deadline = now + 10.0
            elif now > deadline:
                self.poll(wait=True)
                deadline = None
            time.sleep(0)

    def _retire(self, entry) -> None:
        del self.pending[entry.slot]
        self.free.append(entry.slot)

    def _report(self, code, what) -> None:
        if code == self._NOT_YET & 0xFFFFFFFF:
            raise RuntimeError(f"{what}: the status word did not arrive")
        if what.startswith("range:"):
            raise RuntimeError(
                f"{what[6:]}: float32 inputs exceed float16's range (|x| >= 65504) on a path that runs on "
                "float16 tensor-core operands; its results contain inf / nan. Scale the inputs or use bfloat16"
            )
        raise RuntimeError(
            f"{what}: a device-side wait ran out (site {code >> 24}, work unit {code & 0xFFFFFF}); "
            "the results of that call are incomplete"
        )

    def poll(self, wait=False):
        """Checks the entries whose status word has arrived, oldest first (when ``wait``: of all calls enqueued so far,
        after waiting for the device; calls that other threads enqueue meanwhile are left to a later look)."""
        if not self.pending:
            return
        due = ()
        if wait:
            with self.lock:
                due = {e for e in self.pending.values() if e.state != _RESERVED}
            torch.cuda.synchronize(self.device)
        done, code = [], 0
        with self.lock:
            for slot, e in self.pending.items():
                code = self.slots[slot]
                if code == self._NOT_YET:
                    code = 0
                    if e not in due:
                        if wait or e.state != _ENQUEUED:
                            continue
                        break
                    if e.state == _ENQUEUED:
                        done.append(e)
                        code = self._NOT_YET
                        break
                done.append(e)
                if code != 0:
                    break
            for d in done:
                self._retire(d)
        if code != 0:
            self._report(code & 0xFFFFFFFF, e.what)

    def _enqueue(self, what, call, ring) -> None:
        """``call(slot address)`` enqueues what posts a status word there and returns an error code; ``ring`` is the address
        of the first slot."""
        entry = self._reserve(what)
        try:
            rc = call(ring + 4 * entry.slot)
            entry.state = _ENQUEUED
        except BaseException:
            # whether something was enqueued is not known: the slot is not used again before the device has been waited for
            entry.state = _ABANDONED
            raise
        if rc != 0:                             # nothing was enqueued that could post
            with self.lock:
                self._retire(entry)
            _lib.check(rc, what)
        if _SYNC_STATUS:
            self.poll(wait=True)

    def record_range_check(self, tensors, what):
        """fp32 tensors narrowed to fp16 operands: records (asynchronously, like the status word) whether the
        conversion overflowed, so that a later call raises instead of inf / nan passing silently."""
        flag = torch.zeros(4, dtype=torch.uint8, device=tensors[0].device)
        bad = tensors[0].new_zeros((), dtype=torch.bool)
        for t in tensors:
            bad = bad | torch.isinf(t).any()
        flag[0] = bad
        self.record(flag, "range:" + what)

    def launch(self, what, call) -> None:
        """``call(slot address)`` enqueues a call whose last kernel posts its status word there (0: no posting, while a
        CUDA graph is being captured) and returns its error code."""
        if self.capturing(self.index):
            _lib.check(call(0), what)
            return
        self._enqueue(what, call, self.mapped)

    def record(self, ws, what):
        """Posts the status word at the start of ``ws`` with a kernel of its own."""
        if self.capturing(self.index):
            return
        with _OnDevice(self.device):
            self._enqueue(what, lambda slot: _lib.load().rbf_b200_post_device_status(
                ws.data_ptr(), slot, _stream_ptr(ws.device)), self.base)


_SYNC_STATUS = os.environ.get("RBF_B200_SYNC_STATUS", "0") not in ("", "0")
_monitors: dict = {}


def _monitor(device) -> _StatusMonitor:
    key = device.index if device.index is not None else torch.cuda.current_device()
    m = _monitors.get(key)
    if m is None:
        m = _monitors.setdefault(key, _StatusMonitor(device))
    return m


def check_device_status(device=None) -> None:
    """Waits for every operator call made so far on ``device`` (default: the current one) and raises
    ``RuntimeError`` if one of them ended with a device-side wait that ran out."""
    if device is None:
        device = torch.device("cuda", torch.cuda.current_device())
    _monitor(torch.device(device)).poll(wait=True)


def _narrow(tensors, checked: int, mon, what: str):
    """fp32 (B, H, N, D) tensors as fp16 operands, in one launch that also looks whether one of the first ``checked``
    leaves fp16's range (reported like a status word: by a later call). What the kernel's 16-byte loads cannot take goes
    through PyTorch's conversion."""
    prepared = _lib.host().narrow_f32(tensors, checked)
    if prepared is None:
        halves = [t.to(torch.float16) for t in tensors]
        mon.record_range_check(halves[:checked], what)
        return halves
    enqueue, halves = prepared
    mon.launch("range:" + what, enqueue)
    return halves


def _widen(tensors):
    """Dense fp16 tensors of one shape as fp32, in one launch."""
    return _lib.host().widen_f16(tensors)


def _first_columns(t: torch.Tensor, D: int) -> torch.Tensor:
    return t if t.shape[-1] == D else t[..., :D].contiguous()


def _forward(q, k, v, is_causal: bool, softmax: bool):
    host = _lib.host()
    host.validate("q", q, None)
    D = q.shape[3]
    mon = _monitor(q.device)
    mon.poll()
    # fp32 tensors at head dim <= 64: TF32 operands, as the reference's Triton path uses for them (fp32's exponent range)
    narrowed = q.dtype == torch.float32 and D > 64
    if narrowed:
        _validate("k", k, q)
        _validate("v", v, q)
        q, k, v = _narrow((q, k, v), 3, mon, "rbf_b200_fwd")
    enqueue, out, lse = host.attention_fwd(q, k, v, is_causal, softmax)
    mon.launch("rbf_b200_fwd", enqueue)
    out = _first_columns(out, D)
    if narrowed:
        (out,) = _widen([out])
    return out, lse


def _backward(q, k, v, out, lse, dout, is_causal: bool, sm_scale: float, softmax: bool):
    host = _lib.host()
    host.validate("q", q, None)
    D = q.shape[3]
    mon = _monitor(q.device)
    mon.poll()
    # the non-softmax variant takes the forward output when the caller has it: the single-kernel backward needs it
    narrowed = q.dtype == torch.float32
    if narrowed:
        _validate("k", k, q)
        _validate("v", v, q)
        _validate("dout", dout, q)
        q, k, v, dout, *rest = _narrow((q, k, v, dout) if out is None else (q, k, v, dout, out), 4, mon, "rbf_b200_bwd")
        out = rest[0] if rest else None
    enqueue, *grads = host.attention_bwd(q, k, v, out, lse, dout, is_causal, sm_scale, softmax)
    mon.launch("rbf_b200_bwd", enqueue)
    grads = [_first_columns(g, D) for g in grads]
    return tuple(_widen(grads) if narrowed else grads)


# ---------------------------------------------------------------------------------------------
# rbf_attn_v5::scaled_fwd / scaled_bwd  (rbf_attention.py:651-842)
# ---------------------------------------------------------------------------------------------
@torch.library.custom_op("rbf_attn_v5::scaled_fwd", mutates_args=())
def rbf_scaled_fwd(
    q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, is_causal: bool
) -> tuple[torch.Tensor, torch.Tensor]:
    out, lse = _forward(q, k, v, is_causal, softmax=True)
    return out, lse


@rbf_scaled_fwd.register_fake
def _(q, k, v, is_causal):
    B, H, N_CTX, D_HEAD = q.shape
    return (
        torch.empty_like(q, memory_format=torch.contiguous_format),
        torch.empty((B, H, N_CTX), device=q.device, dtype=torch.float32),
    )


@torch.library.custom_op("rbf_attn_v5::scaled_bwd", mutates_args=())
def rbf_scaled_bwd(
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    out: torch.Tensor,
    L: torch.Tensor,
    dout: torch.Tensor,
    is_causal: bool,
    sm_scale: float,
) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    return _backward(q, k, v, out, L, dout, is_causal, sm_scale, softmax=True)


@rbf_scaled_bwd.register_fake
def _(q, k, v, out, L, dout, is_causal, sm_scale):
    return (
        torch.empty_like(q, memory_format=torch.contiguous_format),
        torch.empty_like(k, memory_format=torch.contiguous_format),
        torch.empty_like(v, memory_format=torch.contiguous_format),
    )


def _scaled_setup_context(ctx, inputs, output):
    q, k, v, is_causal = inputs
    out, L = output
    ctx.save_for_backward(q, k, v, out, L)
    ctx.is_causal = is_causal
    ctx.sm_scale = 1.0 / math.sqrt(q.shape[-1])


def _scaled_backward(ctx, dout, dL):
    # the gradient of L is ignored, as in the reference (rbf_attention.py:830)
    q, k, v, out, L = ctx.saved_tensors
    dq, dk, dv = torch.ops.rbf_attn_v5.scaled_bwd(q, k, v, out, L, dout, ctx.is_causal, ctx.sm_scale)
    return dq, dk, dv, None


torch.library.register_autograd(
    "rbf_attn_v5::scaled_fwd", _scaled_backward, setup_context=_scaled_setup_context
)


# ---------------------------------------------------------------------------------------------
# rbf_attn_v5::non_softmax_fwd / non_softmax_bwd  (rbf_attention.py:1355-1511)
# ---------------------------------------------------------------------------------------------
@torch.library.custom_op("rbf_attn_v5::non_softmax_fwd", mutates_args=())
def rbf_non_softmax_fwd(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, is_causal: bool) -> torch.Tensor:
    return _forward(q, k, v, is_causal, softmax=False)[0]


@rbf_non_softmax_fwd.register_fake
def _(q, k, v, is_causal):
    return torch.empty_like(q, memory_format=torch.contiguous_format)


@torch.library.custom_op("rbf_attn_v5::non_softmax_bwd", mutates_args=())
def rbf_non_softmax_bwd(
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    dout: torch.Tensor,
    is_causal: bool,
    sm_scale: float,
) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    # The reference's operator does not receive the forward output. The single-kernel backward needs it
    # (rowsum_j dS_ij = dO_i . O_i), and recomputing it costs less than the two-kernel backward it saves.
    out = _forward(q, k, v, is_causal, softmax=False)[0]
    return _backward(q, k, v, out, None, dout, is_causal, sm_scale, softmax=False)


@rbf_non_softmax_bwd.register_fake
def _(q, k, v, dout, is_causal, sm_scale):
    return (
        torch.empty_like(q, memory_format=torch.contiguous_format),
        torch.empty_like(k, memory_format=torch.contiguous_format),
        torch.empty_like(v, memory_format=torch.contiguous_format),
    )


# Same backward with the forward output passed in (no counterpart in the reference): what autograd calls, since the
# output is at hand there.
@torch.library.custom_op("rbf_attn_v5::non_softmax_bwd_with_out", mutates_args=())
def rbf_non_softmax_bwd_with_out(
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    out: torch.Tensor,
    dout: torch.Tensor,
    is_causal: bool,
    sm_scale: float,
) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    return _backward(q, k, v, out, None, dout, is_causal, sm_scale, softmax=False)


@rbf_non_softmax_bwd_with_out.register_fake
def _(q, k, v, out, dout, is_causal, sm_scale):
    return (
        torch.empty_like(q, memory_format=torch.contiguous_format),
        torch.empty_like(k, memory_format=torch.contiguous_format),
        torch.empty_like(v, memory_format=torch.contiguous_format),
    )


def _non_softmax_setup_context(ctx, inputs, output):
    q, k, v, is_causal = inputs
    ctx.save_for_backward(q, k, v, output)
    ctx.is_causal = is_causal
    ctx.sm_scale = 1.0 / math.sqrt(q.shape[-1])


def _non_softmax_backward(ctx, dout):
    q, k, v, out = ctx.saved_tensors
    dq, dk, dv = torch.ops.rbf_attn_v5.non_softmax_bwd_with_out(q, k, v, out, dout, ctx.is_causal, ctx.sm_scale)
    return dq, dk, dv, None


torch.library.register_autograd(
    "rbf_attn_v5::non_softmax_fwd", _non_softmax_backward, setup_context=_non_softmax_setup_context
)


# ---------------------------------------------------------------------------------------------
# The attention block's RBF branch as one operator: fused q/k preparation (SuSiE positions, register-position rows,
# key norms) + attention, reading and writing the projection layouts in place. Replaces, for the "rbf_triton" and
# "rbf_non_softmax" attention types with SuSiE positions, the torch ops of rbf_attention.py:1659-1688 and :1761
# (split, broadcast adds, concatenation, transpose copy) and their autograd.
# ---------------------------------------------------------------------------------------------
def _susie_block_fwd(
    qkv: torch.Tensor,
    pos_weight: torch.Tensor,
    reg_pos_emb: torch.Tensor | None,
    table: torch.Tensor,
    num_heads: int,
    softmax: bool,
) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """qkv (B, S, 3 H D), pos_weight (H, D/2), reg_pos_emb (H, R, D) or None, table (>= S - R, D) ->
    (out (B, S, H D), L (B, H, S) fp32 [empty when softmax is False], qk (2, B, S, H, D) = the prepared q', k')."""
    enqueue, out, lse, qk = _lib.host().block_fwd(qkv, pos_weight, reg_pos_emb, table, num_heads, softmax)
    mon = _monitor(out.device)
    mon.poll()
    mon.launch("rbf_b200_fwd (attention block)", enqueue)
    return out, lse, qk


susie_block_fwd = torch.library.custom_op("rbf_attn_b200::susie_block_fwd", mutates_args=())(_susie_block_fwd)


@susie_block_fwd.register_fake
def _(qkv, pos_weight, reg_pos_emb, table, num_heads, softmax):
    B, S, E3 = qkv.shape
    E = E3 // 3
    D = E // num_heads
    return (
        qkv.new_empty((B, S, E)),
        qkv.new_empty((B, num_heads, S) if softmax else (0,), dtype=torch.float32),
        qkv.new_empty((2, B, S, num_heads, D)),
    )


def _susie_block_bwd(
    qkv: torch.Tensor,
    qk: torch.Tensor,
    out: torch.Tensor,
    lse: torch.Tensor,
    dout: torch.Tensor,
    table: torch.Tensor,
    num_registers: int,
    softmax: bool,
) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """-> (dqkv (B, S, 3 H D), d_pos_weight (H, D/2) fp32, d_reg_pos_emb (H, R, D) fp32)."""
    enqueue, dqkv, d_pw, d_rp = _lib.host().block_bwd(qkv, qk, out, lse, dout, table, num_registers, softmax)
    mon = _monitor(qkv.device)
    mon.poll()
    mon.launch("rbf_b200_bwd (attention block)", enqueue)
    return dqkv, d_pw, d_rp


susie_block_bwd = torch.library.custom_op("rbf_attn_b200::susie_block_bwd", mutates_args=())(_susie_block_bwd)


@susie_block_bwd.register_fake
def _(qkv, qk, out, lse, dout, table, num_registers, softmax):
    _, B, S, H, D = qk.shape
    return (
        qkv.new_empty((B, S, 3 * H * D)),
        qkv.new_empty((H, D // 2), dtype=torch.float32),
        qkv.new_empty((H, num_registers, D), dtype=torch.float32),
    )


def _susie_block_setup_context(ctx, inputs, output):
    qkv, pos_weight, reg_pos_emb, table, num_heads, softmax = inputs
    out, lse, qk = output
    ctx.save_for_backward(qkv, qk, out, lse, table)
    ctx.softmax = softmax
    ctx.num_registers = 0 if reg_pos_emb is None else reg_pos_emb.shape[-2]
    ctx.pw_dtype = pos_weight.dtype
    ctx.rp_dtype = None if reg_pos_emb is None else reg_pos_emb.dtype
    ctx.set_materialize_grads(False)


def _susie_block_backward(ctx, dout, dlse, dqk):
    # only `out` carries a gradient: L and the saved q', k' are by-products (the reference ignores dL too)
    qkv, qk, out, lse, table = ctx.saved_tensors
    if dout is None:
        return None, None, None, None, None, None
    bwd = _susie_block_bwd if _direct_backward(qkv, qk, out, lse, dout, table) else torch.ops.rbf_attn_b200.susie_block_bwd
    dqkv, d_pw, d_rp = bwd(qkv, qk, out, lse, dout, table, ctx.num_registers, ctx.softmax)
    d_rp = None if ctx.rp_dtype is None else d_rp.to(ctx.rp_dtype)
    return dqkv, d_pw.to(ctx.pw_dtype), d_rp, None, None, None


torch.library.register_autograd(
    "rbf_attn_b200::susie_block_fwd", _susie_block_backward, setup_context=_susie_block_setup_context
)


class _SusieBlock(torch.autograd.Function):
    """``rbf_attn_b200::susie_block_fwd`` and its autograd formula for calls that go around the operator (``_direct``)."""

    @staticmethod
    def forward(ctx, qkv, pos_weight, reg_pos_emb, table, num_heads, softmax):
        out, lse, qk = _susie_block_fwd(qkv, pos_weight, reg_pos_emb, table, num_heads, softmax)
        _susie_block_setup_context(ctx, (qkv, pos_weight, reg_pos_emb, table, num_heads, softmax), (out, lse, qk))
        return out

    @staticmethod
    def backward(ctx, dout):
        return _susie_block_backward(ctx, dout, None, None)


def susie_block_attention(qkv, pos_weight, reg_pos_emb, table, num_heads, softmax=True):
    """Attention of one block from the fused projection output: (B, S, 3 H D) -> (B, S, H D), causal, with the SuSiE
    position term and the register-position rows added to q and k inside the operator."""
    if type(softmax) is bool and type(num_heads) is int and _direct(qkv, pos_weight, reg_pos_emb, table):
        if _needs_grad(qkv, pos_weight, reg_pos_emb):
            return _SusieBlock.apply(qkv, pos_weight, reg_pos_emb, table, num_heads, softmax)
        return _susie_block_fwd(qkv, pos_weight, reg_pos_emb, table, num_heads, softmax)[0]
    return torch.ops.rbf_attn_b200.susie_block_fwd(qkv, pos_weight, reg_pos_emb, table, num_heads, softmax)[0]


# ---------------------------------------------------------------------------------------------
# Exclusive self attention (the block's apply_xsa option, rbf_attention.py:1757-1759) as one fused pass each way
# ---------------------------------------------------------------------------------------------
@torch.library.custom_op("rbf_attn_b200::xsa_fwd", mutates_args=())
def xsa_fwd(o: torch.Tensor, v: torch.Tensor) -> torch.Tensor:
    """out = o - (o . vh) vh with vh = v / max(|v|, 1e-12), row by row; o, v (B, H, N, D)."""
    _validate("o", o)
    _validate("v", v, o)
    if o.dtype not in _DTYPE_CODE:
        raise ValueError(f"unsupported dtype {o.dtype} (bfloat16 or float16)")
    B, H, N, D = o.shape
    lib = _lib.load()
    oc, vc = _tma_ready(o), _tma_ready(v)
    out = torch.empty((B, H, N, D), dtype=o.dtype, device=o.device)
    with _OnDevice(o.device):
        rc = lib.rbf_b200_xsa_fwd(oc.data_ptr(), vc.data_ptr(), out.data_ptr(), _lib.strides3(oc), _lib.strides3(vc),
                                  _lib.strides3(out), B, H, N, D, _DTYPE_CODE[o.dtype], _stream_ptr(o.device))
    _lib.check(rc, "rbf_b200_xsa_fwd")
    return out


@xsa_fwd.register_fake
def _(o, v):
    return torch.empty_like(o, memory_format=torch.contiguous_format)


@torch.library.custom_op("rbf_attn_b200::xsa_bwd", mutates_args=())
def xsa_bwd(g: torch.Tensor, o: torch.Tensor, v: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
    _validate("o", o)
    _validate("v", v, o)
    g = g.to(o.dtype)
    _validate("g", g, o)
    if o.dtype not in _DTYPE_CODE:
        raise ValueError(f"unsupported dtype {o.dtype} (bfloat16 or float16)")
    B, H, N, D = o.shape
    lib = _lib.load()
    gc, oc, vc = _tma_ready(g), _tma_ready(o), _tma_ready(v)
    d_o = torch.empty((B, H, N, D), dtype=o.dtype, device=o.device)
    d_v = torch.empty_like(d_o)
    with _OnDevice(o.device):
        rc = lib.rbf_b200_xsa_bwd(gc.data_ptr(), oc.data_ptr(), vc.data_ptr(), d_o.data_ptr(), d_v.data_ptr(),
                                  _lib.strides3(gc), _lib.strides3(oc), _lib.strides3(vc), _lib.strides3(d_o),
                                  _lib.strides3(d_v), B, H, N, D, _DTYPE_CODE[o.dtype], _stream_ptr(o.device))
    _lib.check(rc, "rbf_b200_xsa_bwd")
    return d_o, d_v


@xsa_bwd.register_fake
def _(g, o, v):
    return (torch.empty_like(o, memory_format=torch.contiguous_format),
            torch.empty_like(o, memory_format=torch.contiguous_format))


def _xsa_setup_context(ctx, inputs, output):
    o, v = inputs
    ctx.save_for_backward(o, v)


def _xsa_backward(ctx, g):
    o, v = ctx.saved_tensors
    return torch.ops.rbf_attn_b200.xsa_bwd(g, o, v)


torch.library.register_autograd("rbf_attn_b200::xsa_fwd", _xsa_backward, setup_context=_xsa_setup_context)


def exclusive_self_attention(o, v):
    """Removes from every attention output row its component along the value row of the same position."""
    return torch.ops.rbf_attn_b200.xsa_fwd(o, v)


# ---------------------------------------------------------------------------------------------
# Linear layers whose bias gradient is the library's column sum (nn.Linear in train_rbf_transformer.py:143, 216 and
# rbf_attention.py:1625-1626)
# ---------------------------------------------------------------------------------------------
def _column_sums(x: torch.Tensor) -> torch.Tensor:
    """fp32 sums over the rows of a 16-bit CUDA matrix (rows, cols), cols a multiple of 8."""
    return _lib.host().column_sums(x)


column_sums = torch.library.custom_op("rbf_attn_b200::column_sums", mutates_args=())(_column_sums)


@column_sums.register_fake
def _(x):
    return x.new_empty(x.shape[1], dtype=torch.float32)


class _LinearBiasSum(torch.autograd.Function):
    """``F.linear`` whose backward takes the bias gradient from ``column_sums`` (the two GEMMs are PyTorch's)."""

    @staticmethod
    def forward(ctx, x, weight, bias):
        ctx.save_for_backward(x, weight)
        return torch.nn.functional.linear(x, weight, bias)

    @staticmethod
    def backward(ctx, g):
        x, weight = ctx.saved_tensors
        g2 = g.reshape(-1, g.shape[-1])
        dx = dw = db = None
        if ctx.needs_input_grad[0]:
            dx = g.matmul(weight)
        if ctx.needs_input_grad[1]:
            dw = g2.t().mm(x.reshape(-1, x.shape[-1]))
        if ctx.needs_input_grad[2]:
            sums = _column_sums if _direct_backward(g2) else torch.ops.rbf_attn_b200.column_sums
            db = sums(g2).to(g.dtype)
        return dx, dw, db


def _gelu_fwd(h: torch.Tensor) -> torch.Tensor:
    """Exact (erf) GELU of a 16-bit CUDA tensor whose element count is a multiple of 8."""
    return _lib.host().gelu_fwd(h)


gelu_fwd = torch.library.custom_op("rbf_attn_b200::gelu_fwd", mutates_args=())(_gelu_fwd)


@gelu_fwd.register_fake
def _(h):
    return torch.empty_like(h, memory_format=torch.contiguous_format)


def _gelu_bwd(h: torch.Tensor, dy: torch.Tensor, with_bias: bool) -> tuple[torch.Tensor, torch.Tensor]:
    """dh = dy * gelu'(h) for (..., cols) tensors and, with ``with_bias``, its fp32 sum over all leading dims."""
    return _lib.host().gelu_bwd(h, dy, with_bias)


gelu_bwd = torch.library.custom_op("rbf_attn_b200::gelu_bwd", mutates_args=())(_gelu_bwd)


@gelu_bwd.register_fake
def _(h, dy, with_bias):
    return (torch.empty_like(h, memory_format=torch.contiguous_format),
            h.new_empty(h.shape[-1] if with_bias else 0, dtype=torch.float32))


class _LinearGelu(torch.autograd.Function):
    """``gelu(F.linear(x, weight, bias))``: the GEMMs are PyTorch's, the activation and its backward - which also
    yields the bias gradient - are the library's."""

    @staticmethod
    def forward(ctx, x, weight, bias):
        h = torch.nn.functional.linear(x, weight, bias)
        ctx.save_for_backward(x, weight, h)
        ctx.bias = bias         # a link for create_graph: its value is not read again, so it may change in place
        return (_gelu_fwd if _direct(h) else torch.ops.rbf_attn_b200.gelu_fwd)(h)

    @staticmethod
    def backward(ctx, g):
        x, weight, h = ctx.saved_tensors
        bwd = _gelu_bwd if _direct_backward(h, g) else torch.ops.rbf_attn_b200.gelu_bwd
        dh, dbias = bwd(h, g, ctx.needs_input_grad[2])
        if torch.is_grad_enabled():         # h was saved without the graph that made it
            dh, dbias = (_FirstOrderOnly.apply("linear_gelu", t, x, weight, ctx.bias, g) for t in (dh, dbias))
        dh2 = dh.reshape(-1, dh.shape[-1])
        dx = dh.matmul(weight) if ctx.needs_input_grad[0] else None
        dw = dh2.t().mm(x.reshape(-1, x.shape[-1])) if ctx.needs_input_grad[1] else None
        db = dbias.to(g.dtype) if ctx.needs_input_grad[2] else None
        return dx, dw, db


def linear_gelu(module: torch.nn.Linear, x: torch.Tensor) -> torch.Tensor:
    """``F.gelu(module(x))`` (exact form) on the library's kernels for 16-bit CUDA activations; anything else through
    PyTorch."""
    if x.is_cuda and x.dtype in _DTYPE_CODE:
        weight, bias = module.weight, module.bias
        if bias is not None and weight.dtype == x.dtype and module.out_features % 8 == 0:
            if _direct(x, weight, bias) and not _needs_grad(x, weight, bias):
                return _gelu_fwd(torch.nn.functional.linear(x, weight, bias))
            return _LinearGelu.apply(x, weight, bias)
    return torch.nn.functional.gelu(module(x))


def linear(module: torch.nn.Linear, x: torch.Tensor) -> torch.Tensor:
    """``module(x)``; for 16-bit CUDA activations and a bias, the bias gradient comes from the library's column-sum
    kernel instead of PyTorch's generic reduction."""
    if torch.is_grad_enabled() and x.is_cuda and x.dtype in _DTYPE_CODE:
        weight, bias = module.weight, module.bias
        if bias is not None and weight.dtype == x.dtype and module.out_features % 8 == 0 and bias.requires_grad:
            return _LinearBiasSum.apply(x, weight, bias)
    return module(x)


# ---------------------------------------------------------------------------------------------
# LayerNorm of the language model's blocks (nn.LayerNorm, train_rbf_transformer.py:139-150, 215, 241)
# ---------------------------------------------------------------------------------------------
def layer_norm_supported(x: torch.Tensor, weight, bias) -> bool:
    """16-bit CUDA activations with an affine LayerNorm over 256, 512, 768 or 1024 columns."""
    return (x.is_cuda and x.dtype in _DTYPE_CODE and weight is not None and bias is not None
            and weight.dtype == x.dtype and bias.dtype == x.dtype
            and x.shape[-1] % 256 == 0 and 0 < x.shape[-1] <= 1024)


def _layer_norm_fwd(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor,
                   eps: float) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """y = (x - mean) * rstd * weight + bias over the last dim; returns (y, mean, rstd), the statistics in fp32."""
    return _lib.host().layer_norm_fwd(x, None, weight, bias, eps)[1:]


layer_norm_fwd = torch.library.custom_op("rbf_attn_b200::layer_norm_fwd", mutates_args=())(_layer_norm_fwd)


@layer_norm_fwd.register_fake
def _(x, weight, bias, eps):
    rows = x.numel() // x.shape[-1]
    return (torch.empty_like(x, memory_format=torch.contiguous_format), x.new_empty(rows, dtype=torch.float32),
            x.new_empty(rows, dtype=torch.float32))


def _layer_norm_bwd(x: torch.Tensor, dy: torch.Tensor, weight: torch.Tensor, mean: torch.Tensor,
                   rstd: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    return _lib.host().layer_norm_bwd(x, dy, None, weight, mean, rstd)


layer_norm_bwd = torch.library.custom_op("rbf_attn_b200::layer_norm_bwd", mutates_args=())(_layer_norm_bwd)


@layer_norm_bwd.register_fake
def _(x, dy, weight, mean, rstd):
    return (torch.empty_like(x, memory_format=torch.contiguous_format), torch.empty_like(weight),
            torch.empty_like(weight))


def _ln_setup_context(ctx, inputs, output):
    x, weight, _bias, _eps = inputs
    ctx.save_for_backward(x, weight, output[1], output[2])
    ctx.set_materialize_grads(False)


def _ln_backward(ctx, g_y, _g_mean, _g_rstd):
    if g_y is None:
        return None, None, None, None
    x, weight, mean, rstd = ctx.saved_tensors
    bwd = _layer_norm_bwd if _direct_backward(x, g_y, weight, mean, rstd) else torch.ops.rbf_attn_b200.layer_norm_bwd
    dx, dgamma, dbeta = bwd(x, g_y, weight, mean, rstd)
    return dx, dgamma, dbeta, None


torch.library.register_autograd("rbf_attn_b200::layer_norm_fwd", _ln_backward, setup_context=_ln_setup_context)


class _LayerNorm(torch.autograd.Function):
    """``rbf_attn_b200::layer_norm_fwd`` and its autograd formula for calls that go around the operator (``_direct``)."""

    @staticmethod
    def forward(ctx, x, weight, bias, eps):
        output = _layer_norm_fwd(x, weight, bias, eps)
        _ln_setup_context(ctx, (x, weight, bias, eps), output)
        return output[0]

    @staticmethod
    def backward(ctx, g_y):
        return _ln_backward(ctx, g_y, None, None)


def layer_norm(x, weight, bias, eps: float = 1e-5):
    """``F.layer_norm(x, (x.shape[-1],), weight, bias, eps)`` on the library's kernels (see layer_norm_supported)."""
    if type(eps) is float and _direct(x, weight, bias):
        if _needs_grad(x, weight, bias):
            return _LayerNorm.apply(x, weight, bias, eps)
        return _layer_norm_fwd(x, weight, bias, eps)[0]
    return torch.ops.rbf_attn_b200.layer_norm_fwd(x, weight, bias, eps)[0]


def _add_layer_norm_fwd(x: torch.Tensor, residual: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor,
                       eps: float) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor]:
    """s = x + residual (rounded to the dtype, as the separate addition leaves it) and y = LayerNorm(s) from one pass;
    returns (s, y, mean, rstd)."""
    return _lib.host().layer_norm_fwd(x, residual, weight, bias, eps)


add_layer_norm_fwd = torch.library.custom_op("rbf_attn_b200::add_layer_norm_fwd", mutates_args=())(_add_layer_norm_fwd)


@add_layer_norm_fwd.register_fake
def _(x, residual, weight, bias, eps):
    rows = x.numel() // x.shape[-1]
    return (torch.empty_like(x, memory_format=torch.contiguous_format),
            torch.empty_like(x, memory_format=torch.contiguous_format), x.new_empty(rows, dtype=torch.float32),
            x.new_empty(rows, dtype=torch.float32))


def _layer_norm_bwd_add(x: torch.Tensor, dy: torch.Tensor, dres: torch.Tensor, weight: torch.Tensor, mean: torch.Tensor,
                       rstd: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """The LayerNorm backward with ``dres`` (the gradient reaching x along the skip path) added to dx before the
    rounding: (dx, dgamma, dbeta)."""
    return _lib.host().layer_norm_bwd(x, dy, dres, weight, mean, rstd)


layer_norm_bwd_add = torch.library.custom_op("rbf_attn_b200::layer_norm_bwd_add", mutates_args=())(_layer_norm_bwd_add)


@layer_norm_bwd_add.register_fake
def _(x, dy, dres, weight, mean, rstd):
    return (torch.empty_like(x, memory_format=torch.contiguous_format), torch.empty_like(weight),
            torch.empty_like(weight))


def _add_ln_setup_context(ctx, inputs, output):
    _x, _residual, weight, _bias, _eps = inputs
    ctx.save_for_backward(output[0], weight, output[2], output[3])
    ctx.set_materialize_grads(False)


def _add_ln_backward(ctx, g_s, g_y, _g_mean, _g_rstd):
    # the sum has one gradient, shared by x and residual: the LayerNorm's plus whatever reached s from elsewhere
    if g_y is None:
        return g_s, g_s, None, None, None
    s, weight, mean, rstd = ctx.saved_tensors
    direct = _direct_backward(s, g_y, g_s, weight, mean, rstd)
    if g_s is None:
        bwd = _layer_norm_bwd if direct else torch.ops.rbf_attn_b200.layer_norm_bwd
        dx, dgamma, dbeta = bwd(s, g_y, weight, mean, rstd)
    else:
        bwd = _layer_norm_bwd_add if direct else torch.ops.rbf_attn_b200.layer_norm_bwd_add
        dx, dgamma, dbeta = bwd(s, g_y, g_s, weight, mean, rstd)
    return dx, dx, dgamma, dbeta, None


torch.library.register_autograd("rbf_attn_b200::add_layer_norm_fwd", _add_ln_backward,
                                setup_context=_add_ln_setup_context)


class _AddLayerNorm(torch.autograd.Function):
    """``rbf_attn_b200::add_layer_norm_fwd`` and its autograd formula for calls that go around the operator."""

    @staticmethod
    def forward(ctx, x, residual, weight, bias, eps):
        output = _add_layer_norm_fwd(x, residual, weight, bias, eps)
        _add_ln_setup_context(ctx, (x, residual, weight, bias, eps), output)
        return output[0], output[1]

    @staticmethod
    def backward(ctx, g_s, g_y):
        return _add_ln_backward(ctx, g_s, g_y, None, None)


def add_layer_norm(x, residual, weight, bias, eps: float = 1e-5):
    """``s = x + residual; y = F.layer_norm(s, (s.shape[-1],), weight, bias, eps)`` in one pass over the activations
    (and one in the backward, which takes the skip path's gradient with it): returns (s, y)."""
    if type(eps) is float and _direct(x, residual, weight, bias):
        if _needs_grad(x, residual, weight, bias):
            return _AddLayerNorm.apply(x, residual, weight, bias, eps)
        return _add_layer_norm_fwd(x, residual, weight, bias, eps)[:2]
    s, y, _mean, _rstd = torch.ops.rbf_attn_b200.add_layer_norm_fwd(x, residual, weight, bias, eps)
    return s, y


# ---------------------------------------------------------------------------------------------
# Cross entropy of the language-model step (torch.nn.CrossEntropyLoss(ignore_index=-100),
# train_rbf_transformer.py:282): loss and d(loss)/d(logits) from one kernel
# ---------------------------------------------------------------------------------------------
_CE_DTYPE = {torch.bfloat16: 0, torch.float16: 1, torch.float32: 2}


def _cross_entropy_fwd(logits: torch.Tensor, targets: torch.Tensor, ignore_index: int) -> tuple[torch.Tensor, torch.Tensor]:
    """Mean cross entropy over the rows whose target is not ``ignore_index`` (fp32 scalar) and its gradient with
    respect to ``logits`` (same shape and dtype), from one pass: logits (rows, cols) with unit column stride,
    targets (rows,) int64."""
    if logits.dim() != 2 or targets.dim() != 1 or targets.shape[0] != logits.shape[0]:
        raise ValueError(f"logits must be (rows, cols) and targets (rows,), got {tuple(logits.shape)}, {tuple(targets.shape)}")
    if not logits.is_cuda or targets.device != logits.device:
        raise RuntimeError("logits and targets must be CUDA tensors on one device: rbf_attention_b200 has no CPU path")
    if logits.dtype not in _CE_DTYPE:
        raise ValueError(f"unsupported dtype {logits.dtype} (bfloat16, float16 or float32)")
    if targets.dtype != torch.int64:
        raise ValueError(f"targets must be int64, got {targets.dtype}")
    rows, cols = logits.shape
    x = logits if logits.stride(1) == 1 and (rows <= 1 or logits.stride(0) >= cols) else logits.contiguous()
    t = targets.contiguous()
    counted = ((t != ignore_index) & (t >= 0) & (t < cols)).sum()
    grad_scale = 1.0 / counted.to(torch.float32)          # no counted row: inf * 0 = nan, as torch's mean of nothing
    loss_rows = torch.empty(rows, dtype=torch.float32, device=x.device)
    dlogits = torch.empty((rows, cols), dtype=x.dtype, device=x.device)
    with _OnDevice(x.device):
        rc = _lib.load().rbf_b200_cross_entropy(
            x.data_ptr(), t.data_ptr(), grad_scale.data_ptr(), loss_rows.data_ptr(), dlogits.data_ptr(), rows, cols,
            x.stride(0) if rows > 1 else cols, cols, int(ignore_index), _CE_DTYPE[x.dtype], _stream_ptr(x.device))
    _lib.check(rc, "rbf_b200_cross_entropy")
    return loss_rows.sum() * grad_scale, dlogits


cross_entropy_fwd = torch.library.custom_op("rbf_attn_b200::cross_entropy_fwd", mutates_args=())(_cross_entropy_fwd)


@cross_entropy_fwd.register_fake
def _(logits, targets, ignore_index):
    return logits.new_empty((), dtype=torch.float32), torch.empty_like(logits, memory_format=torch.contiguous_format)


def _scale_unless_one(x: torch.Tensor, factor: torch.Tensor) -> None:
    """x *= factor (a one-element tensor) unless factor == 1, decided on the device."""
    if not x.is_contiguous():
        raise ValueError("x must be contiguous")
    f = factor.reshape(1).to(device=x.device, dtype=torch.float32)
    with _OnDevice(x.device):
        rc = _lib.load().rbf_b200_scale_unless_one(x.data_ptr(), f.data_ptr(), x.numel(), _CE_DTYPE[x.dtype],
                                                   _stream_ptr(x.device))
    _lib.check(rc, "rbf_b200_scale_unless_one")


scale_unless_one_ = torch.library.custom_op("rbf_attn_b200::scale_unless_one_", mutates_args=("x",))(_scale_unless_one)


def _ce_setup_context(ctx, inputs, output):
    ctx.save_for_backward(output[1])        # an output, so that under create_graph it is linked to the logits
    ctx.set_materialize_grads(False)        # no zero tensor of the logits' size for the unused second output


def _ce_backward(ctx, g_loss, _g_dlogits):
    # the gradient was formed by the forward; it is scaled in place (a no-op for the usual g_loss = 1), so a graph
    # retained for a second backward pass with g_loss != 1 would see it scaled twice
    if g_loss is None:
        return None, None, None
    (dlogits,) = ctx.saved_tensors
    with torch.no_grad():
        if _direct(dlogits, g_loss):
            _scale_unless_one(dlogits, g_loss)
            torch.autograd.graph.increment_version(dlogits)     # as the operator layer does for what it mutates
        else:
            torch.ops.rbf_attn_b200.scale_unless_one_(dlogits, g_loss)
    if torch.is_grad_enabled():
        return _FirstOrderOnly.apply("cross_entropy", dlogits, g_loss), None, None
    return dlogits.detach(), None, None


torch.library.register_autograd("rbf_attn_b200::cross_entropy_fwd", _ce_backward, setup_context=_ce_setup_context)


class _CrossEntropy(torch.autograd.Function):
    """``rbf_attn_b200::cross_entropy_fwd`` and its autograd formula for calls that go around the operator."""

    @staticmethod
    def forward(ctx, logits, targets, ignore_index):
        output = _cross_entropy_fwd(logits, targets, ignore_index)
        _ce_setup_context(ctx, (logits, targets, ignore_index), output)
        return output

    @staticmethod
    def backward(ctx, g_loss, g_dlogits):
        return _ce_backward(ctx, g_loss, g_dlogits)


def cross_entropy(logits, targets, ignore_index: int = -100):
    """``F.cross_entropy(logits, targets, ignore_index=ignore_index)`` (mean reduction) for 2-D CUDA logits, with the
    gradient produced by the forward kernel."""
    if type(ignore_index) is int and _direct(logits, targets):
        if _needs_grad(logits):
            return _CrossEntropy.apply(logits, targets, ignore_index)[0]
        return _cross_entropy_fwd(logits, targets, ignore_index)[0]
    return torch.ops.rbf_attn_b200.cross_entropy_fwd(logits, targets, ignore_index)[0]


# ---------------------------------------------------------------------------------------------
# Wrappers with the reference's names (rbf_attention.py:848-853)
# ---------------------------------------------------------------------------------------------
class _ScaledAttention(torch.autograd.Function):
    """``rbf_attn_v5::scaled_fwd`` and its autograd formula for calls that go around the operator (``_direct``)."""

    @staticmethod
    def forward(ctx, q, k, v, is_causal):
        out, lse = _forward(q, k, v, is_causal, softmax=True)
        ctx.save_for_backward(q, k, v, out, lse)
        ctx.is_causal = is_causal
        return out

    @staticmethod
    def backward(ctx, dout):
        q, k, v, out, lse = ctx.saved_tensors
        sm_scale = 1.0 / math.sqrt(q.shape[-1])
        if _direct_backward(q, k, v, out, lse, dout):
            return *_backward(q, k, v, out, lse, dout, ctx.is_causal, sm_scale, softmax=True), None
        return *torch.ops.rbf_attn_v5.scaled_bwd(q, k, v, out, lse, dout, ctx.is_causal, sm_scale), None


class _NonSoftmaxAttention(torch.autograd.Function):
    """``rbf_attn_v5::non_softmax_fwd`` and its autograd formula for calls that go around the operator (``_direct``)."""

    @staticmethod
    def forward(ctx, q, k, v, is_causal):
        out = _forward(q, k, v, is_causal, softmax=False)[0]
        ctx.save_for_backward(q, k, v, out)
        ctx.is_causal = is_causal
        return out

    @staticmethod
    def backward(ctx, dout):
        q, k, v, out = ctx.saved_tensors
        sm_scale = 1.0 / math.sqrt(q.shape[-1])
        if _direct_backward(q, k, v, out, dout):
            return *_backward(q, k, v, out, None, dout, ctx.is_causal, sm_scale, softmax=False), None
        return *torch.ops.rbf_attn_v5.non_softmax_bwd_with_out(q, k, v, out, dout, ctx.is_causal, sm_scale), None


def run_triton_rbf(q, k, v, is_causal=True):
    """Softmax RBF attention. The name is the reference's; nothing here uses Triton."""
    if type(is_causal) is bool and _direct(q, k, v):
        if _needs_grad(q, k, v):
            return _ScaledAttention.apply(q, k, v, is_causal)
        return _forward(q, k, v, is_causal, softmax=True)[0]
    return torch.ops.rbf_attn_v5.scaled_fwd(q, k, v, is_causal)[0]


def run_triton_non_softmax_rbf(q, k, v, is_causal=True):
    """Non-softmax RBF attention ``exp(-g|q-k|^2) V``. The name is the reference's."""
    if type(is_causal) is bool and _direct(q, k, v):
        if _needs_grad(q, k, v):
            return _NonSoftmaxAttention.apply(q, k, v, is_causal)
        return _forward(q, k, v, is_causal, softmax=False)[0]
    return torch.ops.rbf_attn_v5.non_softmax_fwd(q, k, v, is_causal)
