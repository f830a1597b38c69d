"""The ring of status slots that operator calls post into (``ops._StatusMonitor``), with a host array in the place of mapped
memory and the test in the place of the device: what is tested is the bookkeeping between threads and after errors."""

import contextlib
import threading
import time
import types

import pytest
import torch

from rbf_attention_b200 import ops


@pytest.fixture
def ring(monkeypatch):
    monkeypatch.setattr(torch.Tensor, "pin_memory", lambda t: t)
    monkeypatch.setattr(ops, "_OnDevice", lambda device: contextlib.nullcontext())
    monkeypatch.setattr(ops._lib, "load", lambda: types.SimpleNamespace(rbf_b200_map_status_slots=lambda *a: 0,
                                                                         rbf_b200_last_error=lambda: b"refused"))
    monkeypatch.setattr(torch._C, "_cuda_isCurrentStreamCapturing", lambda: False, raising=False)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda device=None: None)
    ring = ops._StatusMonitor(torch.device("cuda", 0))
    ring.mapped = 0
    return ring


def _post(ring, word=0):
    """A call whose kernels run at once."""
    def call(address):
        ring.slots[address // 4] = word
        return 0
    return call


def test_a_call_that_is_being_enqueued_is_not_late(ring):
    """Another thread has taken its slot and not launched yet: neither a waiting look nor one from a later call may report
    it, and the calls behind it are still checked."""
    taken, go = threading.Event(), threading.Event()

    def slow(address):
        taken.set()
        assert go.wait(30)
        ring.slots[address // 4] = 0
        return 0

    thread = threading.Thread(target=ring.launch, args=("slow", slow))
    thread.start()
    assert taken.wait(30)
    try:
        ring.poll(wait=True)
        ring.launch("quick", _post(ring))
        ring.poll(wait=True)
        ring.launch("bad", _post(ring, (3 << 24) | 5))
        with pytest.raises(RuntimeError, match=r"bad: a device-side wait ran out \(site 3, work unit 5\)"):
            ring.poll()
    finally:
        go.set()
        thread.join()
    ring.poll(wait=True)
    assert not ring.pending


def test_a_call_enqueued_during_the_wait_is_left_to_a_later_look(ring, monkeypatch):
    ring.launch("first", _post(ring))
    slot = []
    monkeypatch.setattr(torch.cuda, "synchronize",
                        lambda device=None: ring.launch("second", lambda address: slot.append(address // 4) or 0))
    ring.poll(wait=True)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda device=None: None)
    ring.slots[slot[0]] = 0
    ring.poll(wait=True)
    assert not ring.pending


def test_a_call_left_by_an_exception_gives_its_slot_back(ring):
    def broken(address):
        raise KeyboardInterrupt

    with pytest.raises(KeyboardInterrupt):
        ring.launch("broken", broken)
    start = time.monotonic()
    for i in range(2 * ring.SLOTS):
        ring.launch(str(i), _post(ring))
        ring.poll()
    assert time.monotonic() - start < 5
    ring.poll(wait=True)
    assert not ring.pending
    with pytest.raises((RuntimeError, ValueError)):
        ring.launch("refused", lambda address: 1)
    ring.poll(wait=True)
    assert not ring.pending


def test_a_word_that_never_arrives_is_reported_once(ring):
    ring.launch("lost", lambda address: 0)
    ring.launch("later", _post(ring))
    ring.poll()
    with pytest.raises(RuntimeError, match="lost: the status word did not arrive"):
        ring.poll(wait=True)
    ring.poll(wait=True)
    assert not ring.pending


def test_a_full_ring_waits_for_its_oldest_word(ring):
    slots = []
    for i in range(ring.SLOTS):
        ring.launch(str(i), lambda address: slots.append(address // 4) or 0)
    timer = threading.Timer(0.2, lambda: ring.slots.__setitem__(slots[0], 0))
    timer.start()
    ring.launch("one more", lambda address: slots.append(address // 4) or 0)
    timer.join()
    assert slots[-1] == slots[0] and sorted(slots[1:]) == list(range(ring.SLOTS))
    for slot in slots[1:]:
        ring.slots[slot] = 0
    ring.poll(wait=True)
    assert not ring.pending


def test_the_oldest_error_is_reported_first_and_each_once(ring):
    ring.launch("a", _post(ring))
    ring.launch("b", _post(ring, (2 << 24) | 1))
    ring.launch("range:c", _post(ring, 1))
    with pytest.raises(RuntimeError, match="b: a device-side wait"):
        ring.poll()
    with pytest.raises(RuntimeError, match="c: float32 inputs exceed"):
        ring.poll(wait=True)
    ring.poll(wait=True)
    assert not ring.pending


def test_threads_share_the_ring(ring):
    errors = []

    def work(n):
        try:
            for i in range(600):
                ring.launch(f"{n}.{i}", _post(ring))
                if i % 37 == 0:
                    ring.poll(wait=True)
                else:
                    ring.poll()
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(n,)) for n in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    ring.poll(wait=True)
    assert not ring.pending
