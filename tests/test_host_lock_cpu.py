"""The extension's entry points copy, allocate and enqueue without the interpreter's lock: what a full launch queue or the
allocator waits for may be another Python thread. The one entry point that also works on host tensors stands for them."""

import threading
import time

import torch

from rbf_attention_b200 import _lib


def test_other_threads_run_while_a_call_copies(built_library):
    host = _lib.host()
    x = torch.zeros(1 << 26, dtype=torch.float16)
    ticks, stop = [], threading.Event()

    def watch():
        while not stop.is_set():
            ticks.append(time.perf_counter())
            time.sleep(2e-4)

    thread = threading.Thread(target=watch)
    thread.start()
    threads = torch.get_num_threads()
    torch.set_num_threads(1)
    try:
        seen = 0
        for _ in range(5):
            start = time.perf_counter()
            (y,) = host.widen_f16([x])
            end = time.perf_counter()
            margin = (end - start) / 5
            seen += sum(start + margin < t < end - margin for t in ticks)
    finally:
        torch.set_num_threads(threads)
        stop.set()
        thread.join()
    assert y.dtype == torch.float32 and not y.count_nonzero()
    assert end - start > 2e-3 and seen > 0, (end - start, seen)
