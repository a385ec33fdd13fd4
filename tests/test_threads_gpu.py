"""Operators called from several threads."""
import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_other_threads_run_while_a_launch_waits():
    """A thread that fills the device's queue behind half a second of work waits in its launches; the
    interpreter stays free for the others meanwhile."""
    from flashlight_b200 import functions as F
    x, out = torch.ones(1024, device="cuda"), torch.empty(1024, device="cuda")
    F.add(x, x, out=out)
    torch.cuda.synchronize()

    def fill():
        torch.cuda._sleep(1_000_000_000)
        for _ in range(4000):
            F.add(x, x, out=out)

    worker = threading.Thread(target=fill)
    longest, last = 0.0, time.perf_counter()
    worker.start()
    while worker.is_alive():
        time.sleep(0.001)
        now = time.perf_counter()
        longest, last = max(longest, now - last), now
    worker.join()
    torch.cuda.synchronize()
    assert longest < 0.2
    assert torch.equal(out, 2 * x)
