"""Library calls beside a CUDA graph capture on another thread."""
import threading
import time

import numpy as np
import pytest

import eiger_b200 as gx
from tests.helpers import to_dev

pytestmark = pytest.mark.gpu


def test_thread_that_ends_during_a_capture():
    # What a thread keeps for its calls is given back when it ends, which must
    # not end the capture of another thread.
    import torch
    x = to_dev(np.arange(100_000) % 3)
    y = torch.ones(1000, device="cuda")
    side, capturing = torch.cuda.Stream(), torch.cuda.Stream()
    called, may_end = threading.Event(), threading.Event()
    counts = []

    def worker():
        counts.append(gx.count_nonzero(x, stream=side))
        called.set()
        may_end.wait(30)

    torch.cuda.synchronize()
    t = threading.Thread(target=worker)
    t.start()
    assert called.wait(30)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=capturing):
        z = y * 2
        may_end.set()
        t.join(30)
        time.sleep(0.2)  # the thread's own objects go after Python has let it end
        z = z + 1
    g.replay()
    torch.cuda.synchronize()
    assert counts == [66_666] and bool((z == 3).all())
