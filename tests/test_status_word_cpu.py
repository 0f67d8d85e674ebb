"""The status word of a device (kernels._StatusWord) from several threads."""
import threading
import time

import torch


def test_threads_that_come_first_share_one_word(monkeypatch):
    """Making the word releases the interpreter lock.  Two words for one device would part what the GEMMs report into from what
    is read and cleared."""
    from triton_int8_b200 import kernels as K
    made = []

    class Slow:
        def __init__(self, dev):
            time.sleep(0.05)
            made.append(dev)

    monkeypatch.setattr(K, "_StatusWord", Slow)
    monkeypatch.setattr(K, "_STATUS", {})
    got, start = [], threading.Barrier(8)

    def use():
        start.wait()
        got.append(K._status_of(torch.device("cuda", 3)))

    ts = [threading.Thread(target=use) for _ in range(8)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert len(made) == 1 and all(g is got[0] for g in got)
