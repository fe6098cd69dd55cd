"""Threads that share an engine: the library calls of a pass, which use the same work areas, are not interleaved with
those of another thread's pass."""
import threading
import time
import types

import pytest
import torch

from diloco_swarm_b200.models.engine_b200 import B200Engine

B, T, D = 2, 6, 16


class Executor:
    d = D

    def __init__(self):
        self.lock, self.calls = threading.RLock(), []

    def enter(self):
        return None

    def sizes(self, *a):
        return 1, 1

    def take(self, *a):
        return types.SimpleNamespace(buf=torch.empty(1))

    def area(self, *a):
        return torch.empty(1)

    def give(self, *a):
        pass

    def _call(self, *a):
        self.calls.append(threading.get_ident())
        time.sleep(1e-3)                             # the other thread's turn, if it gets one

    forward = head = backward = _call


@pytest.mark.parametrize("name", ["forward_backward", "forward_loss"])
def test_a_pass_is_queued_whole(name):
    eng = B200Engine.__new__(B200Engine)
    eng.exec, eng.head_chunks, eng.is_first, eng.is_last = Executor(), 1, False, True
    eng.side, eng.blocks, eng.device = None, [None], torch.device("cpu")
    eng._native = lambda: True
    eng._overlap, eng.fused, eng.world = False, False, types.SimpleNamespace(num_replicas=1)
    hidden, tg = torch.zeros(B, T, D, dtype=torch.bfloat16), torch.zeros(B, T, dtype=torch.long)
    args = (0, None, hidden, tg, None, 1.0) if name == "forward_backward" else (None, hidden, tg, None, 1.0)

    def work():
        for _ in range(10):
            getattr(eng, name)(*args)
    threads = [threading.Thread(target=work) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    per = 3 if name == "forward_backward" else 2
    calls = eng.exec.calls
    assert len(calls) == 20 * per
    for i in range(0, len(calls), per):
        assert len(set(calls[i:i + per])) == 1
