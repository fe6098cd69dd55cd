"""Inputs that the stage executor must not be given: it reads addresses, so a tensor of another type or size is refused
before any launch, in every pass of the engine.  A stand-in for the executor says when a call gets through to it."""
import contextlib
import types

import pytest
import torch

from diloco_swarm_b200.models.engine_b200 import B200Engine

B, T, D = 2, 6, 16


class Reached(Exception):
    pass


class Executor:
    d, lock = D, contextlib.nullcontext()

    def enter(self):
        return None

    def sizes(self, *a):
        raise Reached

    def area(self, *a):
        raise Reached


@pytest.fixture
def engine():
    eng = B200Engine.__new__(B200Engine)
    eng.exec, eng.head_chunks, eng.is_last, eng.side, eng.blocks = Executor(), 1, True, None, [None]
    eng._native = lambda: True
    eng._overlap, eng.fused, eng.world = False, False, types.SimpleNamespace(num_replicas=1)
    return eng


def passes(eng, ids, hidden):
    tg = torch.zeros(B, T, dtype=torch.long)
    return [lambda: eng.forward(0, ids, hidden), lambda: eng.forward_backward(0, ids, hidden, tg, None, 1.0),
            lambda: eng.forward_loss(ids, hidden, tg, None, 1.0), lambda: eng.forward_infer(ids, hidden)]


@pytest.mark.parametrize("dtype,good", [(torch.long, True), (torch.int32, False), (torch.float32, False)])
def test_token_ids(engine, dtype, good):
    engine.is_first = True
    for call in passes(engine, torch.zeros(B, T, dtype=dtype), None):
        with pytest.raises(Reached if good else AssertionError):
            call()


@pytest.mark.parametrize("shape,good", [((B, T, D), True), ((B, T, 4, D // 4), True), ((B, T, D - 8), False), ((B, T, D + 8), False),
                                        ((B, T), False)])
def test_hidden_state(engine, shape, good):
    engine.is_first = False
    for call in passes(engine, None, torch.zeros(shape, dtype=torch.bfloat16)):
        with pytest.raises(Reached if good else AssertionError):
            call()


@pytest.mark.parametrize("shape,good", [((B, T, D), True), ((B * T, D), True), ((B, T, D - 8), False), ((B, T, 2 * D), False),
                                        ((2 * B, T, D), False)])
def test_gradient_of_the_output(engine, shape, good):
    engine.stash = {0: {"area": None, "ids": None, "x": None, "B": B, "T": T}}
    with pytest.raises(Reached if good else AssertionError):
        engine.backward(0, torch.zeros(shape, dtype=torch.bfloat16))
