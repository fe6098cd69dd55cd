"""Passes that are replayed as CUDA graphs against the same passes queued launch by launch, with other inputs, in other
buffers, every time."""
import pytest
import torch

from helpers import make_config
from test_gpu_engine import _batch, _engines
from test_gpu_stage_exec import _stages

pytestmark = pytest.mark.gpu


def _close(a, b):
    # dQ is summed by fp32 reductions in any order, then rounded to bf16: an element may round the other way, and what it
    # goes into differs by that
    assert torch.allclose(a.float(), b.float(), rtol=1e-2, atol=1e-3 * b.float().abs().max().item())


def _both(monkeypatch, make):
    """The same object with and without graphs."""
    out = [make()]
    monkeypatch.setenv("DSWARM_GRAPHS", "0")
    return out + [make()]


def test_a_whole_model(monkeypatch):
    pair = _both(monkeypatch, lambda: _engines()[1])
    cfg = make_config()
    for i in range(6):
        ids, tg, mask = _batch(cfg, B=3, T=50, seed=i)
        got = []
        for eng in pair:
            eng.grad.zero_()
            loss, _ = eng.forward_backward(0, ids.clone(), None, tg.clone(), mask.clone(), 0.5)
            eng._join()
            ev = eng.forward_loss(ids, None, tg, mask, 0.5)
            got.append((eng.forward_infer(ids, None), loss.clone(), ev, eng.grad.clone()))
        (o, l, e, g), (o2, l2, e2, g2) = got
        assert torch.equal(o, o2) and abs(l.item() - l2.item()) < 1e-5 and abs(e.item() - e2.item()) < 1e-5
        _close(g, g2)
    for eng in pair:
        eng.check_status()
    # forward, head before and behind the loss, backward from the third microbatch on; infer and the forward and head of
    # the evaluation likewise
    assert pair[0].exec.graphs() == (5 * 4 + 5 * 2 + 5, 0) and pair[1].exec.graphs() == (0, 0)


def test_a_middle_stage(monkeypatch):
    cfg = make_config(model={"n_layer": 3}, swarm={"num_stages": 3})
    pair = _both(monkeypatch, lambda: _stages(cfg)[1])
    g = torch.Generator(device="cuda").manual_seed(4)
    got = [[], []]
    for i in range(6):
        x, dy = (torch.randn(2, 50, 128, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
        for k, mid in enumerate(pair):
            y = mid.forward(0, None, x.clone())
            got[k].append((y, mid.backward(0, dy.clone())))
    for mid in pair:
        mid._join()
    torch.cuda.synchronize()
    for (y, dx), (y2, dx2) in zip(*got):
        assert torch.equal(y, y2)
        _close(dx, dx2)
    _close(pair[0].grad, pair[1].grad)
    for mid in pair:
        mid.check_status()
    assert pair[0].exec.graphs() == (2 * 5, 0) and pair[1].exec.graphs() == (0, 0)


@pytest.mark.parametrize("stage", [0, 1, 2])
def test_a_stage_with_neighbours_captures_while_it_warms_up(stage):
    """Behind warmup() the passes of up to four microbatches in flight are replayed at once and nothing is captured: in a
    step the device may be held by a receive that waits for a peer."""
    cfg = make_config(model={"n_layer": 3}, swarm={"num_stages": 3})
    eng = _stages(cfg)[stage]
    eng.warmup(2, 50, in_flight=4)
    x = torch.randn(2, 50, 128, device="cuda").to(torch.bfloat16)
    ids, tg, mask = _batch(cfg, B=2, T=50)

    def step(T):
        i, h, t, m = ids[:, :T], x[:, :T], tg[:, :T], mask[:, :T]
        if stage == 2:
            for k in range(4):
                eng.forward_backward(k, None, h, t, m, 0.5)
            return
        for k in range(4):
            eng.forward(k, i if stage == 0 else None, h if stage else None)
        for k in range(4):
            eng.backward(k, h)
    before = eng.exec.graphs()[0]
    step(50)
    assert eng.exec.graphs() == (before + 4 * (4 if stage == 2 else 2), 0)
    before = eng.exec.graphs()[0]
    for _ in range(3):
        step(40)                                         # a size that warmup has not seen
    eng._join()
    torch.cuda.synchronize()
    eng.check_status()
    assert eng.exec.graphs() == (before, 0)
