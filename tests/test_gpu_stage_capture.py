"""Passes of the engine under a CUDA graph capture of the caller's, after the same engine has trained and replayed."""
import pytest
import torch

from test_gpu_engine import _batch, _engines

pytestmark = pytest.mark.gpu


def test_captured_passes_equal_the_eager_ones():
    cfg, eng, _ = _engines()
    ids, tg, mask = _batch(cfg, B=3, T=50, seed=1)
    other = _batch(cfg, B=3, T=50, seed=2)
    for _ in range(4):                                   # queued, captured by the executor, replayed; side work outstanding
        eng.forward_backward(0, other[0], None, other[1], other[2], 0.5)
    eng._join()
    want = [eng.forward_infer(ids, None), eng.forward_loss(ids, None, tg, mask, 0.5)]
    eng.grad.zero_()
    loss, _ = eng.forward_backward(0, ids, None, tg, mask, 0.5)
    eng.sync_gradients()
    want += [loss, eng.grad.clone()]
    eng.forward_backward(0, other[0], None, other[1], other[2], 0.5)
    eng._join()
    torch.cuda.synchronize()
    static = [torch.zeros_like(t) for t in (ids, tg, mask)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        infer = eng.forward_infer(static[0], None)
        ev = eng.forward_loss(static[0], None, static[1], static[2], 0.5)
        trained, _ = eng.forward_backward(0, static[0], None, static[1], static[2], 0.5)
        eng.sync_gradients()
    for s, t in zip(static, (ids, tg, mask)):
        s.copy_(t)
    for _ in range(2):
        eng.forward_backward(0, other[0], None, other[1], other[2], 0.5)      # passes of its own in between
        eng._join()
        eng.grad.zero_()
        graph.replay()
        torch.cuda.synchronize()
        eng.check_status()
        assert torch.equal(infer, want[0])
        assert abs(ev.item() - want[1].item()) < 1e-5 and abs(trained.item() - want[2].item()) < 1e-5
        # fp32 sums of the gradients in another order
        assert torch.allclose(eng.grad, want[3], rtol=1e-3, atol=1e-5 * want[3].abs().max().item())
