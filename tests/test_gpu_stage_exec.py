"""The native stage executor: microbatches in flight, changing sizes and both gradient paths."""
import pytest
import torch

from helpers import make_config, single_world
from test_gpu_engine import _batch, _engines

pytestmark = pytest.mark.gpu


def _grads(eng):
    return {k: eng.g32(k).flatten().clone() for k, _, _ in eng.specs}


def _stages(cfg):
    from diloco_swarm_b200.models.engine_b200 import B200Engine
    from diloco_swarm_b200.models.gpt2 import GPT2Config
    mc = cfg.model
    g = GPT2Config(block_size=mc.block_size, vocab_size=mc.vocab_size, n_layer=mc.n_layer, n_head=mc.n_head, n_embd=mc.n_embd)
    out = []
    for stage in range(3):
        w = single_world()
        w.num_stages, w.stage = 3, stage
        out.append(B200Engine(g, w, cfg, torch.device("cuda", 0)))
    return out


@pytest.mark.parametrize("layers", [3, 7])
def test_interleaved_microbatches_of_different_sizes(layers):
    """Three stages, microbatches of three shapes in flight at once and their backwards in another order: every
    gradient equals that of the same microbatches one after the other (fp32 sums in another order)."""
    cfg = make_config(model={"n_layer": layers}, swarm={"num_stages": 3})
    batches = [_batch(cfg, B=b, T=t, seed=i) for i, (b, t) in enumerate([(4, 64), (3, 50), (1, 128), (4, 64)])]
    results = []
    for order in ([[0], [1], [2], [3]], [[0, 1, 2, 3]]):
        st = _stages(cfg)
        for group in order:
            mids = {}
            for k in group:
                ids, tg, mask = batches[k]
                mids[k] = st[1].forward(k, None, st[0].forward(k, ids, None))
            for k in reversed(group):
                ids, tg, mask = batches[k]
                _, dx = st[2].forward_backward(k, None, mids[k], tg, mask, 0.5)
                st[0].backward(k, st[1].backward(k, dx))
        torch.cuda.synchronize()
        for e in st:
            e.check_status()
        results.append([_grads(e) for e in st])
    for a, b in zip(*results):
        for k in a:
            assert torch.allclose(a[k], b[k], rtol=1e-3, atol=1e-5 * a[k].abs().max().item() + 1e-9), k


def test_a_middle_stage_replays_its_passes():
    """forward and backward of a stage without ends, queued, captured and replayed: the same gradients every time."""
    cfg = make_config(model={"n_layer": 3}, swarm={"num_stages": 3})
    mid = _stages(cfg)[1]
    g = torch.Generator(device="cuda").manual_seed(3)
    x, dy = (torch.randn(3, 50, 128, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    seen = []
    for _ in range(4):
        mid.grad.zero_()
        y = mid.forward(0, None, x)
        dx = mid.backward(0, dy)
        mid._join()
        seen.append((y.clone(), dx.clone(), mid.grad.clone()))
    torch.cuda.synchronize()
    mid.check_status()
    for y, dx, grad in seen[1:]:
        assert torch.equal(y, seen[0][0])
        # dQ is summed by fp32 reductions in any order, then rounded to bf16: an element may round the other way
        assert torch.allclose(dx.float(), seen[0][1].float(), rtol=2 ** -7, atol=2 ** -8 * seen[0][1].abs().max().item())
        assert torch.allclose(grad, seen[0][2], rtol=1e-2, atol=1e-3 * seen[0][2].abs().max().item())


def test_inference_logits_match_the_loss_path():
    """forward_infer's fp32 logits against autograd's, at a length below one tile."""
    cfg, eb, et = _engines()
    ids, tg, mask = _batch(cfg, B=5, T=24)
    out = eb.forward_infer(ids, None)
    ref = et.model(input_ids=ids).float()
    assert out.dtype == torch.float32 and out.shape == ref.shape
    assert (out - ref).abs().max() < 3e-2 * ref.abs().max()


def test_replayed_passes_equal_the_queued_ones():
    """The same microbatch three times (queued, captured, replayed), with other inputs in between and from another
    stream: loss, logits and gradients stay the same."""
    cfg, eng, _ = _engines()
    a, b = _batch(cfg, B=3, T=50, seed=1), _batch(cfg, B=3, T=50, seed=2)
    seen = []
    side = torch.cuda.Stream()
    for i in range(5):
        if i == 3:
            side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side if i >= 3 else torch.cuda.current_stream()):
            ids, tg, mask = (t.clone() for t in a)              # the caller's tensors lie elsewhere every time
            eng.grad.zero_()
            loss, _ = eng.forward_backward(0, ids, None, tg, mask, 0.5)
            eng._join()
            out = eng.forward_infer(ids, None)
            seen.append((loss, out, eng.grad.clone()))
            eng.forward_backward(0, b[0], None, b[1], b[2], 0.5)
    torch.cuda.synchronize()
    eng.check_status()
    for loss, out, grad in seen[1:]:
        assert abs(loss.item() - seen[0][0].item()) < 1e-5 and torch.equal(out, seen[0][1])
        assert torch.allclose(grad, seen[0][2], rtol=1e-3, atol=1e-5 * seen[0][2].abs().max().item())


def test_a_middle_stage_takes_its_tensors_anywhere():
    """Hidden state and gradient in other buffers every pass, before and after the pass has been captured: outputs belong
    to the buffers of their own pass and earlier ones keep theirs."""
    cfg = make_config(model={"n_layer": 3}, swarm={"num_stages": 3})
    mid, other = _stages(cfg)[1], _stages(cfg)[1]
    g = torch.Generator(device="cuda").manual_seed(4)
    ins = [tuple(torch.randn(2, 50, 128, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2)) for _ in range(5)]
    got = []
    for x, dy in ins:
        y = mid.forward(0, None, x)
        got.append((y, mid.backward(0, dy)))
    torch.cuda.synchronize()
    mid.check_status()
    for (x, dy), (y, dx) in zip(ins, got):          # a fresh stage's first pass, queued launch by launch
        other.exec._idle.clear()
        assert torch.equal(other.forward(0, None, x), y)
        ref = other.backward(0, dy)
        # dQ is summed by fp32 reductions in any order, then rounded to bf16: an element may round the other way
        assert torch.allclose(dx.float(), ref.float(), rtol=2 ** -7, atol=2 ** -8 * ref.abs().max().item())
