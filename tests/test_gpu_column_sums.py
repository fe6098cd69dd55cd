"""Bias gradients that come out of the kernels which write dh and dqkv, against the pass that reads them once more."""
import pytest
import torch

from helpers import make_config, single_world

pytestmark = pytest.mark.gpu


# few rows (cluster kernel), several tiles (many rows), one and two tiles per sequence, rows that end inside a tile;
# head sizes 32 and 64
@pytest.mark.parametrize("B,T", [(1, 1), (3, 50), (1, 128), (2, 129), (9, 128), (20, 100), (6, 256)])
@pytest.mark.parametrize("heads,width", [(4, 128), (4, 256), (12, 768)])
def test_sums_are_those_of_a_pass_of_their_own(B, T, heads, width):
    from diloco_swarm_b200.models.engine_b200 import B200Engine
    from diloco_swarm_b200.models.gpt2 import GPT2Config
    from diloco_swarm_b200.ops import kernels as K
    cfg = make_config(model={"n_layer": 2, "n_head": heads, "n_embd": width, "vocab_size": 512, "block_size": 256})
    eng = B200Engine(GPT2Config(block_size=256, vocab_size=512, n_layer=2, n_head=heads, n_embd=width), single_world(), cfg,
                     torch.device("cuda", 0))
    gen = torch.Generator(device="cuda").manual_seed(7)
    ids = torch.randint(0, 512, (B, T + 1), device="cuda", generator=gen)
    mask = torch.ones(B, T, dtype=torch.long, device="cuda")
    got = []
    for apart in (True, False):
        eng.grad.zero_()
        K.set_deterministic(apart)          # sums in atomics are not for a deterministic backward
        try:
            eng.forward_backward(0, ids[:, :-1].contiguous(), None, ids[:, 1:].contiguous(), mask, 1.0)
        finally:
            K.set_deterministic(False)
        torch.cuda.synchronize()
        eng.check_status()
        got.append({k: eng.g32(k).double().clone() for k, _, _ in eng.specs if k.endswith("bias")})
    seen = 0
    for k, a in got[0].items():
        b = got[1][k]
        # terms rounded to bf16 (2^-9 of each) on one side, fp32 on the other; rows are independent, so the sums differ by less
        # than one rounding of the terms' norm, which the sum's norm over the columns is not below by more than sqrt(rows)
        assert (a - b).norm() <= 2 ** -8 * a.norm() * max(1.0, (B * T) ** 0.5 / 8) + 1e-9, k
        seen += "c_fc" in k or "c_attn" in k
    assert seen == 4


@pytest.mark.parametrize("B,T", [(1, 24), (1, 128), (2, 100), (1, 255)])
@pytest.mark.parametrize("heads,width", [(4, 128), (12, 768)])
def test_few_rows_repeat_themselves(B, T, heads, width):
    """Up to 255 rows every sum of a bias gradient is added up in one order, so the same pass gives the same bits."""
    from diloco_swarm_b200.models.engine_b200 import B200Engine
    from diloco_swarm_b200.models.gpt2 import GPT2Config
    cfg = make_config(model={"n_layer": 2, "n_head": heads, "n_embd": width, "vocab_size": 512, "block_size": 256})
    eng = B200Engine(GPT2Config(block_size=256, vocab_size=512, n_layer=2, n_head=heads, n_embd=width), single_world(), cfg,
                     torch.device("cuda", 0))
    gen = torch.Generator(device="cuda").manual_seed(11)
    ids = torch.randint(0, 512, (B, T + 1), device="cuda", generator=gen)
    mask = torch.ones(B, T, dtype=torch.long, device="cuda")
    first = None
    for _ in range(12):
        eng.grad.zero_()
        eng.forward_backward(0, ids[:, :-1].contiguous(), None, ids[:, 1:].contiguous(), mask, 1.0)
        torch.cuda.synchronize()
        got = {k: eng.g32(k).clone() for k, _, _ in eng.specs if k.endswith("bias")}
        first = first or got
        for k in got:
            assert torch.equal(got[k], first[k]), k
    eng.check_status()
