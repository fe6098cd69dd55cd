"""--train.deterministic: gradients are added up in a fixed order."""
import pytest
import torch

from helpers import make_config, single_world

pytestmark = pytest.mark.gpu


# one block to a column and a cluster of eight; rows that do not fill the blocks' shares; column groups that end inside a block
@pytest.mark.parametrize("M,N", [(1, 8), (255, 264), (256, 256), (257, 8), (1000, 776), (5003, 3072), (32768, 264)])
def test_ordered_column_sums(M, N):
    from diloco_swarm_b200.ops import kernels as K
    x = torch.randn(M, N + 8, device="cuda").to(torch.bfloat16)[:, :N]
    K.set_deterministic(True)
    try:
        got = [torch.ones(N + 8, device="cuda") for _ in range(6)]
        for g in got:
            K.colsum_accum(x, g[:N])
    finally:
        K.set_deterministic(False)
    assert all(torch.equal(g, got[0]) for g in got) and bool((got[0][N:] == 1).all())
    # fp32 sums of M terms of size one, at most M / 64 of them in a row
    assert torch.allclose(got[0][:N].double() - 1, x.double().sum(0), rtol=1e-5, atol=2 ** -22 * M ** 0.5 * max(1, M / 64) ** 0.5 + 1e-6)


@pytest.mark.parametrize("heads,width", [(4, 128), (12, 768)])
@pytest.mark.parametrize("B,T", [(1, 100), (20, 100), (40, 128)])
def test_the_same_pass_gives_the_same_gradients(B, T, heads, width):
    from diloco_swarm_b200.models.engine_b200 import B200Engine
    from diloco_swarm_b200.models.gpt2 import GPT2Config
    from diloco_swarm_b200.ops import kernels as K
    cfg = make_config(model={"n_layer": 2, "n_head": heads, "n_embd": width, "vocab_size": 512, "block_size": 1024})
    cfg.train.deterministic = True
    try:
        eng = B200Engine(GPT2Config(block_size=1024, vocab_size=512, n_layer=2, n_head=heads, n_embd=width), single_world(), cfg,
                         torch.device("cuda", 0))
        gen = torch.Generator(device="cuda").manual_seed(5)
        ids = torch.randint(0, 512, (B, T + 1), device="cuda", generator=gen)
        mask = torch.ones(B, T, dtype=torch.long, device="cuda")
        first = None
        for _ in range(8):
            eng.grad.zero_()
            eng.forward_backward(0, ids[:, :-1].contiguous(), None, ids[:, 1:].contiguous(), mask, 1.0)
            torch.cuda.synchronize()
            got = {k: eng.g32(k).clone() for k, _, _ in eng.specs}
            first = first or got
            for k in got:
                assert torch.equal(got[k], first[k]), k
        eng.check_status()
    finally:
        K.set_deterministic(False)
