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
@pytest.mark.parametrize("B,T", [(1, 100), (20, 100), (40, 128), (3, 300), (2, 640), (1, 1000)])
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


@pytest.mark.parametrize("executor", [True, False])
def test_a_tied_head_and_its_embedding_add_in_one_order(executor):
    """One block between a head of 50304 rows, whose weight gradient takes longer than the rest of the backward, and the
    embedding that it shares its weights with; two microbatches."""
    from diloco_swarm_b200.models.engine_b200 import B200Engine
    from diloco_swarm_b200.models.gpt2 import GPT2Config
    from diloco_swarm_b200.ops import kernels as K
    shape = {"n_layer": 1, "n_head": 4, "n_embd": 128, "vocab_size": 50304, "block_size": 256, "parameter_sharing": True}
    cfg = make_config(model=shape)
    cfg.train.deterministic = True
    try:
        eng = B200Engine(GPT2Config(**shape), single_world(), cfg, torch.device("cuda", 0))
        if not executor:
            eng.exec = None
        gen = torch.Generator(device="cuda").manual_seed(5)
        ids = torch.randint(0, 600, (2, 8, 257), device="cuda", generator=gen)
        mask = torch.ones(8, 256, dtype=torch.long, device="cuda")
        first = None
        for _ in range(6):
            eng.grad.zero_()
            for m in ids:
                eng.forward_backward(0, m[:, :-1].contiguous(), None, m[:, 1:].contiguous(), mask, 1.0)
            eng._join()
            torch.cuda.synchronize()
            first = eng.grad.clone() if first is None else first
            assert torch.equal(eng.grad, first)
        eng.check_status()
    finally:
        K.set_deterministic(False)


@pytest.mark.parametrize("B,T,nh,hs", [(1, 129, 1, 64), (2, 384, 4, 32), (3, 1000, 12, 64)])
def test_ordered_attention_backward(B, T, nh, hs):
    """One launch per kv tile: the same dK and dV, and a dQ whose fp32 sums differ in their order only."""
    from diloco_swarm_b200.ops import kernels as K
    from diloco_swarm_b200.ops._lib import Status
    from diloco_swarm_b200.ops.attention import attention_bwd, attention_fwd
    st, d = Status(torch.device("cuda")), nh * hs
    qkv, dout = torch.randn(B * T, 3 * d, device="cuda").to(torch.bfloat16), torch.randn(B * T, d, device="cuda").to(torch.bfloat16)
    _, ctx = attention_fwd(qkv, B, T, nh, status=st)
    any_order = attention_bwd(dout, ctx)
    K.set_deterministic(True)
    try:
        got = [attention_bwd(dout, ctx) for _ in range(6)]
    finally:
        K.set_deterministic(False)
    torch.cuda.synchronize()
    st.raise_if_set()
    assert all(torch.equal(g, got[0]) for g in got) and torch.equal(got[0][:, d:], any_order[:, d:])
    # both rounded to bf16 (2^-9 of a value each) after fp32 sums of at most eight terms
    assert (got[0][:, :d].double() - any_order[:, :d].double()).norm() <= 2 ** -8 * any_order[:, :d].double().norm()
