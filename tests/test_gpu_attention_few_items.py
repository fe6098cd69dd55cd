"""Attention forward of no more items than SMs, whose output rows go straight from their threads, against the same sequences
among many, whose rows pass through shared memory."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one token, part of a tile, whole tiles, a row more than a tile, several items on either side; both head sizes
@pytest.mark.parametrize("T,nh,hs", [(1, 1, 64), (24, 4, 32), (127, 3, 64), (128, 4, 32), (129, 2, 64), (640, 12, 64), (1000, 4, 32)])
def test_few_items_are_as_many(T, nh, hs):
    from diloco_swarm_b200.ops._lib import Status
    from diloco_swarm_b200.ops.attention import attention_fwd
    st, d = Status(torch.device("cuda")), nh * hs
    items = -(-T // 128) * nh
    assert items <= 148
    B = 148 // items + 1                          # more items than SMs
    g = torch.Generator(device="cuda").manual_seed(T)
    qkv = torch.randn(B * T, 3 * d, device="cuda", generator=g).to(torch.bfloat16)
    many, ctx = attention_fwd(qkv, B, T, nh, status=st)
    for b in (0, B - 1):
        few, one = attention_fwd(qkv[b * T:(b + 1) * T].contiguous(), 1, T, nh, status=st)
        assert torch.equal(few, many[b * T:(b + 1) * T])
        assert torch.equal(one.lse, ctx.lse[b * nh * T:(b + 1) * nh * T])
    torch.cuda.synchronize()
    st.raise_if_set()
