"""Sequences of a batch stay apart: infinities and NaN in one of them change nothing in the others."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# shorter than a tile; a tile and five rows; the last row of a tile missing; whole tiles; both head sizes
SHAPES = [(4, 24, 2, 64), (5, 133, 3, 64), (3, 255, 2, 64), (3, 256, 2, 64), (4, 40, 4, 32), (3, 129, 4, 32)]


@pytest.mark.parametrize("poison", [float("inf"), float("nan")])
@pytest.mark.parametrize("B,T,nh,hs", SHAPES)
def test_a_spoiled_sequence_leaves_its_neighbours_alone(B, T, nh, hs, poison):
    from diloco_swarm_b200.ops._lib import Status
    from diloco_swarm_b200.ops.attention import attention_bwd, attention_fwd
    torch.manual_seed(5)
    st = Status(torch.device("cuda"))
    d = nh * hs
    qkv = torch.randn(B, T, 3 * d, device="cuda").to(torch.bfloat16)
    dout = torch.randn(B, T, d, device="cuda").to(torch.bfloat16)
    bad = B // 2
    others = [b for b in range(B) if b != bad]
    got = []
    for spoil in (False, True):
        if spoil:
            qkv, dout = qkv.clone(), dout.clone()
            qkv[bad], dout[bad] = poison, poison
        out, ctx = attention_fwd(qkv.view(B * T, 3 * d), B, T, nh, status=st)
        dqkv = attention_bwd(dout.view(B * T, d), ctx)
        got.append((out.view(B, T, d)[others], ctx.lse.view(B, nh, T)[others], dqkv.view(B, T, 3 * d)[others].float()))
    torch.cuda.synchronize()
    st.raise_if_set()
    (out, lse, grad), (out2, lse2, grad2) = got
    assert torch.isfinite(grad).all() and torch.equal(out, out2) and torch.equal(lse, lse2)
    assert torch.equal(grad[..., d:], grad2[..., d:])
    # the kv tiles of a row add to its dQ in any order: fp32 sums that may round to the neighbouring bf16 value
    dq, dq2 = grad[..., :d], grad2[..., :d]
    assert torch.allclose(dq, dq2, rtol=2 ** -7, atol=2 ** -12 * dq.abs().max().item())
