"""tcgen05 attention at sequence lengths that no tile divides, against fp32 PyTorch attention."""
import pytest
import torch

from test_gpu_attention import _ref

pytestmark = pytest.mark.gpu

# one token; less than a tile; a tile and one row; one row short of a tile; several work items per CTA; ends inside a
# tile at the end of the tensor and in front of another sequence
SHAPES = [(1, 1, 1, 64), (5, 24, 12, 64), (3, 129, 4, 32), (2, 255, 3, 64), (20, 133, 12, 64), (3, 777, 5, 64), (7, 40, 4, 32)]


@pytest.mark.parametrize("B,T,nh,hs", SHAPES)
def test_forward_and_backward(B, T, nh, hs):
    from diloco_swarm_b200.ops._lib import Status
    from diloco_swarm_b200.ops.attention import attention_bwd, attention_fwd
    torch.manual_seed(2)
    st = Status(torch.device("cuda"))
    d = nh * hs
    qkv = torch.randn(B * T, 3 * d, device="cuda").to(torch.bfloat16)
    dout = torch.randn(B * T, d, device="cuda").to(torch.bfloat16)
    out, ctx = attention_fwd(qkv, B, T, nh, status=st)
    dqkv = attention_bwd(dout, ctx)
    torch.cuda.synchronize()
    st.raise_if_set()
    assert ctx.native
    x = qkv.float().requires_grad_(True)
    ref, lse = _ref(x, B, T, nh)
    # P, the output and its row are rounded to bf16 (2^-9 of the value each); sums over T of independent roundings
    # stay below that of one value at the largest element
    assert (out.float() - ref).abs().max() < 2e-2 * ref.abs().max() + 2e-3
    assert (ctx.lse.view(B, nh, T) - lse).abs().max() < 2e-2
    ref.backward(dout.float())
    for name, sl in (("dq", slice(0, d)), ("dk", slice(d, 2 * d)), ("dv", slice(2 * d, 3 * d))):
        got, want = dqkv[:, sl].float(), x.grad[:, sl]
        assert (got - want).abs().max() < 3e-2 * want.abs().max() + 3e-3, name
