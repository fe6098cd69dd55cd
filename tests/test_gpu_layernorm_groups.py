"""LayerNorm backward of rows wider than 128 columns: groups of one to eight warps, rows that do not fill a group's step,
a column count that ends inside the group's last warp."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one round of 148 blocks is 4736 rows up to 256 columns, 2368 up to 512, 1480 up to 768, 1184 up to 1024 and fewer above
@pytest.mark.parametrize("M", [1, 3, 37, 1487, 5003])
@pytest.mark.parametrize("d", [136, 256, 264, 768, 776, 1024, 1288, 1600, 1800, 2048])
@pytest.mark.parametrize("dres", [False, True])
def test_backward_against_64_bits(M, d, dres):
    from diloco_swarm_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(M + d)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    whole = (rnd(M + 2, d) * 2 + 0.5).to(torch.bfloat16)          # rows behind the last one hold other values
    x, w, b = whole[:M], rnd(d), rnd(d)
    _, mean, rstd = K.layernorm_fwd(x, w, b)
    dy, r = rnd(M, d).to(torch.bfloat16), (rnd(M, d).to(torch.bfloat16) if dres else None)
    dw, db, rs = (torch.ones(d, device="cuda") for _ in range(3))
    dx = K.layernorm_bwd(dy, x, w, mean, rstd, dw, db, dres=r, dres_sum=rs if dres else None)
    x6, dy6 = x.double(), dy.double()
    mu = x6.mean(1, keepdim=True)
    rs6 = (x6.var(1, unbiased=False, keepdim=True) + 1e-5).rsqrt()
    xhat, gy = (x6 - mu) * rs6, dy6 * w.double()
    ref = rs6 * (gy - gy.mean(1, keepdim=True) - xhat * (gy * xhat).mean(1, keepdim=True)) + (r.double() if dres else 0)
    # dx is rounded once to bf16 (2^-9 of the value); column sums are fp32 sums of M terms of size one
    assert torch.allclose(dx.double(), ref, rtol=2 ** -8, atol=2 ** -9 * ref.abs().max().item())
    sums = [(dw, (dy6 * xhat).sum(0)), (db, dy6.sum(0))] + ([(rs, r.double().sum(0))] if dres else [])
    for got, want in sums:
        assert torch.allclose(got.double() - 1, want, rtol=1e-4, atol=1e-5 * max(M, 4) ** 0.5)
    assert dres or torch.equal(rs, torch.ones_like(rs))
