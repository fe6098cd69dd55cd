"""LayerNorm of rows of up to 128 columns: two rows per warp, odd row counts and rows behind the last one."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 2, 33, 9473])          # 9473 = one more than a whole sweep of the forward's grid
@pytest.mark.parametrize("d", [8, 72, 128, 136])
@pytest.mark.parametrize("dres", [False, True])
def test_forward_and_backward_against_fp32(M, d, dres):
    from diloco_swarm_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(M + d)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    whole = (rnd(M + 2, d) * 2 + 0.5).to(torch.bfloat16)          # rows behind the last one hold other values
    x, w, b = whole[:M], rnd(d), rnd(d)
    y, mean, rstd = K.layernorm_fwd(x, w, b)
    xr, wr, br = x.double().requires_grad_(), w.double().requires_grad_(), b.double().requires_grad_()
    yr = F.layer_norm(xr, (d,), wr, br, 1e-5)
    dy, r = rnd(M, d).to(torch.bfloat16), (rnd(M, d).to(torch.bfloat16) if dres else None)
    yr.backward(dy.double())
    dw, db, rs = (torch.zeros(d, device="cuda") for _ in range(3))
    dx = K.layernorm_bwd(dy, x, w, mean, rstd, dw, db, dres=r, dres_sum=rs if dres else None)
    # outputs rounded once to bf16 (2^-9); fp32 sums over M rows in another order for the column sums
    ref_dx = xr.grad + (r.double() if dres else 0)
    assert torch.allclose(y.double(), yr, rtol=2 ** -8, atol=2 ** -9)
    assert torch.allclose(dx.double(), ref_dx, rtol=2 ** -8, atol=2 ** -9 * ref_dx.abs().max().item())
    for got, ref in ((dw, wr.grad), (db, br.grad)) + (((rs, r.double().sum(0)),) if dres else ()):
        assert torch.allclose(got.double(), ref, rtol=1e-4, atol=1e-5 * M ** 0.5)
