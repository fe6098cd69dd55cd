"""The split-K cluster GEMM for few rows against a plain fp32 matmul of the same bf16 inputs."""
import pytest
import torch

from test_gpu_gemm import _close, _mk

pytestmark = pytest.mark.gpu

# one row, a ragged tile, exactly one tile, a second tile of one row; column and k remainders; one k-block
SHAPES = [(1, 64, 512), (120, 768, 768), (128, 136, 640), (129, 264, 1032), (300, 512, 64), (77, 200, 3072)]
TILES = [(32, 1), (32, 4), (64, 1), (64, 2), (64, 8), (128, 1), (128, 4), (128, 8)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("bn,split", TILES)
def test_epilogues(M, N, K, bn, split):
    from diloco_swarm_b200.ops import kernels as Kn
    from diloco_swarm_b200.ops._lib import Status
    if split > (K + 63) // 64:
        pytest.skip("fewer k-blocks than slices")
    st = Status(torch.device("cuda"))
    kw = dict(bn=1000 + bn, split_k=split, status=st)
    a, b = _mk((M, K), seed=1), _mk((N, K), 0.05, seed=2)
    bias = torch.randn(N, device="cuda")
    acc = a.float() @ b.float().t()
    guard = 7.0

    def padded():
        return torch.full((M + 8, N + 8), guard, dtype=torch.bfloat16, device="cuda")

    def untouched(t):
        assert bool((t[M:, :] == guard).all()) and bool((t[:, N:] == guard).all())
    o = padded()
    Kn.gemm(a, b, bias=bias, out=o[:M, :N], **kw)
    _close(o[:M, :N], acc + bias, "bias"), untouched(o)
    o, dg = padded(), padded()
    Kn.gemm(a, b, mode=Kn.EPI_GELU, bias=bias, aux_out=dg[:M, :N], out=o[:M, :N], **kw)
    x = (acc + bias).requires_grad_(True)
    torch.nn.functional.gelu(x).sum().backward()
    _close(o[:M, :N], torch.nn.functional.gelu(x.detach()), "gelu"), untouched(o)
    _close(dg[:M, :N], x.grad, "gelu derivative"), untouched(dg)
    res = _mk((M, N), seed=3)
    o = padded()
    Kn.gemm(a, b, mode=Kn.EPI_RESID, bias=bias, resid=res, out=o[:M, :N], **kw)
    _close(o[:M, :N], acc + bias + res.float(), "residual"), untouched(o)
    if bn >= 64:                                     # B stored [K, N], as in dx = dy W
        o = padded()
        Kn.gemm(a, b.t().contiguous(), b_t=False, mode=Kn.EPI_MUL, aux_in=res, out=o[:M, :N], **kw)
        _close(o[:M, :N], acc * res.float(), "multiply"), untouched(o)
    torch.cuda.synchronize()
    st.raise_if_set()
