"""GELU without its derivative is the same number as with it, on every kernel."""
import pytest
import torch

from test_gpu_gemm import _mk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (300, 520, 200), (1000, 136, 768)])
@pytest.mark.parametrize("bn", [0, 128, 256, 384, 512])
def test_the_same_activation(M, N, K, bn):
    from diloco_swarm_b200.ops import kernels as Kn
    a, b, bias = _mk((M, K), seed=1), _mk((N, K), 0.05, seed=2), torch.randn(N, device="cuda")
    both = [torch.full((M + 8, N + 8), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    Kn.gemm(a, b, mode=Kn.EPI_GELU, bias=bias, aux_out=torch.empty(M, N, dtype=torch.bfloat16, device="cuda"), out=both[0][:M, :N], bn=bn)
    Kn.gemm(a, b, mode=Kn.EPI_GELU, bias=bias, out=both[1][:M, :N], bn=bn)
    if bn:
        assert torch.equal(both[0], both[1])
    else:          # other tiles may be chosen: the same sums in another order, rounded once
        assert torch.allclose(both[0].float(), both[1].float(), rtol=2 ** -7, atol=2 ** -9)
    assert bool((both[1][M:] == 7).all()) and bool((both[1][:, N:] == 7).all())
