"""The residual epilogue with a low half: out + aux_out is acc + bias + resid + aux_in to fp32 precision, whichever kernel
the size rule picks, for products that are not exact in bf16."""
import pytest
import torch

from test_gpu_gemm import _mk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bn,split", [(128, 1), (256, 1), (384, 1), (512, 1), (1064, 2), (0, 1)])
@pytest.mark.parametrize("M,N,K", [(300, 264, 1032), (129, 8, 64), (520, 392, 768)])
def test_the_sum_is_rounded_once(M, N, K, bn, split):
    from diloco_swarm_b200.ops import kernels as Kn
    from diloco_swarm_b200.ops._lib import check, cuda_lib, stream_ptr
    if split > (K + 63) // 64 or (bn >= 384 and bn < 1000 and M < 256):
        pytest.skip("the kernel does not take the shape")
    a, b = _mk((M, K), seed=1), _mk((N, K), 0.05, seed=2)
    bias = torch.randn(N, device="cuda")
    hi, lo = _mk((M, N), 4.0, seed=3), _mk((M, N), 0.01, seed=4)
    prod = a.double() @ b.double().t()
    want = prod + bias.double() + hi.double() + lo.double()
    for with_in in (True, False):
        out = torch.full((M + 8, N + 8), 7.0, dtype=torch.bfloat16, device="cuda")
        low = out.clone()
        ldo = N + 8
        check(cuda_lib().dsw_gemm_bf16(a.data_ptr(), K, 0, b.data_ptr(), K, 0, M, N, K, Kn.EPI_RESID, split, out.data_ptr(), ldo,
                                       bias.data_ptr(), hi.data_ptr(), N, low.data_ptr(), None, ldo, bn, 0, None, stream_ptr())
              if not with_in else
              cuda_lib().dsw_gemm_bf16(a.data_ptr(), K, 0, b.data_ptr(), K, 0, M, N, K, Kn.EPI_RESID, split, out.data_ptr(), ldo,
                                       bias.data_ptr(), hi.data_ptr(), N, low.data_ptr(), _padded(lo, ldo).data_ptr(), ldo, bn, 0,
                                       None, stream_ptr()), "dsw_gemm_bf16")
        torch.cuda.synchronize()
        assert bool((out[M:] == 7).all()) and bool((out[:, N:] == 7).all()) and bool((low[M:] == 7).all()) and bool((low[:, N:] == 7).all())
        o, l = out[:M, :N], low[:M, :N]
        ref = want if with_in else want - lo.double()
        # out is the sum to half a unit of bf16 (2^-9), what is left of it goes to bf16 once more (2^-18 of the sum); the
        # accumulator takes K / 16 additions of fp32, each off by at most 2^-23 of the running sum, which the sum of the
        # products' magnitudes bounds, and four more fp32 operations follow
        mag = a.double().abs() @ b.double().abs().t() + bias.double().abs() + hi.double().abs()
        bound = 2.0 ** -17 * ref.abs() + (K / 16 + 4) * 2.0 ** -23 * mag
        assert bool(((o.double() + l.double() - ref).abs() <= bound).all())
        assert bool(((o.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + bound).all())


def _padded(t, ld):
    global _kept                                         # alive until the launch has run
    _kept = torch.zeros(t.shape[0], ld, dtype=t.dtype, device=t.device)
    _kept[:, :t.shape[1]] = t
    return _kept
