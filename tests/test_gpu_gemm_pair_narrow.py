"""The 256 x 128 CTA-pair tile and the library's own choice of tile and split against a plain fp32 matmul."""
import pytest
import torch

from test_gpu_gemm import _close, _mk

pytestmark = pytest.mark.gpu

# one pair with missing rows; remainders of every kind; more tiles than pairs; one narrow column block
SHAPES = [(129, 136, 72), (256, 128, 64), (520, 264, 200), (4104, 776, 264), (2048, 128, 4096)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("bn", [384, 0])
def test_layouts_and_epilogues(M, N, K, bn):
    from diloco_swarm_b200.ops import kernels as Kn
    from diloco_swarm_b200.ops._lib import Status
    st = Status(torch.device("cuda"))
    a, b = _mk((M, K), seed=1), _mk((N, K), 0.05, seed=2)
    bias, res = torch.randn(N, device="cuda"), _mk((M, N), seed=3)
    acc = a.float() @ b.float().t()
    kw = dict(bn=bn, status=st)
    _close(Kn.gemm(a, b, bias=bias, **kw), acc + bias, "bias")
    _close(Kn.gemm(a, b, mode=Kn.EPI_RESID, bias=bias, resid=res, **kw), acc + bias + res.float(), "residual")
    _close(Kn.gemm(a, b.t().contiguous(), b_t=False, mode=Kn.EPI_MUL, aux_in=res, **kw), acc * res.float(), "multiply")
    if M % 8 == 0:
        base = torch.randn(M, N, device="cuda")
        for split in (1, 2, 0):
            out = base.clone()
            Kn.gemm(a.t().contiguous(), b.t().contiguous(), a_t=True, b_t=False, mode=Kn.EPI_ATOMIC_F32, out=out,
                    split_k=split, **kw)
            _close(out, base + acc, f"weight gradient, split {split}")
    torch.cuda.synchronize()
    st.raise_if_set()


def test_residual_with_a_low_half():
    """out + aux_out is the sum to fp32 precision where the accumulator is exact; every kernel takes the operand."""
    from diloco_swarm_b200.ops import kernels as Kn
    M, N, K = 300, 256, 128
    a = torch.zeros(M, K, dtype=torch.bfloat16, device="cuda")
    a[:, 0] = 1.0
    b = _mk((N, K), seed=4)                              # the product is b[:, 0]: exact in bf16
    hi, lo = _mk((M, N), 8.0, seed=5), _mk((M, N), 0.02, seed=6)
    want = b[:, 0].float() + hi.float() + lo.float()
    for bn, split in ((128, 1), (256, 1), (384, 1), (512, 1), (1064, 2)):
        low = torch.empty_like(lo)
        from diloco_swarm_b200.ops._lib import check, cuda_lib, stream_ptr
        out = torch.empty_like(hi)
        check(cuda_lib().dsw_gemm_bf16(a.data_ptr(), K, 0, b.data_ptr(), K, 0, M, N, K, Kn.EPI_RESID, split, out.data_ptr(), N,
                                       None, hi.data_ptr(), N, low.data_ptr(), lo.data_ptr(), N, bn, 0, None, stream_ptr()),
              "dsw_gemm_bf16")
        # the remainder of a bf16 rounding fits bf16 to 2^-9 of itself: 2^-18 of the sum, and fp32 roundings of the sum
        assert (out.float() + low.float() - want).abs().max() < 2 ** -16 * want.abs().max()
