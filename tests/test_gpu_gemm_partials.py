"""Products split along K into stored partial sums: against fp64, and the same bits in every run."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(8, 64, 64), (130, 136, 1000), (256, 128, 4096), (300, 768, 50304), (2000, 1600, 2048)])
def test_sum_of_partials(M, N, K):
    from diloco_swarm_b200.ops._lib import Status, check, cuda_lib, ptr, stream_ptr
    lib, status = cuda_lib(), Status(torch.device("cuda", 0))
    g = torch.Generator(device="cuda").manual_seed(5)
    a = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    b = (torch.randn(K, N, device="cuda", generator=g) / K ** 0.5).to(torch.bfloat16)
    most, seen = 8, []
    for _ in range(3):
        parts = torch.full((most, M, N), float("nan"), device="cuda")
        out, n = torch.empty(M, N, dtype=torch.bfloat16, device="cuda"), ctypes.c_int()
        check(lib.dsw_gemm_partials(ptr(a), ptr(b), M, N, K, ptr(parts), most, ctypes.byref(n), status.ptr, stream_ptr()), "partials")
        assert 1 <= n.value <= most
        check(lib.dsw_sum_partials_bf16(ptr(parts), n.value, ptr(out), M * N, stream_ptr()), "sum")
        seen.append(out)
    torch.cuda.synchronize()
    status.raise_if_set()
    ref = a.double() @ b.double()
    # one rounding to bf16; before it K / 16 accumulations of sums of the order of one, each cut to 24 bits
    assert torch.allclose(seen[0].double(), ref, rtol=2 ** -8, atol=1e-6 + K / 16 * 2 ** -23)
    assert torch.equal(seen[0], seen[1]) and torch.equal(seen[0], seen[2])
