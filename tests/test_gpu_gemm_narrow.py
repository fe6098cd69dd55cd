"""GEMM of few rows and a short K on mma.sync (csrc/gemm_narrow.cuh), alone and with the LayerNorm ahead of it: the bits of the
cluster kernel and of the LayerNorm kernel."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
SMS = 148


def _choice(M, N, K, mode, b_mn, derivative):
    from diloco_swarm_b200.ops._lib import cuda_lib
    split = ctypes.c_int(0)
    return cuda_lib().dsw_gemm_choice(M, N, K, mode, b_mn, derivative, SMS, ctypes.byref(split)), split.value


# one row, remainders of 32 rows and columns, whole tiles; K of one k-block, several, split; both weight layouts
@pytest.mark.parametrize("M,N,K", [(1, 128, 128), (24, 384, 128), (31, 40, 64), (33, 136, 192), (120, 512, 128), (128, 128, 512), (100, 128, 384),
                                   (256, 520, 128), (65, 264, 256), (40, 768, 768), (20, 72, 1024)])
@pytest.mark.parametrize("b_t", [True, False])
def test_bits_of_the_cluster_kernel(M, N, K, b_t):
    from diloco_swarm_b200.ops import kernels as k
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    rnd = lambda *s, std=1.0: (torch.randn(*s, device="cuda", generator=g) * std).to(torch.bfloat16)
    a, w, resid, low, aux = rnd(M, K), rnd(N, K, std=0.05) if b_t else rnd(K, N, std=0.05), rnd(M, N), rnd(M, N, std=2 ** -9), rnd(M, N)
    bias = torch.randn(N, device="cuda", generator=g)
    empty = lambda: torch.full((M, N), 9.0, device="cuda", dtype=torch.bfloat16)
    taken = 0
    for mode, kw, keeps in ((k.EPI_STORE, dict(bias=bias), False), (k.EPI_STORE, {}, False), (k.EPI_GELU, dict(bias=bias), False),
                            (k.EPI_GELU, dict(bias=bias), True), (k.EPI_RESID, dict(bias=bias, resid=resid), False),
                            (k.EPI_RESID, dict(bias=bias, resid=resid, aux_in=low), True), (k.EPI_MUL, dict(aux_in=aux), False)):
        bn, split = _choice(M, N, K, mode, int(not b_t), int(mode == k.EPI_GELU and keeps))
        if bn < 1000:
            continue
        taken += 1
        got, want, got_aux, want_aux = empty(), empty(), empty(), empty()
        k.gemm(a, w, b_t=b_t, mode=mode, out=got, aux_out=got_aux if keeps else None, **kw)
        k.gemm(a, w, b_t=b_t, mode=mode, out=want, aux_out=want_aux if keeps else None, bn=bn, split_k=split, **kw)
        assert torch.equal(got, want) and torch.equal(got_aux, want_aux), (mode, bn, split)
        if mode == k.EPI_STORE:
            exact = a.double() @ (w.double().t() if b_t else w.double()) + (bias.double() if kw else 0.0)
            # rounded to bf16 once
            assert (got.double() - exact).norm() <= 2 ** -8 * exact.norm()
    assert taken >= 3, (M, N, K)


@pytest.mark.parametrize("M", [1, 24, 33, 128, 500])
@pytest.mark.parametrize("K,N,gelu", [(128, 384, False), (128, 512, True), (64, 72, False), (128, 8, True)])
@pytest.mark.parametrize("low,keep", [(False, True), (True, False)])
def test_layernorm_ahead(M, K, N, gelu, low, keep):
    from diloco_swarm_b200.ops import kernels as k
    from diloco_swarm_b200.ops._lib import Status, check, cuda_lib, ptr, stream_ptr
    lib, status = cuda_lib(), Status(torch.device("cuda", 0))
    mode = k.EPI_GELU if gelu else k.EPI_STORE
    if not lib.dsw_layernorm_gemm_fits(M, N, K, mode, int(gelu and keep), SMS):
        assert M > 128
        pytest.skip("two launches")
    g = torch.Generator(device="cuda").manual_seed(M)
    x = (torch.randn(M, K, device="cuda", generator=g) * 3 + 1).to(torch.bfloat16)
    lo = (torch.randn(M, K, device="cuda", generator=g) * 2 ** -8).to(torch.bfloat16) if low else None
    gamma, beta, bias = (torch.randn(n, device="cuda", generator=g) for n in (K, K, N))
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.1).to(torch.bfloat16)
    bf = lambda *s: torch.full(s, 9.0, device="cuda", dtype=torch.bfloat16)
    f32 = lambda *s: torch.full(s, 9.0, device="cuda")
    y, mu, rs, out, aux = bf(M, K), f32(M), f32(M), bf(M, N), bf(M, N)
    check(lib.dsw_layernorm_fwd_lo(ptr(x), ptr(lo), ptr(gamma), ptr(beta), ptr(y), ptr(mu), ptr(rs), M, K, 1e-5, stream_ptr()), "ln")
    bn, split = _choice(M, N, K, mode, 0, int(gelu and keep))
    k.gemm(y, w, mode=mode, bias=bias, out=out, aux_out=aux if gelu and keep else None, bn=bn, split_k=split)
    y2, mu2, rs2, out2, aux2 = bf(M, K), f32(M), f32(M), bf(M, N), bf(M, N)
    check(lib.dsw_layernorm_gemm(ptr(x), ptr(lo), ptr(gamma), ptr(beta), ptr(y2) if keep else None, ptr(mu2) if keep else None,
                                 ptr(rs2) if keep else None, 1e-5, ptr(w), ptr(bias), ptr(out2), mode, ptr(aux2) if gelu and keep else None,
                                 M, N, K, status.ptr, stream_ptr()), "ln gemm")
    torch.cuda.synchronize()
    status.raise_if_set()
    assert torch.equal(out, out2) and torch.equal(aux, aux2)
    if keep:
        assert torch.equal(y, y2) and torch.equal(mu, mu2) and torch.equal(rs, rs2)


def test_an_unaligned_bias_is_accepted():
    """Four bytes of alignment are enough for the cluster kernel, which such calls keep."""
    from diloco_swarm_b200.ops import kernels as k
    a, w = (torch.randn(n, 128, device="cuda").to(torch.bfloat16) for n in (24, 384))
    room = torch.randn(385, device="cuda")
    bias = room[1:]
    assert bias.data_ptr() % 16
    assert torch.equal(k.gemm(a, w, bias=bias), k.gemm(a, w, bias=bias.clone()))
