"""LayerNorm backward in two calls, the rows on one stream and the column sums on another, is the one call."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _noalloc():
    import ctypes
    from diloco_swarm_b200.ops._lib import cuda_lib
    call = cuda_lib().dsw_layernorm_bwd_noalloc
    call.restype, call.argtypes = ctypes.c_int, [ctypes.c_void_p] * 10 + [ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
    return call


@pytest.mark.parametrize("M,d", [(5, 128), (700, 128), (5, 776), (3001, 768)])
@pytest.mark.parametrize("dres", [False, True])
def test_two_calls_are_one(M, d, dres):
    from diloco_swarm_b200.ops import kernels as K
    from diloco_swarm_b200.ops._lib import cuda_lib, ptr
    lib, g = cuda_lib(), torch.Generator(device="cuda").manual_seed(d)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, dy, r, w = rnd(M, d).bfloat16(), rnd(M, d).bfloat16(), rnd(M, d).bfloat16() if dres else None, rnd(d)
    _, mean, rstd = K.layernorm_fwd(x, w, rnd(d))
    sums = [[torch.ones(d, device="cuda") for _ in range(3)] for _ in range(2)]
    res = [s[2] if dres else None for s in sums]
    one = K.layernorm_bwd(dy, x, w, mean, rstd, sums[0][0], sums[0][1], dres=r, dres_sum=res[0])
    two = torch.empty_like(x)
    scratch = torch.full((lib.dsw_layernorm_bwd_blocks(M) * 3 * d,), float("nan"), device="cuda")
    main, side = torch.cuda.current_stream(), torch.cuda.Stream()
    assert lib.dsw_layernorm_bwd(dy.data_ptr(), x.data_ptr(), w.data_ptr(), mean.data_ptr(), rstd.data_ptr(), ptr(r), two.data_ptr(),
                                 None, None, None, scratch.data_ptr(), M, d, main.cuda_stream) == 0
    side.wait_stream(main)
    assert lib.dsw_layernorm_bwd(None, None, None, None, None, None, None, sums[1][0].data_ptr(), sums[1][1].data_ptr(), ptr(res[1]),
                                 scratch.data_ptr(), M, d, side.cuda_stream) == 0
    main.wait_stream(side)
    assert torch.equal(one, two)
    for a, b in zip(*sums):
        assert torch.equal(a, b) and torch.isfinite(b).all()
    # neither part asked for
    assert lib.dsw_layernorm_bwd(dy.data_ptr(), x.data_ptr(), w.data_ptr(), mean.data_ptr(), rstd.data_ptr(), None, None, None, None,
                                 None, scratch.data_ptr(), M, d, main.cuda_stream) == -10


@pytest.mark.parametrize("M,d", [(37, 128), (700, 768)])
@pytest.mark.parametrize("asked", [(0,), (1,), (2,), (1, 2), (0, 2), ()])
def test_each_sum_is_optional(M, d, asked):
    """dgamma, dbeta and the sum of dres come one without the others; without any, dx alone does."""
    from diloco_swarm_b200.ops import kernels as K
    from diloco_swarm_b200.ops._lib import cuda_lib, ptr
    lib, g = cuda_lib(), torch.Generator(device="cuda").manual_seed(M)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, dy, r, w = rnd(M, d).bfloat16(), rnd(M, d).bfloat16(), rnd(M, d).bfloat16(), rnd(d)
    _, mean, rstd = K.layernorm_fwd(x, w, rnd(d))
    whole = [torch.ones(d, device="cuda") for _ in range(3)]
    want = K.layernorm_bwd(dy, x, w, mean, rstd, whole[0], whole[1], dres=r, dres_sum=whole[2])
    scratch = torch.empty(lib.dsw_layernorm_bwd_blocks(M) * 3 * d, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    for noalloc in (False, True):
        got, dx = [torch.ones(d, device="cuda") if i in asked else None for i in range(3)], torch.empty_like(x)
        front = [dy.data_ptr(), x.data_ptr(), w.data_ptr(), mean.data_ptr(), rstd.data_ptr(), r.data_ptr(), dx.data_ptr()]
        front += [ptr(t) for t in got]
        if noalloc:
            assert _noalloc()(*front, M, d, st) == 0
        else:
            assert lib.dsw_layernorm_bwd(*front, scratch.data_ptr(), M, d, st) == 0
        assert torch.equal(dx, want)
        for i in asked:
            assert torch.equal(got[i], whole[i]), i


def test_the_shared_scratch_is_not_asked_for_sums_alone():
    d = 128
    sums = torch.ones(3, d, device="cuda")
    rc = _noalloc()(None, None, None, None, None, None, None, sums[0].data_ptr(), sums[1].data_ptr(), sums[2].data_ptr(), 8, d,
                    torch.cuda.current_stream().cuda_stream)
    assert rc == -20
    torch.cuda.synchronize()
    assert bool((sums == 1).all())
