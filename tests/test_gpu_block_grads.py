"""Side work of a block with few tokens in two launches (csrc/block_grads.cu, block_sums_kernel)."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _array(kind, values):
    return (kind * len(values))(*values)


# one token, remainders of 16 tokens, the most; outputs of a remainder of a 64-wide tile on either side
@pytest.mark.parametrize("M", [1, 15, 16, 17, 100, 128, 255, 256])
@pytest.mark.parametrize("shapes", [[(128, 512), (512, 128), (128, 128), (384, 128)], [(72, 8), (8, 200)], [(1600, 264)]])
def test_weight_gradients(M, shapes):
    from diloco_swarm_b200.ops._lib import check, cuda_lib, stream_ptr
    g = torch.Generator(device="cuda").manual_seed(M)
    dy = [torch.randn(M, o, device="cuda", generator=g).to(torch.bfloat16) for o, _ in shapes]
    x = [torch.randn(M, i, device="cuda", generator=g).to(torch.bfloat16) for _, i in shapes]
    dw = [torch.ones(o, i, device="cuda") for o, i in shapes]
    lib = cuda_lib()
    ptrs = lambda ts: ctypes.cast(_array(ctypes.c_void_p, [t.data_ptr() for t in ts]), ctypes.c_void_p)
    ints = lambda vs: ctypes.cast(_array(ctypes.c_int, vs), ctypes.c_void_p)
    args = [ptrs(dy), ptrs(x), ptrs(dw), ints([o for o, _ in shapes]), ints([i for _, i in shapes])]
    check(lib.dsw_block_wgrads(*args, len(shapes), M, stream_ptr()), "wgrads")
    torch.cuda.synchronize()
    for a, b, w in zip(dy, x, dw):
        want = a.double().t() @ b.double()
        # fp32 sums of M exact products, added to ones
        assert (w.double() - 1.0 - want).abs().max() <= 2 ** -22 * (M + 1) * 16, (w - 1 - want).abs().max()


@pytest.mark.parametrize("M,d", [(1, 128), (24, 64), (128, 128), (255, 128), (17, 256), (100, 768), (255, 768), (255, 1600), (200, 2048)])
def test_sums_are_those_of_the_single_calls(M, d):
    from diloco_swarm_b200.ops._lib import check, cuda_lib, ptr, stream_ptr
    lib, st = cuda_lib(), stream_ptr()
    g = torch.Generator(device="cuda").manual_seed(M + d)
    a, b = (torch.randn(M, n * d, device="cuda", generator=g).to(torch.bfloat16) for n in (4, 3))
    ln = [torch.randn(lib.dsw_layernorm_bwd_scratch(M, d), device="cuda", generator=g) for _ in range(2)]
    outs = []
    for one in (False, True):
        o = [torch.ones(n * d, device="cuda") for n in (4, 3, 1, 1, 1, 1, 1, 1)]
        p = [ptr(t) for t in o]
        if one:
            check(lib.dsw_block_sums(ptr(a), 4 * d, p[0], ptr(b), 3 * d, p[1], ptr(ln[0]), *p[2:5], ptr(ln[1]), *p[5:8], M, d, st), "sums")
        else:
            check(lib.dsw_colsum_accum(ptr(a), 4 * d, p[0], M, 4 * d, st), "a")
            check(lib.dsw_colsum_accum(ptr(b), 3 * d, p[1], M, 3 * d, st), "b")
            for i in range(2):
                check(lib.dsw_layernorm_bwd(*[None] * 7, *p[2 + 3 * i:5 + 3 * i], ptr(ln[i]), M, d, st), "ln")
        outs.append(o)
    torch.cuda.synchronize()
    assert all(torch.equal(s, t) for s, t in zip(*outs))
