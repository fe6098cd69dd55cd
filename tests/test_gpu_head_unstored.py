"""LM head and cross-entropy without stored logits: partial log-sum-exps, row records and the logits' gradient."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(M, V, K, masked, scale, seed):
    from diloco_swarm_b200.ops._lib import Status, check, cuda_lib, ptr, stream_ptr
    lib, status = cuda_lib(), Status(torch.device("cuda", 0))
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(V, K, device="cuda", generator=g) * 3 / K ** 0.5).to(torch.bfloat16)
    tg = torch.randint(0, V, (M,), device="cuda", generator=g)
    edges = torch.tensor([0, V - 1, min(31, V - 1), min(32, V - 1), min(63, V - 1), min(64, V - 1), min(255, V - 1),
                          min(256, V - 1)], device="cuda")
    tg[:8] = edges[:min(8, M)]
    mask = (torch.rand(M, device="cuda", generator=g) < 0.7).long() if masked else None
    if masked:
        mask[0] = 1
        tg[mask == 0] = -100                      # never looked at
    parts = torch.empty((V + 63) // 64, M, device="cuda")
    tlogit = torch.empty(M, device="cuda")
    rows = torch.empty(M, 4, device="cuda")
    loss = torch.zeros((), device="cuda")
    count = torch.tensor([float(mask.sum()) if masked else float(M)], device="cuda")
    dl = torch.full((M, V), 7.0, dtype=torch.bfloat16, device="cuda")
    check(lib.dsw_head_lse(ptr(x), ptr(w), ptr(tg), ptr(parts), ptr(tlogit), M, V, K, status.ptr, stream_ptr()), "lse")
    check(lib.dsw_head_rows(ptr(parts), ptr(tlogit), ptr(tg), ptr(mask), ptr(count), scale, ptr(loss), ptr(rows), M, V,
                            status.ptr, stream_ptr()), "rows")
    check(lib.dsw_head_dlogits(ptr(x), ptr(w), ptr(rows), ptr(dl), M, V, K, status.ptr, stream_ptr()), "dlogits")
    torch.cuda.synchronize()
    status.raise_if_set()
    return x, w, tg, mask, loss, dl


@pytest.mark.parametrize("M,V,K", [(8, 136, 64), (130, 264, 128), (255, 512, 128), (257, 1000, 72), (300, 50304, 128)])
@pytest.mark.parametrize("masked", [False, True])
def test_loss_and_gradient_against_fp32(M, V, K, masked):
    scale = 0.5
    x, w, tg, mask, loss, dl = _run(M, V, K, masked, scale, 11)
    logits = (x.double() @ w.double().t()).requires_grad_()
    keep = mask.bool() if masked else torch.ones(M, dtype=torch.bool, device="cuda")
    want = torch.nn.functional.cross_entropy(logits[keep], tg[keep]) * scale
    want.backward()
    # fp32 sums over V columns in base 2: a few 1e-6 of a loss of the order of ten
    assert abs(loss.item() - want.item()) <= 1e-5 * max(1.0, abs(want.item()))
    # the gradient is rounded to bf16 once (2^-9), its fp32 value is good to some 1e-5 (exponent of the order of 20)
    assert torch.allclose(dl.double(), logits.grad, rtol=2 ** -8, atol=1e-7 * scale / keep.sum().item())
    if masked:
        assert torch.all(dl[~keep] == 0)


def test_masked_rows_stay_zero_and_kept_rows_report_bad_targets():
    """A logit that overflows in a masked row reaches neither loss nor gradient; a target outside the vocabulary in a
    kept row sets the status word."""
    from diloco_swarm_b200.ops._lib import Status, check, cuda_lib, ptr, stream_ptr
    lib, status = cuda_lib(), Status(torch.device("cuda", 0))
    M, V, K = 40, 264, 64
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    x[3] = float("inf")
    w = torch.randn(V, K, device="cuda").to(torch.bfloat16)
    mask = torch.ones(M, dtype=torch.long, device="cuda")
    mask[3] = 0
    parts, tlogit = torch.empty((V + 63) // 64, M, device="cuda"), torch.empty(M, device="cuda")
    rows, loss = torch.empty(M, 4, device="cuda"), torch.zeros((), device="cuda")
    count, dl = torch.tensor([M - 1.0], device="cuda"), torch.empty(M, V, dtype=torch.bfloat16, device="cuda")
    for bad in (False, True):
        tg = torch.zeros(M, dtype=torch.long, device="cuda")
        tg[5] = V if bad else V - 1
        loss.zero_()
        check(lib.dsw_head_lse(ptr(x), ptr(w), ptr(tg), ptr(parts), ptr(tlogit), M, V, K, status.ptr, stream_ptr()), "lse")
        check(lib.dsw_head_rows(ptr(parts), ptr(tlogit), ptr(tg), ptr(mask), ptr(count), 1.0, ptr(loss), ptr(rows), M, V,
                                status.ptr, stream_ptr()), "rows")
        check(lib.dsw_head_dlogits(ptr(x), ptr(w), ptr(rows), ptr(dl), M, V, K, status.ptr, stream_ptr()), "dlogits")
        torch.cuda.synchronize()
        assert torch.isfinite(loss) and torch.all(dl[3] == 0) and torch.isfinite(dl.float()).all()
        if bad:
            with pytest.raises(RuntimeError):
                status.raise_if_set()
        else:
            status.raise_if_set()
