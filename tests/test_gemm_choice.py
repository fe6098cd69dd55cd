"""Which GEMM kernel a call takes, against times measured on a B200.  Host arithmetic, no GPU."""
import ctypes

import pytest

from diloco_swarm_b200.ops._lib import cuda_lib

STORE, GELU, RESID, MUL = range(4)

# (rows, columns, K, epilogue, B stored [K, N], GELU with its derivative): us of the kernels in question, weights cold in
# L2, one graph of launches ("kernel / split of K").  Widths on both sides of the 768 columns that the rule was fitted to.
FEW_ROWS = [
    ((120, 768, 3072, RESID, 0, 0), {"1064/8": 7.93, "1032/4": 7.79, "128/1": 17.2}),
    ((24, 3072, 1024, STORE, 0, 0), {"1064/2": 8.07, "1032/1": 9.47}),
    ((24, 4096, 1024, GELU, 0, 0), {"1064/2": 9.54, "1032/1": 10.75}),
    ((24, 4096, 1024, GELU, 0, 1), {"1064/2": 9.62, "1032/1": 10.79}),
    ((64, 3840, 1280, STORE, 0, 0), {"1064/2": 8.66, "1032/1": 9.17}),
    ((128, 3840, 1280, STORE, 0, 0), {"1064/2": 8.76, "1032/1": 9.33}),
    ((512, 1280, 1280, STORE, 1, 0), {"1128/2": 9.09, "128/1": 9.84}),
    ((768, 1280, 1280, STORE, 1, 0), {"1128/2": 9.71, "128/1": 10.32}),
    ((64, 4800, 1600, STORE, 0, 0), {"1128/2": 11.04, "128/1": 11.53}),
    ((128, 4800, 1600, STORE, 0, 0), {"1128/2": 11.24, "128/1": 11.89}),
    ((512, 3072, 768, GELU, 0, 1), {"128/1": 10.7, "1128/1": 11.65, "384/1": 10.69}),
    ((256, 3072, 768, MUL, 1, 0), {"128/1": 9.12, "1064/1": 9.49, "384/1": 8.95}),
    ((384, 4096, 1024, GELU, 0, 1), {"128/1": 11.84, "1128/1": 12.97, "384/1": 11.59}),
    ((256, 6400, 1600, GELU, 0, 1), {"384/1": 13.93, "1128/1": 15.73}),
]
# GELU without its derivative (evaluation): "kernel / split of K" as before
GELU_ONLY = [
    ((1024, 3072, 768, GELU, 0, 0), {"384/1": 12.16, "512/1": 13.21}),
    ((1536, 3072, 768, GELU, 0, 0), {"384/1": 12.6, "512/1": 13.57}),
    ((2560, 3072, 768, GELU, 0, 0), {"256/1": 18.62, "512/1": 20.65}),
    ((3072, 3072, 768, GELU, 0, 0), {"256/1": 18.88, "512/1": 20.67}),
    ((8192, 3072, 768, GELU, 0, 0), {"256/1": 40.57, "512/1": 39.55}),
    ((32768, 3072, 768, GELU, 0, 0), {"256/1": 139.9, "512/1": 132.2}),
    ((768, 4096, 1024, GELU, 0, 0), {"384/1": 13.69, "512/1": 14.59}),
    ((1024, 5120, 1280, GELU, 0, 0), {"384/1": 19.87, "512/1": 22.37}),
    ((1024, 6400, 1600, GELU, 0, 0), {"384/1": 23.95, "512/1": 26.62}),
]


def _choice(call):
    split = ctypes.c_int(0)
    bn = cuda_lib().dsw_gemm_choice(*call, 148, ctypes.byref(split))
    assert bn > 0
    return f"{bn}/{split.value}"


@pytest.mark.parametrize("call,us", FEW_ROWS)
def test_few_rows_take_a_kernel_that_is_near_the_best(call, us):
    got = _choice(call)
    assert got in us and us[got] <= 1.035 * min(us.values()), (got, us)


@pytest.mark.parametrize("call,us", GELU_ONLY)
def test_gelu_without_derivative_takes_a_tile_that_is_near_the_best(call, us):
    got = _choice(call)
    assert got in us and us[got] <= 1.02 * min(us.values()), (got, us)


def test_the_split_of_a_call_is_that_of_its_recorded_outputs():
    """Partial sums are added in the order of the split, so another split is another rounding of the same logits."""
    for n, k, want in [(2304, 768, "1032/2"), (768, 768, "1032/4"), (3072, 768, "1032/1"), (768, 3072, "1064/8")]:
        assert _choice((120, n, k, RESID if n == 768 else STORE, 0, 0)) == want
