"""Which GEMM kernel a projection runs is decided on the host, from the capacity in rows: checked without a GPU."""
import ctypes as C

import pytest

from effective_transformer_b200 import _capi
from routes import SPLIT_ROUTES, route


def test_every_number_of_ctas_per_tile_is_covered_by_the_gpu_tests():
    """The rule picks 8, 6, 5, 4, 3, 2 (fp16 also 1) CTAs per tile; 3, 5 and 6 do not divide a tile's 128 rows."""
    fp16 = {plan for dtype, *_, plan in SPLIT_ROUTES if dtype == "fp16"}
    fp32 = {plan for dtype, *_, plan in SPLIT_ROUTES if dtype == "fp32"}
    assert fp16 == {(64, s) for s in (1, 2, 3, 4, 5, 6, 8)}
    assert {(64, s) for s in (2, 3, 4, 5, 6, 8)} | {(128, s) for s in (2, 3, 4, 5, 8)} == fp32


@pytest.mark.parametrize("dtype,m,cap,n,k,epi,plan", SPLIT_ROUTES)
def test_routes_of_the_gpu_tests(dtype, m, cap, n, k, epi, plan):
    """The shapes of the GPU tests reach the plan they are listed with (148 SMs)."""
    assert route(dtype, cap, n, k, epi) == plan


@pytest.mark.parametrize("hidden,ffn", [(768, 3072), (1024, 4096)])
def test_large_batches_run_the_persistent_kernels(hidden, ffn):
    for n, k, epi in ((3 * hidden, hidden, 7), (hidden, hidden, 9), (ffn, hidden, 8), (hidden, ffn, 9)):
        for rows in (2305, 8000, 64000, 524288):
            assert route("fp16", rows, n, k, epi)[1] == 0
            assert route("fp32", rows, n, k, 1)[1] == 0
        # the LayerNorm inside the GEMM kernel is the persistent kernel's at any size
        for epi_ln in (5, 6):
            assert route("fp16", 64, n, k, epi_ln)[1] == 0


@pytest.mark.parametrize("hidden,splits", [(256, 0), (384, 0), (512, 3), (640, 3), (768, 1), (896, 3), (1024, 3), (1152, 3)])
def test_projection_in_front_of_the_attention_by_hidden_size(hidden, splits):
    """One row tile: the plans as they were measured on both sides of each line; more rows, the persistent kernels."""
    for epi in (1, 7):
        for rows in (1, 64, 128):
            assert route("fp16", rows, 3 * hidden, hidden, epi)[1] == splits
        assert route("fp16", 129, 3 * hidden, hidden, epi)[1] == 0


def test_invalid_shapes_are_refused():
    lib, a, b = _capi.load(), C.c_int(), C.c_int()
    for dtype, rows, n, k, epi in ((7, 8, 128, 64, 0), (0, 0, 128, 64, 0), (0, 8, 100, 64, 0), (0, 8, 128, 0, 0),
                                   (0, 8, 128, 64, 10), (0, 8, 128, 64, -1)):
        assert lib.et_gemm_route(dtype, rows, n, k, epi, C.byref(a), C.byref(b)) == _capi.ET_INVALID_ARGUMENT
    assert lib.et_gemm_route(0, 8, 128, 64, 0, None, C.byref(b)) == _capi.ET_INVALID_ARGUMENT
