"""Shapes whose projections split a tile's K range over a cluster, with the plan each of them reaches."""
import ctypes as C

from effective_transformer_b200 import _capi


def route(dtype, rows, n, k, epi):
    """(tile width, CTAs per tile; 0 = the persistent kernels)"""
    tile_n, splits = C.c_int(0), C.c_int(0)
    code = _capi.load().et_gemm_route(_capi.ET_FP16 if dtype == "fp16" else _capi.ET_FP32, rows, n, k, epi,
                                      C.byref(tile_n), C.byref(splits))
    assert code == _capi.ET_OK
    return tile_n.value, splits.value


# dtype, valid rows, capacity, N, K, epilogue, (tile width, CTAs per tile).  Valid rows on the edges of a row tile, of
# a warp's 32 rows and of the rows dealt to a CTA; row tiles the batch leaves empty.
SPLIT_ROUTES = [
    ("fp16", 128, 128, 2304, 768, 1, (64, 1)),
    ("fp16", 1, 50, 2304, 768, 1, (64, 1)),
    ("fp16", 40, 256, 3072, 768, 2, (64, 2)),
    ("fp16", 639, 640, 1024, 4096, 4, (64, 2)),
    ("fp16", 64, 64, 3072, 1024, 1, (64, 3)),
    ("fp16", 97, 128, 1536, 512, 1, (64, 3)),
    ("fp16", 128, 128, 2688, 896, 1, (64, 3)),
    ("fp16", 2, 128, 4096, 1024, 2, (64, 3)),
    ("fp16", 385, 512, 1024, 1024, 4, (64, 3)),
    ("fp16", 512, 512, 1024, 4096, 4, (64, 3)),
    ("fp16", 127, 128, 768, 768, 0, (64, 4)),
    ("fp16", 257, 384, 1024, 4096, 4, (64, 4)),
    ("fp16", 33, 128, 1024, 1024, 4, (64, 5)),
    ("fp16", 255, 256, 1024, 4096, 4, (64, 6)),
    ("fp16", 129, 256, 1024, 4096, 0, (64, 6)),
    ("fp16", 3, 64, 768, 3072, 4, (64, 8)),
    ("fp32", 385, 700, 768, 3072, 0, (64, 2)),
    ("fp32", 30, 50, 2304, 768, 1, (64, 3)),
    ("fp32", 256, 256, 1024, 4096, 0, (64, 4)),
    ("fp32", 200, 256, 768, 768, 1, (64, 5)),
    ("fp32", 100, 128, 1024, 4096, 0, (64, 6)),
    ("fp32", 127, 128, 1024, 1024, 1, (64, 6)),
    ("fp32", 3, 64, 768, 3072, 0, (64, 8)),
    ("fp32", 40, 256, 3072, 768, 2, (128, 2)),
    ("fp32", 513, 640, 1024, 1024, 0, (128, 3)),
    ("fp32", 700, 1024, 768, 3072, 0, (128, 4)),
    ("fp32", 60, 64, 3072, 1024, 1, (128, 5)),
    ("fp32", 129, 256, 768, 3072, 3, (128, 8)),
]
