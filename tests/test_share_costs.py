"""Which of the ways to share a forward's tiles out the tensor-core GEMM takes, at sizes where one of them was measured to be shorter
than the others by more than runs differ (microseconds of the whole call on a B200, back to back)."""
import ctypes

import pytest

from unifur_b200 import _lib

SIZES = [
    # rows, d_in, d_out: activation rows of a tile, pairs to a tile (at least, at most)
    (146, 2176, 1024, 256, 4, 16),    # 14.8 to 15.4; whole tiles of 128 16.4
    (62, 1792, 640, 128, 2, 8),       # in the other orientation 14.9; a pair to a tile 16.3
    (117, 7680, 704, 128, 4, 16),     # 16.6 to 17.4; every pair 24 stages, one collecting, 24.2
    (74, 11200, 320, 128, 8, 24),     # 14.5 to 15.0; likewise 19.5
    (52, 6848, 1280, 128, 4, 12),     # 12.6 to 13.2; likewise 17.4
    (1155, 5888, 2560, 256, 1, 1),    # 43.2; divided by stages 49.6
    (172, 4864, 11520, 256, 1, 1),    # 46.5; divided by stages 51.7
    (31, 2816, 13824, 128, 1, 1),     # 16.9; divided by stages 22.0
    (512, 4096, 4096, 128, 1, 1),
    (203, 3584, 18944, 256, 1, 1),    # 74 tiles: a pair each
]


@pytest.mark.parametrize("rows,d_in,d_out,height,least,most", SIZES)
def test_the_shorter_way(rows, d_in, d_out, height, least, most):
    L = _lib.load()
    ctas, tile_rows = ctypes.c_uint32(0), ctypes.c_uint32(0)
    seg = (ctypes.c_uint32 * 300)()
    assert L.nf4_prefill_forward_plan(rows, d_in, d_out, 0, ctypes.byref(tile_rows), ctypes.byref(ctas), seg, 100) >= 0
    assert tile_rows.value == height
    tiles = ((rows + height - 1) // height) * ((d_out + 255) // 256)
    assert least * tiles <= ctas.value // 2 <= most * tiles
