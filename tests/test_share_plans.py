"""The tensor-core kernel's sharing of tiles between CTAs, checked on the host (no GPU): every
main k-stage of every tile is multiplied exactly once, a tile split between CTAs is split between
neighbours in ascending order with the last stages on the highest CTA, every CTA dumps at most one
unfinished piece and works on it first, and the CTAs' loads differ by less than one tile."""
import ctypes

import pytest

from unifur_b200 import _lib

SHAPES = [
    (2048, 4096, 14336),   # configuration 3: 896 tiles on 148 CTAs
    (4096, 3584, 3584), (4096, 3584, 512), (4096, 3584, 18944), (4096, 18944, 3584),   # the block's projections
    (4096, 18944, 1792), (4096, 18944, 896), (4096, 18944, 448), (4096, 3584, 64),     # and their shards
    (2048, 4096, 7168), (2048, 4096, 1792),
    (99, 20288, 512), (512, 4096, 4096), (2514, 15104, 320),   # fewer tiles than pairs: several pairs to a tile
    (600, 16384, 10240),                                       # ... divided by stages
    (512, 4096, 256), (300, 3072, 200), (768, 1536, 6400), (17, 64, 8), (40, 64, 40000), (257, 192, 136),
]


def _plan(rows, d_in, d_out):
    L = _lib.load()
    ctas = ctypes.c_uint32(0)
    cap = 4096
    seg = (ctypes.c_uint32 * (3 * cap))()
    n0 = L.nf4_prefill_share_plan(rows, d_in, d_out, 0, ctypes.byref(ctas), seg, cap)
    assert n0 >= 0 and 1 <= ctas.value <= 148
    out = []
    for c in range(ctas.value):
        n = L.nf4_prefill_share_plan(rows, d_in, d_out, c, None, seg, cap)
        assert 0 <= n <= cap
        out.append([(seg[3 * j], seg[3 * j + 1], seg[3 * j + 2]) for j in range(n)])
    return out


@pytest.mark.parametrize("rows,d_in,d_out", SHAPES)
def test_every_stage_once_and_neighbours_share(rows, d_in, d_out):
    plan = _plan(rows, d_in, d_out)
    ks = d_in // 64
    tiles = ((rows + 255) // 256) * ((d_out + 127) // 128)
    pieces = {}
    for c, segs in enumerate(plan):
        unfinished = [j for j, (_t, _b, e) in enumerate(segs) if e != ks]
        assert len(unfinished) <= 1 and (not unfinished or unfinished[0] == 0)   # dumped first, at most one
        for tile, b, e in segs:
            assert tile < tiles and 0 <= b < e <= ks
            pieces.setdefault(tile, []).append((b, e, c))
    assert sorted(pieces) == list(range(tiles))
    for tile, ps in pieces.items():
        ps.sort()
        assert ps[0][0] == 0 and ps[-1][1] == ks
        for (b0, e0, c0), (b1, e1, c1) in zip(ps, ps[1:]):
            assert e0 == b1 and c1 == c0 + 1        # contiguous stages, consecutive CTAs
    loads = [sum(e - b for _t, b, e in segs) for segs in plan]
    assert max(loads) - min(loads) <= ks             # nobody has a whole tile more than anybody else


NARROW = [  # more than 128 rows in tiles of 128
    (512, 4096, 4096), (2050, 2112, 64), (129, 1024, 9472), (200, 64, 8), (640, 3584, 3584), (224, 3584, 9472), (300, 1088, 640),
]


def _forward_plan(rows, d_in, d_out):
    L = _lib.load()
    ctas, height, cap = ctypes.c_uint32(0), ctypes.c_uint32(0), 4096
    seg = (ctypes.c_uint32 * (3 * cap))()
    assert L.nf4_prefill_forward_plan(rows, d_in, d_out, 0, ctypes.byref(height), ctypes.byref(ctas), seg, cap) >= 0
    assert 1 <= ctas.value <= 148
    out = []
    for c in range(ctas.value):
        n = L.nf4_prefill_forward_plan(rows, d_in, d_out, c, None, None, seg, cap)
        assert 0 <= n <= cap
        out.append([(seg[3 * j], seg[3 * j + 1], seg[3 * j + 2]) for j in range(n)])
    return height.value, out


@pytest.mark.parametrize("rows,d_in,d_out", SHAPES + NARROW)
def test_what_a_forward_follows(rows, d_in, d_out):
    height, plan = _forward_plan(rows, d_in, d_out)
    if (rows, d_in, d_out) in NARROW or rows <= 128:
        assert height == 128
    ks = d_in // 64
    tiles = ((rows + height - 1) // height) * ((d_out + 127) // 128)
    pieces = {}
    for c, segs in enumerate(plan):
        unfinished = [j for j, (_t, _b, e) in enumerate(segs) if e != ks]
        assert len(unfinished) <= 1 and (not unfinished or unfinished[0] == 0)
        for tile, b, e in segs:
            assert tile < tiles and 0 <= b < e <= ks
            assert ks % 2 or (b % 2 == 0 and e % 2 == 0)   # whole steps of two stages, where a tile consists of them
            pieces.setdefault(tile, []).append((b, e, c))
    assert sorted(pieces) == list(range(tiles))
    for ps in pieces.values():
        ps.sort()
        assert ps[0][0] == 0 and ps[-1][1] == ks
        for (_b0, e0, c0), (b1, _e1, c1) in zip(ps, ps[1:]):
            assert e0 == b1 and c1 == c0 + 1
    if rows > 128 and height == 128:
        assert all(len(segs) <= 1 and (not segs or segs[0][1:] == (0, ks)) for segs in plan)  # one whole tile at most


def test_rejects_what_the_kernel_does_not_take():
    L = _lib.load()
    seg = (ctypes.c_uint32 * 3)()
    assert L.nf4_prefill_share_plan(16, 4096, 4096, 0, None, seg, 1) < 0      # decode-sized
    assert L.nf4_prefill_share_plan(64, 100, 4096, 0, None, seg, 1) < 0       # d_in not a multiple of 64
    assert L.nf4_prefill_share_plan(64, 4096, 4096, 500, None, seg, 1) < 0    # no such CTA


@pytest.mark.parametrize("rows,d_in,d_out,rank", [
    (1, 4096, 11008, 16), (16, 4096, 11008, 16), (8, 3584, 3584, 16), (8, 3584, 512, 16), (8, 3584, 18944, 16),
    (8, 18944, 3584, 16), (4, 2048, 64, 0), (5, 1024, 1000, 16), (3, 512, 200, 8), (5, 32768, 48, 32),
    (16, 4096, 160, 64), (1, 8192, 384, 16), (8, 4352, 96, 8), (1, 256, 16, 0),
])
def test_decode_kernel_shares_rows_and_k_exactly(rows, d_in, d_out, rank):
    # every (row of W, k) belongs to exactly one CTA: the parts of K tile [0, d_in), and within a
    # part the CTAs' row ranges tile [0, d_out) in order
    L = _lib.load()
    out = (ctypes.c_uint32 * 4)()
    ctas = L.nf4_decode_share_plan(rows, d_in, d_out, rank, 0, out)
    assert 1 <= ctas <= 148
    parts = {}
    for c in range(ctas):
        assert L.nf4_decode_share_plan(rows, d_in, d_out, rank, c, out) == ctas
        k0, k1, n0, n1 = out[0], out[1], out[2], out[3]
        assert k0 < k1 <= d_in and k1 - k0 <= 4096 and n0 <= n1 <= d_out
        parts.setdefault((k0, k1), []).append((n0, n1))
    ks = sorted(parts)
    assert ks[0][0] == 0 and ks[-1][1] == d_in and all(a[1] == b[0] for a, b in zip(ks, ks[1:]))
    for ranges in parts.values():
        assert ranges[0][0] == 0 and ranges[-1][1] == d_out
        assert all(a[1] == b[0] for a, b in zip(ranges, ranges[1:]))
    assert L.nf4_decode_share_plan(17, 4096, 64, 0, 0, out) < 0 and L.nf4_decode_share_plan(4, 100, 64, 0, 0, out) < 0


def _clusters(tiles, length, unit, room):
    return _lib.load().nf4_cluster_share_plan(tiles, length, unit, (ctypes.c_uint32 * 5)(*room))


ROOM = (296, 148, 71, 33, 14)


@pytest.mark.parametrize("tiles,length,unit,want", [
    (1, 64, 64, 1), (1, 65, 64, 2), (4, 4096, 64, 16), (14, 4096, 64, 16), (15, 4096, 64, 8), (33, 4096, 64, 8),
    (34, 4096, 64, 4), (71, 4096, 64, 4), (72, 4096, 64, 2), (148, 4096, 64, 2), (149, 4096, 64, 1),
    (1, 1024, 64, 16), (1, 512, 64, 8), (8, 2048, 256, 8), (8, 2049, 256, 16), (112, 2048, 256, 2),
])
def test_clusters_fill_the_device_once(tiles, length, unit, want):
    assert _clusters(tiles, length, unit, ROOM) == want


def test_clusters_where_large_ones_have_no_place():
    # what a device cannot place is not launched: the next smaller size is, down to a CTA by itself
    assert [_clusters(4, 4096, 64, ROOM[:i] + (0,) * (5 - i)) for i in (5, 4, 3, 2, 1, 0)] == [16, 8, 4, 2, 1, 1]
    assert _clusters(4, 4096, 64, (18, 9, 4, 2, 1)) == 4   # a slice of a device
    assert _lib.load().nf4_cluster_share_plan(1, 1, 0, (ctypes.c_uint32 * 5)(*ROOM)) == -1
