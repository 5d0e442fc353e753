"""Generates nf4_tables.inc: the NF4 level table and the fifteen exact decision
thresholds used by the CUDA quantize kernel.

The reference picks a code by scanning the sixteen levels for the smallest
f32 distance |v - L_i| with a strict '<' (src/quantize.rs:208-219).  Because
fl(v - L_i) is monotone in v and neighbouring levels are ~0.08 apart (far more
than an ulp), the scan's answer for a finite v is `number of i with v >= T_i`,
where T_i is the smallest f32 for which the scan prefers level i+1 over level
i.  This script finds every T_i by bisection over f32 bit patterns using a
numpy-float32 restatement of that scan, and writes them as hex float bit
patterns.  tests/test_thresholds.py re-checks the table against the C oracle.

Run:  python unifur_b200/csrc/gen_nf4_tables.py
"""
import os

import numpy as np

LEVELS_F64 = [
    -1.0, -0.6961928009986877, -0.5250730514526367, -0.39491748809814453,
    -0.28444138169288635, -0.18477343022823334, -0.09105003625154495, 0.0,
    0.07958029955625534, 0.16093020141124725, 0.24611230194568634, 0.33791524171829224,
    0.44070982933044434, 0.5626170039176941, 0.7229568362236023, 1.0,
]
LEVELS = np.array(LEVELS_F64, dtype=np.float64).astype(np.float32)


def scan_code(v: np.float32) -> int:
    best, best_dist = 0, np.float32(np.inf)
    for i in range(16):
        d = np.abs(np.float32(v - LEVELS[i]))
        if d < best_dist:
            best_dist, best = d, i
    return best


def key(f: np.float32) -> int:
    """Monotone integer key of a float (orders like the float)."""
    u = int(np.float32(f).view(np.uint32))
    return (u ^ 0xFFFFFFFF) if (u & 0x80000000) else (u | 0x80000000)


def unkey(k: int) -> np.float32:
    u = (k & 0x7FFFFFFF) if (k & 0x80000000) else (k ^ 0xFFFFFFFF)
    return np.array([u], dtype=np.uint32).view(np.float32)[0]


def threshold(i: int) -> np.float32:
    lo, hi = key(LEVELS[i]), key(LEVELS[i + 1])
    assert scan_code(unkey(lo)) == i and scan_code(unkey(hi)) == i + 1
    while hi - lo > 1:
        mid = (lo + hi) // 2
        if scan_code(unkey(mid)) >= i + 1:
            hi = mid
        else:
            lo = mid
    return unkey(hi)


CELL_MARGIN = 2  # units of 2^-21 on either side of a threshold where the exact path decides (errors add up to < 1.4)


def bf16_cut(t: np.float32) -> int:
    """The integer (units of 2^-21) that splits the quotients of two bf16 numbers as the threshold t does.

    There are few such quotients (two eight-bit significands and a power of two), so around every threshold they leave a gap, and
    the kernel's approximation (within half a unit of rounding and a quarter for the reciprocal) stays on their side of
    its middle: no value has to be looked at again."""
    m = np.arange(128, 256, dtype=np.float64)
    q = np.unique(np.concatenate([s * (m[:, None] / m[None, :]).ravel() * 2.0 ** -k for k in range(12) for s in (1, -1)] + [np.zeros(1)]))
    q = q[np.abs(q) <= 1.0]
    up = q.astype(np.float32) >= t  # the reference compares the quotient as f32
    below, above = float(q[~up].max()), float(q[up].min())
    last, first = np.floor(below * 2 ** 21 + 0.25 * abs(below) + 0.5), np.ceil(above * 2 ** 21 - 0.25 * abs(above) - 0.5)
    assert first - last >= 2
    return int((last + first + 1) // 2)


def main():
    th = [threshold(i) for i in range(15)]
    lines = [
        "// Generated by gen_nf4_tables.py -- do not edit by hand.",
        "// NF4 levels (f32 bit patterns of the published codebook, src/quantize.rs:49-66)",
        "// and the fifteen exact decision thresholds: code(v) = #{i : v >= T_i}.",
        "#define NF4_LEVEL_BITS_LIST \\",
    ]
    lines.append("  " + ", ".join("0x%08xu" % int(l.view(np.uint32)) for l in LEVELS))
    lines.append("#define NF4_THRESHOLD_BITS_LIST \\")
    lines.append("  " + ", ".join("0x%08xu" % int(np.float32(t).view(np.uint32)) for t in th))
    lines.append("// the sixteen levels rounded to f16 (round to nearest even), as bit patterns")
    lines.append("#define NF4_LEVEL_F16_BITS_LIST \\")
    lines.append("  " + ", ".join("0x%04xu" % int(np.float16(l).view(np.uint16)) for l in LEVELS))
    # 33 uniform cells of width 1/16 over [-1, 1]: a value v is rounded to n = round(64 v + 64) and
    # belongs to cell n >> 2, so cell c is [(4c - 0.5) / 64 - 1, (4c + 3.5) / 64 - 1), which holds at most
    # one threshold (they are >= 0.08 apart).  v itself enters as the bits of the f32 v * 2^21 + 1.5 * 2^23,
    # which are 0x4b400000 + round(v * 2^21); the cell's word W is such that the top four bits of bits - W
    # are the code and the low 28 bits are below 2 * MARGIN exactly when v is within MARGIN units of 2^-21 of
    # the threshold.  Padded to 64 words; the last one (a NaN's bits index it) is always "within".
    cells, cells_bf16 = [], []
    for c in range(33):
        lo, hi = (4 * c - 0.5) / 64.0 - 1.0, (4 * c + 3.5) / 64.0 - 1.0
        inside = [t for t in th if lo <= float(t) < hi]
        assert len(inside) <= 1
        base = sum(1 for t in th if float(t) < lo)
        # no threshold may sit within rounding distance of a cell edge
        for t in th:
            assert min(abs(float(t) - lo), abs(float(t) - hi)) > 1e-4
        units = int(round(float(inside[0]) * 2 ** 21)) if inside else 1 << 26  # out of reach: never within, never above
        cells.append((0x4B400000 + units - CELL_MARGIN - ((base + 1) << 28)) & 0xFFFFFFFF)
        cut = bf16_cut(inside[0]) if inside else 1 << 26
        cells_bf16.append((0x4B400000 + cut - ((base + 1) << 28)) & 0xFFFFFFFF)
    cells += [0x7FFFFFFF] * (64 - len(cells))
    cells_bf16 += [0x7FFFFFFF] * (64 - len(cells_bf16))
    lines.append("// 33 cells of width 1/16 over [-1, 1], padded to 64 (see nf4_common.cuh: FastCodes)")
    lines.append("#define NF4_CELL_MARGIN %d" % CELL_MARGIN)
    lines.append("#define NF4_CELL_TABLE_LIST \\")
    lines.append("  " + ", ".join("0x%08xu" % c for c in cells))
    lines.append("// the same for quotients of bf16 numbers, with cuts that need no margin (see nf4_common.cuh: codes_of_bf16)")
    lines.append("#define NF4_CELL_BF16_TABLE_LIST \\")
    lines.append("  " + ", ".join("0x%08xu" % c for c in cells_bf16))
    lines.append("// thresholds as decimals: " + ", ".join(repr(float(t)) for t in th))
    out = os.path.join(os.path.dirname(os.path.abspath(__file__)), "nf4_tables.inc")
    with open(out, "w") as f:
        f.write("\n".join(lines) + "\n")
    print("wrote", out)
    for i, t in enumerate(th):
        print(i, repr(float(t)), "mid", 0.5 * (LEVELS_F64[i] + LEVELS_F64[i + 1]))


if __name__ == "__main__":
    main()
