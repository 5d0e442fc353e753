"""The strip kernel of the reference's orientation: runs of K units shared out between CTAs, every row count's variant."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from test_gpu_linear import run_forward  # noqa: E402
from unifur_b200 import _lib  # noqa: E402


@pytest.mark.parametrize("rows,d_in,d_out,r,dq,f32", [
    (1, 1, 64, 0, False, True),          # one row of W, one block: a quarter of a strip
    (1, 4096, 320, 16, True, True),      # many CTAs per strip, the last strip a quarter full
    (2, 65, 576, 4, False, False),       # the second unit has one row
    (3, 1000, 256, 0, True, False),
    (4, 2048, 4672, 8, False, True),     # strips whose K is split between two CTAs
    (6, 8192, 64, 64, True, True),
    (8, 640, 11008, 16, False, True),    # CTAs with the end of one strip and the start of the next
    (13, 4160, 1344, 32, True, True),    # activations of K in several pieces
    (2, 300, 2304, 4, False, True),      # a cluster to a strip, a unit to a CTA, the last one short
    (1, 4096, 10944, 0, True, True),     # clusters of three with unequal parts, the last strip three quarters full
    (7, 3072, 8192, 16, False, False),
    (11, 1536, 6976, 24, True, True),
    (16, 20480, 128, 8, False, False),
    (37, 100, 192, 3, False, True),      # d_in the tensor-core path does not take: sixteen rows per launch
    (5, 64, 63552, 0, True, False),      # more strips than counters: whole strips per CTA
])
def test_against_f64(oracle, rows, d_in, d_out, r, dq, f32):
    rng = np.random.default_rng(300 + rows + d_in + d_out)
    w = (rng.standard_normal((d_in, d_out)) * 0.02).astype(np.float32)
    packed, absmax = oracle.quantize_packed(w)
    sc = sos = None
    if dq:
        sc, sos = oracle.double_quantize(absmax)
    x = rng.uniform(-1, 1, (rows, d_in)).astype(np.float32)
    la = (rng.standard_normal((d_in, r)) * 0.05).astype(np.float32) if r else None
    lb = rng.uniform(-0.5, 0.5, (r, d_out)).astype(np.float32) if r else None
    if not f32:
        x = oracle.round_bf16(x)
        la, lb = (oracle.round_bf16(la), oracle.round_bf16(lb)) if r else (None, None)
    bias = rng.standard_normal(d_out).astype(np.float32)
    ref = oracle.qlora_forward_burn(x, packed, None if dq else absmax, d_in, d_out, la, lb, 2.0, bias, sc, 0.0 if sos is None else sos)
    kw = dict(bias=bias, lora_a=la, lora_b=lb, scale=2.0, scale_codes=sc, sos=sos)
    dt = _lib.DTYPE_F32 if f32 else _lib.DTYPE_BF16
    run = lambda: run_forward(_lib.LAYOUT_IN_OUT, dt, x, packed, None if dq else absmax, d_in, d_out, y_f32=True, calls=2, **kw)  # noqa: E731
    got = run()
    assert np.linalg.norm(got - ref) <= 2e-6 * np.linalg.norm(ref)
    assert got.tobytes() == run().tobytes()  # sums in a fixed order
