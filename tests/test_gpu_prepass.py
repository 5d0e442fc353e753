"""The pre-pass of the tensor-core path and the adapter gradients: pieces of K over a cluster, ragged rows and ranks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from gpu_util import DEV  # noqa: E402
from unifur_b200 import _lib  # noqa: E402


def layer(M, K, N, r, layout, dt, seed, x_std=1.0):
    from unifur_b200.quantize import PackedNf4Tensor
    from unifur_b200.qwennet import Nf4Linear, QloraLinear

    gen = torch.Generator(device=DEV).manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen)  # noqa: E731
    out_in = layout == _lib.LAYOUT_OUT_IN
    a, b = ((r, K), (N, r)) if out_in else ((K, r), (r, N))
    base = Nf4Linear(PackedNf4Tensor.quantize(rnd(K * N) * 0.02), K, N, None, layout)
    q = QloraLinear(base, (rnd(*a) * 0.1).to(dt), (rnd(*b) * 0.1).to(dt), 1.5)
    w = base.dequantized_weight().double()
    w = w.t() if out_in else w                                       # [K, N]
    A, B = q.lora_a.double(), q.lora_b.double()
    A, B = (A.t(), B.t()) if out_in else (A, B)                      # [K, r], [r, N]
    x = rnd(M, K) * x_std
    x = x * torch.logspace(-12, 12, M, base=2.0, device=DEV)[:, None]  # rows far apart in magnitude
    return q, w, A, B, x.to(dt), rnd


def rel(got, ref):
    return float((got.double() - ref).norm() / ref.norm())


@pytest.mark.parametrize("M,K,N,r,layout,f32", [
    (17, 64, 64, 8, 0, False),         # one stage of K, one CTA
    (33, 320, 128, 16, 0, False),      # K pieces of unequal length, one row in the second tile
    (100, 4096, 256, 64, 0, False),    # sixteen CTAs per tile
    (300, 2112, 192, 72, 0, False),    # more than 64 ranks
    (64, 704, 320, 24, 1, False),      # the factor [K, r] through transposing loads
    (40, 1024, 128, 12, 0, True),      # f32: converted in place
    (70, 4160, 64, 4, 1, True),
    (20, 65536, 64, 8, 0, False),      # K in several pieces of shared memory
    (18, 40960, 64, 8, 0, True),
    (513, 192, 136, 8, 0, False),      # 64 rows to a tile: one row in the last, stages of 128 k half empty
    (600, 1088, 128, 20, 1, False),    # the same, the factor [K, r] in odd places
    (545, 576, 64, 12, 0, True),       # f32, 64 rows to a tile
    (1029, 4160, 64, 24, 0, False),    # from four million values on the tcgen05 kernel: ragged rows, ranks and pieces of K
    (2050, 2112, 64, 64, 1, False),    # the factor [K, r] as the MMA's MN-major operand
    (16500, 256, 64, 8, 0, False),     # a CTA by itself
    (1200, 2112, 64, 40, 1, True),
])
def test_forward(M, K, N, r, layout, f32):
    dt = torch.float32 if f32 else torch.bfloat16
    q, w, A, B, x, _ = layer(M, K, N, r, layout, dt, M + K + N)
    y = q.forward(x)
    ref = x.double() @ w + 1.5 * (x.double() @ A) @ B
    per_row = ((y.double() - ref).norm(dim=1) / ref.norm(dim=1)).max()
    assert float(per_row) < (1e-3 if f32 else 4e-3)


@pytest.mark.parametrize("first,std", [(0.0, 1.0), (float("inf"), 1.0), (3e38, 1e-4), (1e-30, 1.0), (1e-3, 1e-3)])
def test_rows_far_from_the_first_values(first, std):
    # The copy's common factor follows the first row's first values; rows it does not suit get their own.
    # (Row 0 itself may be infinite.)  8 bits of x and 11 of the weights: the bound of the other forwards.
    q, w, A, B, x, _ = layer(1030, 4096, 64, 16, 0, torch.bfloat16, 7, x_std=std)
    x[0] = first
    y = q.forward(x)
    ref = x.double() @ w + 1.5 * (x.double() @ A) @ B
    per_row = (y[1:].double() - ref[1:]).norm(dim=1) / ref[1:].norm(dim=1)
    assert float(per_row.max()) < 4e-3


@pytest.mark.parametrize("first", [1000.0, 1e-30, 0.0, 0.5])
@pytest.mark.parametrize("big", [1.0, 3e4, 1e5, 2.0 ** -9])
def test_a_row_does_not_depend_on_the_first_row(first, big):
    # Rows of small values around one large one that meets a zero weight (and a zero of the factor): what the outputs are
    # made of lies 2^-16 below the row's maximum, where a copy with a factor that suits other rows keeps few of its bits.
    # The bound of the other forwards, and the same bits whatever stands in row 0.
    from unifur_b200.quantize import PackedNf4Tensor
    from unifur_b200.qwennet import Nf4Linear, QloraLinear

    M, K, N, r = 1030, 4096, 64, 16
    gen = torch.Generator(device=DEV).manual_seed(11)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen)  # noqa: E731
    W, A, B = rnd(N, K) * 0.02, (rnd(r, K) * 0.1).bfloat16(), (rnd(N, r) * 0.1).bfloat16()
    W[:, 300] = 0
    A[:, 300] = 0
    base = Nf4Linear(PackedNf4Tensor.quantize(W.flatten()), K, N, None, _lib.LAYOUT_OUT_IN)
    q = QloraLinear(base, A, B, 1.5)
    w = base.dequantized_weight().double().t()
    assert not w[300].any()
    x = (rnd(M, K) * big * 2.0 ** -16).bfloat16()
    x[:, 300] = big
    x[0] = first
    y = q.forward(x)
    ref = x.double() @ w + 1.5 * (x.double() @ A.double().t()) @ B.double().t()
    per_row = (y[1:].double() - ref[1:]).norm(dim=1) / ref[1:].norm(dim=1)
    assert float(per_row.max()) < 4e-3
    x[0] = 1.0
    assert torch.equal(q.forward(x)[1:], y[1:])


@pytest.mark.parametrize("M,K,N,r,layout", [
    (1, 64, 128, 8, 0), (5, 200, 136, 5, 1), (16, 1024, 512, 16, 0),   # decode sizes: both intermediates by the product-only mode
    (63, 256, 384, 16, 1), (513, 640, 200, 80, 0), (2049, 576, 1344, 64, 1),   # shares of the rows, ragged pieces of columns
    (1100, 128, 32000, 8, 0),                                          # 250 tiles of columns by CTAs on their own, one by a cluster of eight
])
def test_backward(M, K, N, r, layout):
    q, w, A, B, x, rnd = layer(M, K, N, r, layout, torch.bfloat16, M + K + N)
    x = torch.randn(M, K, device=DEV).bfloat16()
    gy = (rnd(M, N) * 1e-3).bfloat16()
    gx, ga, gb = q.backward(x, gy)
    again = q.backward(x, gy)
    assert all(torch.equal(u, v) for u, v in zip((gx, ga, gb), again))
    X, G = x.double(), gy.double()
    gA, gB = 1.5 * X.t() @ (G @ B.t()), 1.5 * (X @ A).t() @ G
    gA, gB = (gA.t(), gB.t()) if layout == _lib.LAYOUT_OUT_IN else (gA, gB)
    assert rel(gx, G @ w.t() + 1.5 * (G @ B.t()) @ A.t()) < 4e-3
    assert rel(ga, gA) < 3e-3 and rel(gb, gB) < 3e-3
