"""The f32 pre-pass takes a row's factor from the row's largest value wherever that stands: in any CTA's piece of K, in the part of a long
piece that is read a second time, in its last part."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from gpu_util import DEV  # noqa: E402
from unifur_b200 import _lib  # noqa: E402


@pytest.mark.parametrize("layout", [_lib.LAYOUT_OUT_IN, _lib.LAYOUT_IN_OUT])
@pytest.mark.parametrize("M,K,r", [
    (64, 512, 16),       # pieces of 64 k
    (64, 8256, 20),      # 576 k, in two parts
    (33, 20480, 8),      # 1280 k, in three
    (2100, 1088, 36),    # two CTAs or one to a row
    (64, 8256, 0),       # the copy alone
])
def test_maximum_anywhere(M, K, r, layout):
    from unifur_b200.quantize import PackedNf4Tensor
    from unifur_b200.qwennet import Nf4Linear, QloraLinear

    N, out_in = 64, layout == _lib.LAYOUT_OUT_IN
    gen = torch.Generator(device=DEV).manual_seed(M + K + r)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen)  # noqa: E731
    rows = torch.arange(M, device=DEV)
    places = rows % 64 * (K - 1) // min(M - 1, 63)  # from the first k to the last; weight and factor are zero there
    W, a = rnd(K, N) * 0.02, rnd(K, max(r, 1)) * 0.1
    W[places], a[places] = 0, 0
    base = Nf4Linear(PackedNf4Tensor.quantize((W.t() if out_in else W).contiguous().flatten()), K, N, None, layout)
    q = base
    if r:
        b = rnd(N, r) * 0.1
        q = QloraLinear(base, a.t().contiguous() if out_in else a, b if out_in else b.t().contiguous(), 1.5)
    x = rnd(M, K)
    x[rows, places] = 0
    y = q.forward(x)
    # A value far below a row's largest one leaves its factor as it is, and counts for nothing.
    x[rows, places] = 2.0 ** -90
    assert torch.equal(q.forward(x), y)
    # One above it moves the factor, by a power of two: the copy keeps eleven bits of every value down to 2^-14 of f16, here 2^-17 of x
    # (N(0, 1): 1e-5 of the values lie below, and lose 2^-28 at most).  A largest value that was not seen would overflow f16 to an infinity.
    for factor in (2.0 ** 12, -(2.0 ** 12)):
        x[rows, places] = factor
        z = q.forward(x)
        assert float((z - y).norm() / y.norm()) < 1e-6
