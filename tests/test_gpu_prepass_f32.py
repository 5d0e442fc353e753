"""The f32 pre-pass: pieces of K that stay in registers and longer ones, empty pieces, groups of sixteen ranks, factors at odd places."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from gpu_util import DEV  # noqa: E402
from unifur_b200 import _lib  # noqa: E402


def reference(x, w, A, B):
    return x.double() @ w + 1.5 * (x.double() @ A) @ B


@pytest.mark.parametrize("layout", [_lib.LAYOUT_OUT_IN, _lib.LAYOUT_IN_OUT])
@pytest.mark.parametrize("M,K,N,r,odd", [
    (17, 64, 64, 4, False),        # one CTA, two of its sixteen units of 32 k
    (32, 512, 128, 16, False),     # a whole tile and group of ranks
    (33, 576, 64, 20, False),      # a row and a group begun; a CTA without k
    (64, 8256, 64, 128, False),    # a piece in more than one part, the most ranks
    (2100, 1088, 64, 36, False),   # more clusters than there is room for at once
    (40, 320, 64, 12, True),       # a factor off 16 bytes
])
def test_forward(M, K, N, r, odd, layout):
    from unifur_b200.quantize import PackedNf4Tensor
    from unifur_b200.qwennet import Nf4Linear, QloraLinear

    gen = torch.Generator(device=DEV).manual_seed(M + K + r)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen)  # noqa: E731
    out_in = layout == _lib.LAYOUT_OUT_IN
    base = Nf4Linear(PackedNf4Tensor.quantize(rnd(K * N) * 0.02), K, N, None, layout)
    w = base.dequantized_weight().double()
    w = w.t() if out_in else w
    a = torch.empty(K * r + 1, device=DEV)[int(odd):][:K * r].view((r, K) if out_in else (K, r)).copy_(rnd(K * r).view((r, K) if out_in else (K, r)) * 0.1)
    b = rnd(*((N, r) if out_in else (r, N))) * 0.1
    q = QloraLinear(base, a, b, 1.5)
    A, B = (a.double().t(), b.double().t()) if out_in else (a.double(), b.double())
    x = rnd(M, K) * torch.logspace(-30, 30, M, base=2.0, device=DEV)[:, None]
    y = q.forward(x)
    ref = reference(x, w, A, B)
    # f16 operands: 2^-11 a factor of a product, twice, at random over the sum; the C header's bound
    assert float(((y.double() - ref).norm(dim=1) / ref.norm(dim=1)).max()) < 1e-3
    assert torch.equal(q.forward(x), y)

    x[3], x[5, 7], x[6, K - 1] = 0.0, float("inf"), float("nan")
    x[4, :32], x[7, 40:] = 1e-30, 1e-9  # rows far from their first values
    x[8, :20], x[9, 60] = 0.0, 1e30
    z = q.forward(x)
    rest = [i for i in range(M) if i not in range(3, 10)]
    assert torch.equal(z[rest], y[rest]) and not z[3].any() and not z[5].isfinite().any() and z[6].isnan().all()
    ref = reference(x, w, A, B)
    odd = [4, 7, 8, 9]
    assert float(((z.double() - ref)[odd].norm(dim=1) / ref[odd].norm(dim=1)).max()) < 1e-3


def test_rows_far_from_their_first_values():
    # the copy's first factor follows a row's first sixteen values; the outputs do not
    from unifur_b200.quantize import PackedNf4Tensor
    from unifur_b200.qwennet import Nf4Linear, QloraLinear

    M, K, N, r = 70, 1024, 64, 16
    gen = torch.Generator(device=DEV).manual_seed(3)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen)  # noqa: E731
    W, a = rnd(N, K) * 0.02, rnd(r, K) * 0.1
    W[:, :16] = 0
    a[:, :16] = 0
    base = Nf4Linear(PackedNf4Tensor.quantize(W.flatten()), K, N, None, _lib.LAYOUT_OUT_IN)
    w = base.dequantized_weight().double().t()
    assert not w[:16].any()
    q = QloraLinear(base, a, rnd(N, r) * 0.1, 1.5)
    x = rnd(M, K)
    x[:, :16] = 0
    y = q.forward(x)
    for first in (1.0, 2.0 ** -40, 2.0 ** -17, 2.0 ** 12):
        x[:, 3] = first
        z = q.forward(x)
        assert float((z.double() - y.double()).norm() / y.double().norm()) < 1e-5  # the order of T's sums at most
    # 2^60 and more away T is taken in f32: it then lacks the other rows' rounding of x and A to eleven bits
    x[:, 3] = 2.0 ** -90
    assert float((q.forward(x).double() - y.double()).norm() / y.double().norm()) < 1e-3
    x[:, 3] = 0
    for far in (2.0 ** 100, 2.0 ** -100):
        z = q.forward(x * far).double() / far
        assert float((z - y.double()).norm() / y.double().norm()) < 1e-3
