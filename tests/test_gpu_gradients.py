"""The adapter's gradients: the ring of six stages and its wrap, the number of tiles from which it has three."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from gpu_util import DEV  # noqa: E402
from unifur_b200 import _lib  # noqa: E402


@pytest.mark.parametrize("M,K,N,r", [
    (384, 128, 18816, 8),    # 148 tiles, each a CTA's: six stages, the ring once
    (385, 128, 18816, 8),    # a stage begins it again
    (833, 128, 18816, 64),   # twice around and one row
    (385, 128, 18944, 8),    # 149 tiles: three stages, two CTAs on an SM
    (385, 128, 9472, 72),    # 75 tiles, twice for 72 ranks
])
def test_gradients(M, K, N, r):
    from unifur_b200.quantize import PackedNf4Tensor
    from unifur_b200.qwennet import Nf4Linear, QloraLinear

    gen = torch.Generator(device=DEV).manual_seed(M + N + r)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen)  # noqa: E731
    base = Nf4Linear(PackedNf4Tensor.quantize(rnd(K * N) * 0.02), K, N, None, _lib.LAYOUT_OUT_IN)
    q = QloraLinear(base, (rnd(r, K) * 0.1).bfloat16(), (rnd(N, r) * 0.1).bfloat16(), 1.5)
    x, gy = rnd(M, K).bfloat16(), (rnd(M, N) * 1e-3).bfloat16()
    _, ga, gb = q.backward(x, gy)
    A, B, X, G = (t.double() for t in (q.lora_a, q.lora_b, x, gy))
    for got, ref in ((ga, 1.5 * (G @ B).t() @ X), (gb, 1.5 * G.t() @ (X @ A.t()))):
        # T and U as pairs of bf16 (2^-17), f32 sums, one rounding to bf16: 2^-9 an element at most
        assert float((got.double() - ref).norm() / ref.norm()) < 2.0 ** -9
    again = q.backward(x, gy)
    assert torch.equal(again[1], ga) and torch.equal(again[2], gb)
