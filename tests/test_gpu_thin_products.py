"""The adapter's products on CUDA cores: tiles of 64 with 16, 32 or 64 ranks, shares of the long side, rows off any vector."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from gpu_util import DEV  # noqa: E402
from unifur_b200 import _lib  # noqa: E402


@pytest.mark.parametrize("M,K,N,r,layout,dt", [
    (1, 64, 64, 1, 0, torch.float32),
    (3, 100, 70, 5, 1, torch.float32),         # no multiple of four anywhere
    (64, 256, 320, 16, 0, torch.float32),      # whole tiles
    (65, 4096, 192, 17, 1, torch.float32),     # a row more, a rank more; shares of K
    (512, 1000, 1028, 32, 0, torch.float32),
    (700, 320, 64, 33, 1, torch.float32),
    (300, 1088, 640, 64, 0, torch.float32),
    (130, 192, 256, 130, 1, torch.float32),    # three chunks of ranks
    (70, 100, 66, 12, 0, torch.bfloat16),      # bf16 of sizes the tensor-core gradients do not take
    (33, 132, 36, 40, 1, torch.bfloat16),
])
def test_gradients(M, K, N, r, layout, dt):
    from unifur_b200.quantize import PackedNf4Tensor
    from unifur_b200.qwennet import Nf4Linear, QloraLinear

    gen = torch.Generator(device=DEV).manual_seed(M + K + N + r)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen)  # noqa: E731
    a, b = ((r, K), (N, r)) if layout == _lib.LAYOUT_OUT_IN else ((K, r), (r, N))
    base = Nf4Linear(PackedNf4Tensor.quantize(rnd(K * N) * 0.02), K, N, None, layout)
    q = QloraLinear(base, (rnd(*a) * 0.1).to(dt), (rnd(*b) * 0.1).to(dt), 1.5)
    x, gy = rnd(M, K).to(dt), (rnd(M, N) * 1e-3).to(dt)
    _, ga, gb = q.backward(x, gy)
    A, B, X, G = (t.double() for t in (q.lora_a, q.lora_b, x, gy))
    A, B = (A.t(), B.t()) if layout == _lib.LAYOUT_OUT_IN else (A, B)
    ra, rb = 1.5 * X.t() @ (G @ B.t()), 1.5 * (X @ A).t() @ G
    if layout == _lib.LAYOUT_OUT_IN:
        ra, rb = ra.t(), rb.t()
    # two f32 products in sums of 32 and of those: 2^-24 sqrt(32 + Q / 32) each at random; bf16 rounds the result (2^-9)
    bound = 2.0 ** -24 * 2 * (32 + max(M, K, N) / 32) ** 0.5 + (2.0 ** -9 if dt == torch.bfloat16 else 0.0)
    for got, ref in ((ga, ra), (gb, rb)):
        assert float((got.double() - ref).norm() / ref.norm()) < bound
    again = q.backward(x, gy)
    assert torch.equal(again[1], ga) and torch.equal(again[2], gb)
