"""The tensor-core GEMM's steps of two k-stages: odd counts of stages, adapters of several chunks in the activations' ring, the
ways its scales come in, and both widths of its tiles at their edges."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from gpu_util import DEV  # noqa: E402
from unifur_b200 import _lib  # noqa: E402


@pytest.mark.parametrize("M,K,N,r,layout,f32,double", [
    (17, 64, 136, 8, 0, False, False),       # half a step
    (128, 192, 264, 0, 0, False, False),     # a step and a half; the last row of a narrow tile
    (129, 192, 264, 72, 0, False, False),    # the first of a wide one; two chunks of the adapter
    (31, 256, 256, 200, 0, False, False),    # scales by TMA: a single box; four chunks, fewer main steps than slots
    (33, 1024, 520, 16, 0, False, True),     # u8 scales by TMA
    (96, 2048, 256, 136, 0, False, True),
    (127, 960, 384, 24, 0, True, True),      # u8 scales loaded; f32 tensors
    (256, 4160, 512, 16, 0, False, False),   # an odd number of stages, divided between pairs
    (257, 1280, 40000, 40, 0, False, False), # more tiles than pairs: whole and shared ones, the shared odd
    (100, 1344, 40000, 130, 0, False, True),
    (640, 2624, 5120, 0, 0, True, False),
    (224, 3584, 9472, 16, 0, False, True),   # a tile to half of the pairs
    (65, 448, 320, 64, 1, False, False),     # the other orientation: a scale for every k
    (300, 1088, 640, 72, 1, True, True),
    (90, 8256, 256, 8, 1, False, False),
])
def test_steps(M, K, N, r, layout, f32, double):
    from unifur_b200.quantize import PackedNf4Tensor
    from unifur_b200.qwennet import Nf4Linear, QloraLinear

    dt = torch.float32 if f32 else torch.bfloat16
    gen = torch.Generator(device=DEV).manual_seed(M * K + N)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen)  # noqa: E731
    packed = PackedNf4Tensor.quantize(rnd(K * N) * 0.02)
    base = Nf4Linear(packed.with_double_quantization() if double else packed, K, N, rnd(N), layout)
    w = base.dequantized_weight().double()
    w = w.t() if layout == 0 else w
    x = rnd(M, K).to(dt)
    ref = x.double() @ w + base.bias.double()
    if r:
        a, b = ((r, K), (N, r)) if layout == 0 else ((K, r), (r, N))
        base = QloraLinear(base, (rnd(*a) * 0.1).to(dt), (rnd(*b) * 0.1).to(dt), 1.5)
        A, B = base.lora_a.double(), base.lora_b.double()
        ref += 1.5 * (x.double() @ (A.t() if layout == 0 else A)) @ (B.t() if layout == 0 else B)
    y = base.forward(x).double()
    per_row = ((y - ref).norm(dim=1) / ref.norm(dim=1)).max()
    assert float(per_row) < (1e-3 if f32 else 4e-3)  # the C header's bound; bf16 results round once more (2^-9)
    per_column = ((y - ref).norm(dim=0) / ref.norm(dim=0)).max()
    assert float(per_column) < (1e-3 if f32 else 4e-3)
    assert torch.equal(y, base.forward(x).double())  # results do not depend on timing


@pytest.mark.parametrize("M,K,N,r,layout,f32,double", [
    (100, 4096, 4096, 16, 0, False, False),   # narrow tiles: scales by TMA, a chunk of the adapter
    (64, 3584, 9472, 136, 0, False, True),    # u8 scales loaded, three chunks
    (48, 2048, 20480, 8, 0, False, True),     # u8 scales by TMA, more tiles than pairs
    (128, 4160, 4096, 136, 1, False, False),  # a scale for every k, three chunks, an odd last step
    (100, 1024, 20480, 8, 1, True, False),    # the same of f32 tensors, tiles divided between pairs
    (600, 4096, 10240, 64, 0, False, False),  # wide tiles
])
def test_codes_that_come_late(M, K, N, r, layout, f32, double):
    # the codes' copies land from a cold L2 and in no order; the ring's protocol is tests/test_code_ring.py's
    from unifur_b200.quantize import PackedNf4Tensor
    from unifur_b200.qwennet import Nf4Linear, QloraLinear

    dt = torch.float32 if f32 else torch.bfloat16
    gen = torch.Generator(device=DEV).manual_seed(M + N)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen)  # noqa: E731
    packed = PackedNf4Tensor.quantize(rnd(K * N) * 0.02)
    base = Nf4Linear(packed.with_double_quantization() if double else packed, K, N, None, layout)
    a, b = ((r, K), (N, r)) if layout == 0 else ((K, r), (r, N))
    q = QloraLinear(base, (rnd(*a) * 0.1).to(dt), (rnd(*b) * 0.1).to(dt), 1.5)
    x, flush = rnd(M, K).to(dt), torch.empty(1 << 28, dtype=torch.uint8, device=DEV)
    first = q.forward(x)
    for i in range(20):
        flush.fill_(i)
        assert torch.equal(q.forward(x), first)
