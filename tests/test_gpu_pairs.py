"""The tensor-core kernel where its pairs of CTAs have uneven halves: an odd number of 128-row tiles, activation
tiles whose second half lies beyond the rows, tiles split at stages that are no multiple of four, adapters of one to
four chunks (the dequantisers take turns on the adapter's stages too)."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from test_gpu_linear import check_out_in, make_case  # noqa: E402


@pytest.mark.parametrize("M,K,N,r,dq,bias", [
    (17, 64, 128, 0, False, False),     # one stage, one CTA of the pair without weight rows
    (128, 192, 136, 8, True, True),     # the second half of the activations is empty, rows of W end in a tile
    (129, 448, 640, 16, False, True),
    (300, 1216, 2440, 64, True, False),  # 19 stages: the split tiles' pieces are odd
    (513, 832, 1160, 128, False, False),
    (257, 3008, 392, 256, True, True),  # eight adapter stages behind pieces of a few
    (600, 320, 5000, 256, False, False),  # whole tiles of five stages
    (33, 2048, 520, 16, False, True),   # MMAs of 64 columns, split tiles with three of sixteen chunks of rows
    (96, 4096, 264, 64, True, False),   # of 96, both sets of epilogue warps with and without rows
    (479, 1536, 768, 8, False, False),  # of 224 in the second tile
])
def test_uneven_pairs(oracle, M, K, N, r, dq, bias):
    c = make_case(oracle, 4000 + M + K + N, M, K, N, r, dq=dq, bias=bias)
    check_out_in(oracle, c, M, K, N, 1.5)


@pytest.mark.parametrize("M,K,N,r", [(40, 64, 192, 8), (700, 704, 2496, 64), (2048, 1088, 9536, 128)])
def test_reference_orientation_in_f32(M, K, N, r):
    # f32 factors are two bf16 ranks each: up to eight adapter stages
    from unifur_b200 import _lib
    from unifur_b200.quantize import PackedNf4Tensor, linear_forward

    g = torch.Generator(device="cuda").manual_seed(M)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    p = PackedNf4Tensor.quantize(rnd(K * N) * 0.02)
    x, a, b = rnd(M, K), rnd(K, r) * 0.05, rnd(r, N) * 0.05
    y = linear_forward(x, p, K, N, _lib.LAYOUT_IN_OUT, lora_a=a, lora_b=b, lora_scale=2.0)
    ref = x.double() @ p.dequantize().view(K, N).double() + 2.0 * (x.double() @ a.double()) @ b.double()
    assert float((y.double() - ref).norm() / ref.norm()) < 1e-3


@pytest.mark.parametrize("M,K,N,ld,f32,in_out", [
    (17, 1792, 64, 64, False, False),    # 28 stages in three or four parts
    (19, 4160, 43, 48, False, False),    # the last columns are no whole pieces
    (300, 3008, 392, 400, False, True),  # parts of unequal length, two tiles of rows, the last odd CTA without weight rows
    (65, 20288, 130, 136, True, False),  # two tiles of columns in the most parts
    (257, 2560, 448, 448, True, True),   # one row in the second tile
])
def test_tiles_of_several_pairs(M, K, N, ld, f32, in_out):
    # f16 weights and f32 sums: 1e-3 for f32 results, bf16's own rounding for the others
    from unifur_b200 import _lib
    from unifur_b200.quantize import PackedNf4Tensor, linear_forward

    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    dt, r = torch.float32 if f32 else torch.bfloat16, 8
    p = PackedNf4Tensor.quantize(rnd(K * N) * 0.02)
    a, b = rnd(K, r) * 0.05, rnd(r, N) * 0.05
    x, bias, a, b = rnd(M, K).to(dt), rnd(N), a.to(dt), b.to(dt)
    la, lb = (a, b) if in_out else (a.t().contiguous(), b.t().contiguous())
    w = p.dequantize().double()
    w = w.view(K, N) if in_out else w.view(N, K).t()
    ref = x.double() @ w + bias.double() + 1.5 * (x.double() @ a.double()) @ b.double()
    buf = torch.full((M + 1, ld), 7.0, dtype=dt, device="cuda")
    layout = _lib.LAYOUT_IN_OUT if in_out else _lib.LAYOUT_OUT_IN
    for _ in range(2):
        y = linear_forward(x, p, K, N, layout, bias=bias, lora_a=la, lora_b=lb, lora_scale=1.5, out=buf[:M, :N])
        assert float((y.double() - ref).norm() / ref.norm()) < (1e-3 if f32 else 4e-3)
    first = y.clone()
    assert torch.equal(first, linear_forward(x, p, K, N, layout, bias=bias, lora_a=la, lora_b=lb, lora_scale=1.5, out=buf[:M, :N]))
    assert bool((buf[:, N:] == 7.0).all()) and bool((buf[M] == 7.0).all())


def test_repeated_calls_agree():
    # several tiles to a pair, so that the epilogue's traffic runs beside the dequantisers': a slot of the rings given
    # back too early shows as a few weight rows that differ from call to call
    from unifur_b200 import _lib
    from unifur_b200.quantize import PackedNf4Tensor, linear_forward

    g = torch.Generator(device="cuda").manual_seed(5)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    m, k, n = 512, 4096, 18944
    p = PackedNf4Tensor.quantize(rnd(n * k) * 0.02)
    x, flush = rnd(m, k).bfloat16(), torch.empty(48 << 20, device="cuda")
    first = linear_forward(x, p, k, n, _lib.LAYOUT_OUT_IN).clone()
    for i in range(200):
        if i % 2:
            flush.zero_()
        assert torch.equal(first, linear_forward(x, p, k, n, _lib.LAYOUT_OUT_IN)), i
