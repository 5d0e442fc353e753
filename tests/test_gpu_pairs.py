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
