"""Decode sizes whose d_in is whole quantization blocks but no multiple of a warp's slice of 256."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from test_gpu_linear import check_out_in, make_case  # noqa: E402


@pytest.mark.parametrize("M,K,N,r,dq,bias", [
    (1, 64, 48, 0, False, False),       # one block: three of the slice's four are missing
    (4, 192, 200, 8, True, True),       # byte-wise u8 scales, rows beyond N in the last tile
    (8, 448, 1000, 16, False, True),
    (9, 960, 320, 64, True, False),     # two MMA columns of rows
    (16, 3904, 4720, 32, False, False),
    (3, 4160, 272, 16, True, False),    # K in two parts, the second one block long at its end
    (16, 8384, 144, 8, False, True),
    (2, 32704, 64, 16, False, False),   # the longest K: eight parts
])
def test_d_in_of_whole_blocks(oracle, M, K, N, r, dq, bias):
    c = make_case(oracle, 2000 + M + K + N, M, K, N, r, dq=dq, bias=bias)
    check_out_in(oracle, c, M, K, N, 1.5)


@pytest.mark.parametrize("dq", [False, True])
def test_grouped_projections_of_such_a_d_in(oracle, dq):
    from unifur_b200 import _lib
    from unifur_b200.quantize import PackedNf4Tensor, linear_forward, linear_forward_grouped

    gen = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    k = 1344
    x = rnd(5, k).bfloat16()
    prs = []
    for n in (640, 64, 72):
        p = PackedNf4Tensor.quantize(rnd(n * k) * 0.02)
        prs.append({"packed": p.with_double_quantization() if dq else p, "d_out": n, "lora_a": (rnd(16, k) * 0.05).bfloat16(),
                    "lora_b": (rnd(n, 16) * 0.05).bfloat16(), "lora_scale": 2.0})
    ys = linear_forward_grouped(x, k, _lib.LAYOUT_OUT_IN, prs)
    for y, pr in zip(ys, prs):
        one = linear_forward(x, pr["packed"], k, pr["d_out"], _lib.LAYOUT_OUT_IN, lora_a=pr["lora_a"], lora_b=pr["lora_b"],
                             lora_scale=2.0)
        assert torch.equal(y, one)
        w = pr["packed"].dequantize().view(pr["d_out"], k).double()
        ref = x.double() @ w.t() + 2.0 * (x.double() @ pr["lora_a"].double().t()) @ pr["lora_b"].double().t()
        assert float((y.double() - ref).norm() / ref.norm()) < 4e-3
