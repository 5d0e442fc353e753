"""A checkpoint's matrix to a double-quantized weight in one call: the same bytes as in two, whichever kernels take it."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from gpu_util import DEV, ptr  # noqa: E402
from unifur_b200 import _lib  # noqa: E402


@pytest.mark.parametrize("rows,cols,dtype", [
    (4096, 4096, torch.bfloat16),    # the quantizer's CTAs have the maxima: a tile or two each
    (1024, 8192, torch.bfloat16),    # 256 tiles
    (4416, 4096, torch.float32),     # 69 segments of f32
    (14336, 1032, torch.bfloat16),   # a strip of four words
    (256, 512, torch.bfloat16),      # without TMA
    (70, 36, torch.float32),         # transposed first
    (0, 64, torch.float32),
])
@pytest.mark.parametrize("where", ["first", "last", "zeros"])
def test_same_as_two_calls(rows, cols, dtype, where):
    from unifur_b200.quantize import PackedNf4Tensor
    from unifur_b200.qwennet import Nf4Linear

    gen = torch.Generator(device=DEV).manual_seed(rows + cols)
    w = torch.randn(rows, cols, device=DEV, generator=gen) * (0.0 if where == "zeros" else 0.02)
    if w.numel() and where != "zeros":
        w[(0, 0) if where == "first" else (-1, -1)] = -3.0  # the largest scale is one end's
    w = w.to(dtype)
    two = PackedNf4Tensor.quantize_transposed(w).with_double_quantization()
    one = Nf4Linear.from_checkpoint(w).packed() if rows else PackedNf4Tensor._from_checkpoint(w)
    assert torch.equal(one.codes, two.codes) and torch.equal(one.scale_codes, two.scale_codes)
    assert torch.equal(one.scale_of_scales, two.scale_of_scales)
    if w.numel() and where != "zeros":
        assert float(one.scale_of_scales) == 3.0


def test_workspace_is_checked():
    L = _lib.load()
    rows, cols = 4096, 4096
    w = torch.zeros(rows, cols, device=DEV, dtype=torch.bfloat16)
    codes, absmax = torch.empty(rows * cols // 2, dtype=torch.uint8, device=DEV), torch.empty(rows * cols // 64, device=DEV)
    sc, sos = torch.empty(rows * cols // 64, dtype=torch.uint8, device=DEV), torch.empty(1, device=DEV)
    need = L.nf4_quantize_transposed_double_workspace_bytes(rows, cols)
    ws = torch.empty(need, dtype=torch.uint8, device=DEV)
    call = lambda p, n: L.nf4_quantize_transposed_double_dev(  # noqa: E731
        ptr(w), _lib.DTYPE_BF16, rows, cols, ptr(codes), ptr(absmax), ptr(sc), ptr(sos), p, n, None)
    assert call(ptr(ws), need - 1) != 0 and call(None, need) != 0
    assert call(ptr(ws), need) == 0
    torch.cuda.synchronize()
    assert float(sos) == 0.0 and not sc.any()
