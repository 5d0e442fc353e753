"""f32 tensors at decode sizes on W [d_out, d_in]: the kernels around the decode kernel, at odd ranks, widths and rows."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from gpu_util import DEV  # noqa: E402
from unifur_b200 import _lib  # noqa: E402


@pytest.mark.parametrize("rows,k,n,r,shift", [
    (1, 256, 40, 3, 0),        # one value of B at a time, a column group that is not full
    (3, 512, 257, 0, 0),
    (8, 1024, 96, 6, 0),       # four values of B, then two
    (9, 512, 100, 260, 0),     # two passes, the second of one row; more ranks than shared memory holds
    (16, 320, 65, 12, 1),      # B at an odd address
])
def test_f32_rows_against_f64(rows, k, n, r, shift):
    # weights in f16 and sums in f32 bound the error by 1e-3 (the C header's figure); the adapter term is f32 throughout
    from unifur_b200.quantize import PackedNf4Tensor, linear_forward

    g = torch.Generator(device=DEV).manual_seed(rows + k + n)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    p, x, bias = PackedNf4Tensor.quantize(rnd(k * n) * 0.02), rnd(rows, k), rnd(n)
    ref = x.double() @ p.dequantize().view(n, k).t().double() + bias.double()
    kw = {}
    if r:
        a, b = rnd(r, k) * 0.05, torch.cat([torch.zeros(shift, device=DEV), (rnd(n, r) * 0.05).reshape(-1)])[shift:].view(n, r)
        kw = dict(lora_a=a, lora_b=b, lora_scale=1.5)
        ref += 1.5 * (x.double() @ a.t().double()) @ b.t().double()
    buf = torch.full((rows + 1, n + 3), 7.0, device=DEV)
    y = linear_forward(x, p, k, n, _lib.LAYOUT_OUT_IN, bias=bias, out=buf[:rows, :n], **kw)
    assert float((y.double() - ref).norm() / ref.norm()) < 1e-3
    assert bool((buf[:, n:] == 7.0).all()) and bool((buf[rows] == 7.0).all())
