"""Quantize / dequantize of lengths that are no multiple of a block, on aligned buffers (one launch) and unaligned ones;
forwards whose output is a part of a wider buffer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from gpu_util import DEV, bits_equal, lib, ptr  # noqa: E402
from unifur_b200 import _lib  # noqa: E402


@pytest.mark.parametrize("n", [1, 7, 8, 63, 64 + 9, 2048 + 33, 6 * 148 * 2048 + 64 * 5 + 1, 9 * 148 * 2048 + 63])
@pytest.mark.parametrize("shift", [0, 1, 4])  # elements the f32 buffers start past a 512-byte boundary
@pytest.mark.parametrize("packed", [True, False])
def test_any_length_and_alignment(oracle, n, shift, packed):
    L = lib()
    rng = np.random.default_rng(n + shift)
    v = (rng.standard_normal(n) * 0.02).astype(np.float32)
    if n > 100:
        v[5], v[70], v[64:80] = np.nan, np.inf, 0.0
    buf = torch.zeros(n + 8, dtype=torch.float32, device=DEV)
    buf[shift:shift + n] = torch.from_numpy(v).to(DEV)
    src = buf[shift:shift + n]
    codes = torch.full(((n + 1) // 2 if packed else n,), 0xEE, dtype=torch.uint8, device=DEV)
    absmax = torch.full(((n + 63) // 64,), -7.0, dtype=torch.float32, device=DEV)
    _lib.check((L.nf4_quantize_dev if packed else L.nf4_quantize_unpacked_dev)(ptr(src), n, ptr(codes), ptr(absmax), None))
    want, want_absmax = oracle.quantize_packed(v)
    got = codes.cpu().numpy()
    if not packed:
        got = np.concatenate([got, np.zeros(n & 1, np.uint8)])
        got = got[0::2] | (got[1::2] << 4)
    assert got.tobytes() == want.tobytes()
    assert bits_equal(absmax.cpu().numpy(), want_absmax)
    out = torch.full((n + 8,), 123.0, dtype=torch.float32, device=DEV)
    dst = out[shift:shift + n]
    _lib.check((L.nf4_dequantize_dev if packed else L.nf4_dequantize_unpacked_dev)(ptr(codes), n, ptr(absmax), None, None, ptr(dst), None))
    assert bits_equal(dst.cpu().numpy(), oracle.dequantize_packed(want, n, want_absmax))
    rest = torch.cat([out[:shift], out[shift + n:]]).cpu().numpy()
    assert (rest == 123.0).all()


@pytest.mark.parametrize("nb", [1, 3, 4, 63, 4096 + 1, 131072, 131073, 131072 * 4 + 7, (1 << 20) + 5])  # one launch, one cluster, and beyond
def test_double_quantization_of_any_length(oracle, nb):
    from gpu_util import double_quantize_dev

    rng = np.random.default_rng(nb)
    s = np.abs(rng.standard_normal(nb)).astype(np.float32)
    s[:: 7] = s.max() * (np.arange(len(s[:: 7])) % 256 + 0.5) / 255  # next to the rounding boundaries
    sc, sos = double_quantize_dev(s)
    o_sc, o_sos = oracle.double_quantize(s)
    assert sc.tobytes() == o_sc.tobytes() and np.float32(sos).tobytes() == np.float32(o_sos).tobytes()
    d, out, m = torch.from_numpy(s).to(DEV), torch.full((nb + 2,), 77, dtype=torch.uint8, device=DEV), torch.zeros(1, device=DEV)
    _lib.check(_lib.load().nf4_double_quantize_dev(d.data_ptr(), nb, out.data_ptr() + 1, m.data_ptr(), None))  # codes at an odd address
    assert out[1:-1].cpu().numpy().tobytes() == o_sc.tobytes() and out[0] == 77 and out[-1] == 77


@pytest.mark.parametrize("rows", [1, 16, 17, 100, 361])
@pytest.mark.parametrize("n,ld", [(41, 44), (43, 48), (47, 48), (65, 72), (130, 136), (300, 304), (300, 301), (192, 200), (1000, 1024)])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_a_row_s_padding_is_left_alone(rows, n, ld, dt):
    # outputs that end inside a 16-byte piece, in buffers whose rows go on: a tensor map's store writes whole pieces
    from unifur_b200.quantize import PackedNf4Tensor, linear_forward

    k = 128
    g = torch.Generator(device=DEV).manual_seed(rows + n)
    p = PackedNf4Tensor.quantize(torch.randn(k * n, device=DEV, generator=g) * 0.02)
    x = torch.randn(rows, k, device=DEV, generator=g).to(dt)
    buf = torch.full((rows + 1, ld), 7.0, dtype=dt, device=DEV)
    y = linear_forward(x, p, k, n, _lib.LAYOUT_OUT_IN, out=buf[:rows, :n])
    ref = x.double() @ p.dequantize().view(n, k).t().double()
    assert float((y.double() - ref).norm() / ref.norm()) < (1e-3 if dt == torch.float32 else 4e-3)
    assert bool((buf[:, n:] == 7.0).all()) and bool((buf[rows] == 7.0).all())
