"""The workspace's contract: whatever kernel a call is routed to, the first 256 bytes are zero after it as they were
before it, so that a workspace that has served one call serves any other."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from gpu_util import DEV, lib  # noqa: E402
from unifur_b200 import _lib  # noqa: E402

OUT_IN, IN_OUT = _lib.LAYOUT_OUT_IN, _lib.LAYOUT_IN_OUT
BF16, F32 = torch.bfloat16, torch.float32

ROUTES = [
    (4, 512, 256, 16, OUT_IN, BF16),     # decode kernel, adapter
    (3, 8192, 192, 8, OUT_IN, BF16),     # decode kernel, K in parts
    (5, 1024, 256, 24, OUT_IN, BF16),    # split-K kernel: a rank the decode kernel does not multiply
    (16, 512, 320, 56, OUT_IN, BF16),
    (16, 512, 136, 1, OUT_IN, BF16),     # split-K kernel, the smallest rank
    (2, 36864, 128, 12, OUT_IN, BF16),   # split-K kernel, d_in beyond the decode kernel's
    (2, 256, 320, 4, IN_OUT, F32),       # strip kernel
    (20, 320, 192, 3, IN_OUT, F32),      # strip kernel, two launches
    (3, 512, 256, 8, OUT_IN, F32),       # f32 rows as bf16 halves
    (9, 36864, 64, 4, OUT_IN, F32),      # the same through the split-K kernel, two passes
    (40, 256, 192, 16, OUT_IN, BF16),    # tensor-core GEMM
    (40, 256, 192, 8, IN_OUT, F32),      # tensor-core GEMM, repacked
    (5, 200, 100, 5, OUT_IN, BF16),      # general kernel
]


class Call:
    """One forward's operands and what its workspace has to hold."""

    def __init__(self, rows, k, n, r, layout, dt, seed):
        from unifur_b200.quantize import PackedNf4Tensor

        g = torch.Generator(device=DEV).manual_seed(seed)
        rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
        a, b = ((r, k), (n, r)) if layout == OUT_IN else ((k, r), (r, n))
        self.p = PackedNf4Tensor.quantize(rnd(k * n) * 0.02)
        self.x, self.la, self.lb = rnd(rows, k).to(dt), (rnd(*a) * 0.05).to(dt), (rnd(*b) * 0.05).to(dt)
        self.gy = rnd(rows, n).to(dt)
        self.y = torch.empty(rows, n, dtype=dt, device=DEV)
        self.rank, self.sizes = r, (rows, k, n, r)
        s = self.args = _lib.LinearArgs()
        s.struct_bytes = ctypes.sizeof(s)
        s.layout, s.io_dtype = layout, _lib.DTYPE_F32 if dt == F32 else _lib.DTYPE_BF16
        s.rows, s.d_in, s.d_out = rows, k, n
        s.x, s.packed, s.absmax = self.x.data_ptr(), self.p.codes.data_ptr(), self.p.absmax.data_ptr()
        s.lora_a, s.lora_b, s.lora_rank, s.lora_scale = self.la.data_ptr(), self.lb.data_ptr(), r, 1.5
        s.y, s.ldy = self.y.data_ptr(), n

    def forward(self, ws):
        self.args.workspace, self.args.workspace_bytes = ws.data_ptr(), ws.numel()
        _lib.check(lib().nf4_linear_forward_dev(ctypes.byref(self.args), None))
        return self.y

    def backward(self, ws):
        self.args.workspace, self.args.workspace_bytes = ws.data_ptr(), ws.numel()
        out = [torch.empty_like(t) for t in (self.x, self.la, self.lb)]
        _lib.check(lib().nf4_qlora_backward_dev(ctypes.byref(self.args), self.gy.data_ptr(), *[t.data_ptr() for t in out], None))
        return out

    def bytes(self, backward=False):
        return int((lib().nf4_qlora_backward_workspace_bytes if backward else lib().nf4_linear_workspace_bytes)(*self.sizes))


def workspace(*sizes):
    return torch.zeros(max(256, *sizes), dtype=torch.uint8, device=DEV)


@pytest.mark.parametrize("backward", [False, True])
@pytest.mark.parametrize("route", ROUTES)
def test_flag_words_are_left_zero(route, backward):
    c, decode = Call(*route, seed=sum(route[:4])), Call(*ROUTES[0], seed=1)
    want = decode.forward(workspace(decode.bytes())).clone()
    ws = workspace(c.bytes(backward), decode.bytes())
    c.backward(ws) if backward else c.forward(ws)
    torch.cuda.synchronize()
    assert int(ws[:256].count_nonzero()) == 0
    decode.y.zero_()
    assert torch.equal(decode.forward(ws), want)
    _lib.check(lib().nf4_device_status(None, None, None))


@pytest.mark.parametrize("backward", [False, True])
@pytest.mark.parametrize("route", [r for r in ROUTES if r[:4] in (
    (5, 1024, 256, 24), (2, 36864, 128, 12), (40, 256, 192, 16), (40, 256, 192, 8), (5, 200, 100, 5))])
def test_routes_without_flag_words_run_on_any_workspace(route, backward):
    c = Call(*route, seed=sum(route[:4]))
    run = c.backward if backward else c.forward
    c.args.y = c.y.data_ptr()
    gx = torch.empty_like(c.x)
    flags = lib().nf4_qlora_backward_flag_bytes(ctypes.byref(c.args), c.gy.data_ptr(), gx.data_ptr()) if backward else \
        lib().nf4_linear_flag_bytes(ctypes.byref(c.args))
    assert flags == (256 if backward and route[0] <= 16 and route[1] % 64 == 0 else 0)  # (strip kernel)
    want = [t.clone() for t in run(workspace(c.bytes(backward)))]
    ws = workspace(c.bytes(backward))
    ws[flags:] = 0xAB
    got = run(ws)
    assert all(torch.equal(u, v) for u, v in zip(got, want))
    assert torch.equal(ws[:256], torch.full_like(ws[:256], 0 if flags else 0xAB))
    _lib.check(lib().nf4_device_status(None, None, None))


def test_a_wait_for_arrivals_that_gives_up_leaves_the_counter_and_the_workspace_usable():
    # One rank, whose counter nothing but this test adds to: the forwards wait out their second and say so.  An
    # unsigned counter would wrap when the arrivals are taken off, and the next wait would pass without any.
    L = lib()
    rows, k, n, r = 4, 512, 256, 16
    c = Call(rows, k, n, r, OUT_IN, BF16, seed=3)
    want = c.forward(workspace(c.bytes())).clone()
    ws, counters = workspace(c.bytes()), torch.zeros(2, dtype=torch.int32, device=DEV)
    c.args.workspace, c.args.workspace_bytes = ws.data_ptr(), ws.numel()
    y = torch.zeros(rows, n, dtype=BF16, device=DEV)
    po = _lib.PeerOutputs()
    po.struct_bytes, po.world, po.rank, po.ldy_full = ctypes.sizeof(po), 1, 0, n
    po.y_full[0], po.arrivals[0], po.signal = y.data_ptr(), counters[1:].data_ptr(), 1
    po.wait_arrivals, po.wait_expected = counters[:1].data_ptr(), 1
    for step in (1, 2):
        _lib.check(L.nf4_linear_forward_scatter_dev(ctypes.byref(c.args), ctypes.byref(po), None))
        assert L.nf4_device_status(None, None, None) == -5
        assert counters.tolist() == [-step, step]
        assert int(ws[:256].count_nonzero()) == 0
    counters[0] += 3  # both late arrivals and the next one
    _lib.check(L.nf4_linear_forward_scatter_dev(ctypes.byref(c.args), ctypes.byref(po), None))
    _lib.check(L.nf4_device_status(None, None, None))
    assert counters.tolist() == [0, 3] and torch.equal(y, want)
    # the wait by itself, a millisecond
    _lib.check(L.nf4_peer_arrivals_wait_dev(counters.data_ptr(), 2, 1_000_000, None))
    assert L.nf4_device_status(None, None, None) == -5
    counters[0] += 2
    assert counters.tolist() == [0, 3]
    assert torch.equal(c.forward(ws), want)
