"""The mirror's native host path: workspaces kept per thread and stream must serve calls of any mix of shapes."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from gpu_util import DEV  # noqa: E402
from unifur_b200 import _lib  # noqa: E402


def layers():
    from unifur_b200.quantize import PackedNf4Tensor

    gen = torch.Generator(device=DEV).manual_seed(5)
    out = []
    # decode with an adapter, K in parts, strip kernel, d_in no multiple of 256, prefill (its workspace is larger), K in
    # parts again, the split-K kernel (a rank the decode kernel does not multiply)
    for rows, k, n, r, layout, dt in ((4, 512, 256, 16, 0, torch.bfloat16), (3, 8192, 192, 8, 0, torch.bfloat16),
                                      (2, 256, 320, 4, 1, torch.float32), (5, 320, 192, 8, 0, torch.bfloat16),
                                      (40, 256, 192, 16, 0, torch.bfloat16), (16, 4352, 64, 64, 0, torch.bfloat16),
                                      (5, 1024, 192, 24, 0, torch.bfloat16)):
        rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen)  # noqa: E731
        a, b = ((r, k), (n, r)) if layout == 0 else ((k, r), (r, n))
        out.append((rnd(rows, k).to(dt), PackedNf4Tensor.quantize(rnd(k * n) * 0.02), k, n, layout,
                    (rnd(*a) * 0.05).to(dt), (rnd(*b) * 0.05).to(dt)))
    return out


def forward(x, p, k, n, layout, a, b):
    from unifur_b200.quantize import linear_forward

    return linear_forward(x, p, k, n, layout, lora_a=a, lora_b=b, lora_scale=1.5)


@pytest.mark.parametrize("threads", [1, 3])
def test_kept_workspaces_serve_any_mix_of_calls(threads):
    cases = layers()
    want = []
    for c in cases:
        _lib.host().release_workspaces()  # a fresh workspace for every reference result
        want.append(forward(*c).cpu())
    torch.cuda.synchronize()
    bad = []

    def work(seed):
        order = np.random.default_rng(seed).permutation(np.arange(len(cases)).repeat(6))
        streams = [torch.cuda.Stream() for _ in range(2)]
        got = []
        for j, i in enumerate(order):
            with torch.cuda.stream(streams[j % 2]):
                got.append((i, forward(*cases[i])))
        torch.cuda.synchronize()
        bad.extend(i for i, y in got if not torch.equal(y.cpu(), want[i]))

    ts = [threading.Thread(target=work, args=(t,)) for t in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
    _lib.check(_lib.load().nf4_device_status(None, None, None))


@pytest.mark.parametrize("trained", [False, True])
def test_factors_written_right_ahead_of_a_forward(trained):
    # converted by the call itself, or by an optimizer's step before it: the decode kernel asks for factors early
    from unifur_b200.quantize import linear_forward

    x, p, k, n, layout, a, b = layers()[0]
    want = [linear_forward(x, p, k, n, layout, lora_a=a * s, lora_b=b * s, lora_scale=1.5) for s in (1, -2)]
    torch.cuda.synchronize()
    if trained:
        fa, fb = (torch.nn.Parameter(t.clone()) for t in (a, b))
    got = []
    for i in range(100):
        s = (1, -2)[i % 2]
        if trained:
            with torch.no_grad():
                torch.mul(a, s, out=fa.data)
                torch.mul(b, s, out=fb.data)
        else:
            fa, fb = (a * s).float(), (b * s).float()
        got.append(linear_forward(x, p, k, n, layout, lora_a=fa, lora_b=fb, lora_scale=1.5))
    assert all(torch.equal(y, want[i % 2]) for i, y in enumerate(got))


def test_the_workspace_unused_longest_goes_first():
    # sixteen are kept: a call on a seventeenth stream displaces the one whose last use is furthest back
    x, p, k, n, layout, a, b = layers()[0]
    out = torch.empty(x.shape[0], n, dtype=x.dtype, device=DEV)
    streams, seen = [], set()
    while len(streams) < 17:  # (torch hands its pool's streams out in turn)
        s = torch.cuda.Stream()
        if s.cuda_stream not in seen:
            seen.add(s.cuda_stream)
            streams.append(s)

    def allocations(stream):
        from unifur_b200.quantize import linear_forward

        before = torch.cuda.memory_stats()["allocation.all.allocated"]
        with torch.cuda.stream(stream):
            linear_forward(x, p, k, n, layout, lora_a=a, lora_b=b, lora_scale=1.5, out=out)
        torch.cuda.synchronize()
        return torch.cuda.memory_stats()["allocation.all.allocated"] - before

    _lib.host().release_workspaces()
    assert [allocations(s) for s in streams[:16]] == [1] * 16
    assert allocations(streams[0]) == 0                     # the oldest entry becomes the newest
    assert allocations(streams[16]) == 1                    # displaces streams[1]'s
    assert [allocations(s) for s in (streams[0], *streams[2:])] == [0] * 16
    assert allocations(streams[1]) == 1
    _lib.host().release_workspaces()


def test_forward_under_capture_replays_beside_eager_calls():
    c = layers()[0]
    want = forward(*c)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        y = forward(*c)
    for _ in range(3):
        g.replay()
        again = forward(*c)
    torch.cuda.synchronize()
    assert torch.equal(y, want) and torch.equal(again, want)


@pytest.mark.parametrize("rows,k,n,r", [
    (1, 256, 16, 0),         # one CTA fetches x and is the last as well
    (16, 20480, 1024, 8),    # more of x than the first CTAs fetch at a time, K in parts
    (3, 4352, 96, 16),
    (5, 320, 192, 8),        # d_in the kernel does not fetch for: copies and the stream's synchronise
])
def test_page_locked_calls_give_the_same_bits(rows, k, n, r):
    # x fetched by the kernel and its word to the host, against copies of pageable memory; new values every call, from two
    # threads at a time
    import ctypes
    import threading

    from unifur_b200.quantize import PackedNf4Tensor

    L, g = _lib.load(), torch.Generator(device="cuda").manual_seed(k + n)
    p = PackedNf4Tensor.quantize(torch.randn(k * n, device="cuda", generator=g) * 0.02)
    codes, absmax = p.codes.cpu(), p.absmax.cpu()
    a, b = (torch.randn(*s, device="cuda", generator=g).bfloat16().cpu() * 0.05 for s in ((max(r, 1), k), (n, max(r, 1))))
    h = ctypes.c_void_p()
    _lib.check(L.nf4_weight_from_packed_host(codes.data_ptr(), absmax.data_ptr(), None, 0.0, k, n, _lib.LAYOUT_OUT_IN, ctypes.byref(h)))
    if r:
        _lib.check(L.nf4_weight_attach_lora_host(h, a.data_ptr(), b.data_ptr(), r, 1.5, _lib.DTYPE_BF16))
    call = lambda x, y: _lib.check(L.nf4_weight_linear_forward_host(  # noqa: E731
        h, x.data_ptr(), rows, _lib.DTYPE_BF16, None, None, None, 0, 0.0, y.data_ptr()))
    wrong = []

    def work(seed):
        gen = torch.Generator().manual_seed(seed)
        xl, yl = torch.empty(rows, k, dtype=torch.bfloat16).pin_memory(), torch.empty(rows, n, dtype=torch.bfloat16).pin_memory()
        for _ in range(25):
            x, y = torch.randn(rows, k, generator=gen).bfloat16(), torch.empty(rows, n, dtype=torch.bfloat16)
            xl.copy_(x)
            yl.fill_(7.0)
            call(xl, yl)
            got = yl.clone()
            call(x, y)
            if not torch.equal(got, y):
                wrong.append(seed)

    try:
        threads = [threading.Thread(target=work, args=(s,)) for s in (1, 2)]
        [t.start() for t in threads]
        [t.join() for t in threads]
        assert not wrong
    finally:
        L.nf4_weight_free(h)


def test_a_host_call_behind_the_kernel_that_writes_its_x():
    # Stream order holds on the stream the host calls work on: a forward there writes page-locked memory, and the host
    # call that takes it as x follows without a synchronise.  Forwards of few CTAs ahead, so that the host call's could start
    # beside them; the one right ahead writes other values every time.
    import ctypes

    from unifur_b200.quantize import PackedNf4Tensor

    L, g, bf16 = _lib.load(), torch.Generator(device="cuda").manual_seed(3), torch.bfloat16
    rows, k0, k, n = 16, 4096, 256, 512
    first, second = (PackedNf4Tensor.quantize(torch.randn(a * b, device="cuda", generator=g) * 0.02) for a, b in ((k0, k), (k, n)))
    codes, absmax = second.codes.cpu(), second.absmax.cpu()
    h = ctypes.c_void_p()
    _lib.check(L.nf4_weight_from_packed_host(codes.data_ptr(), absmax.data_ptr(), None, 0.0, k, n, _lib.LAYOUT_OUT_IN, ctypes.byref(h)))
    xs = [torch.randn(rows, k0, device="cuda", generator=g).to(bf16) for _ in range(2)]
    mid, y = torch.empty(rows, k, dtype=bf16).pin_memory(), torch.empty(rows, n, dtype=bf16).pin_memory()
    per_thread = ctypes.c_void_p(2)  # cudaStreamPerThread
    scratch = torch.zeros(L.nf4_linear_workspace_bytes(rows, k0, k, 0), dtype=torch.uint8, device="cuda")

    def ahead(x):
        a = _lib.LinearArgs(struct_bytes=ctypes.sizeof(_lib.LinearArgs), layout=_lib.LAYOUT_OUT_IN, io_dtype=_lib.DTYPE_BF16, rows=rows,
                            d_in=k0, d_out=k, x=x.data_ptr(), packed=first.codes.data_ptr(), absmax=first.absmax.data_ptr(),
                            y=mid.data_ptr(), ldy=k, workspace=scratch.data_ptr(), workspace_bytes=scratch.numel())
        _lib.check(L.nf4_linear_forward_dev(ctypes.byref(a), per_thread))

    def host():
        _lib.check(L.nf4_weight_linear_forward_host(h, mid.data_ptr(), rows, _lib.DTYPE_BF16, None, None, None, 0, 0.0, y.data_ptr()))
        return y.clone()

    torch.cuda.synchronize()
    try:
        want = []
        for x in xs:
            ahead(x)
            torch.cuda.synchronize()
            want.append(host())
        assert not torch.equal(*want)
        for i in range(60):
            for j in range(7):
                ahead(xs[(i + j) % 2])  # (the last one's x: i % 2)
            assert torch.equal(host(), want[i % 2])
    finally:
        L.nf4_weight_free(h)


BLOCKING_CHILD = """
import ctypes, sys, time
drv = ctypes.CDLL("libcuda.so.1")
assert drv.cuInit(0) == 0 and drv.cuDevicePrimaryCtxSetFlags_v2(0, int(sys.argv[1])) == 0
import torch
from unifur_b200 import _lib
L, rows, k, n = _lib.load(), 4, 512, 256
codes, absmax = torch.zeros(k * n // 2, dtype=torch.uint8), torch.ones(k * n // 64)
h = ctypes.c_void_p()
torch.cuda.init()
_lib.check(L.nf4_weight_from_packed_host(codes.data_ptr(), absmax.data_ptr(), None, 0.0, k, n, _lib.LAYOUT_OUT_IN, ctypes.byref(h)))
x, y = torch.ones(rows, k, dtype=torch.bfloat16).pin_memory(), torch.empty(rows, n, dtype=torch.bfloat16).pin_memory()
call = lambda: _lib.check(L.nf4_weight_linear_forward_host(h, x.data_ptr(), rows, _lib.DTYPE_BF16, None, None, None, 0, 0.0, y.data_ptr()))
call()
with torch.cuda.stream(torch.cuda.ExternalStream(2)):  # the calls' stream has a tenth of a second to do first
    torch.cuda._sleep(200_000_000)
wall, cpu = time.perf_counter(), time.thread_time()
call()
print(time.perf_counter() - wall, time.thread_time() - cpu, bool((y == -k).all()))
"""


@pytest.mark.parametrize("schedule", [2, 4])  # CU_CTX_SCHED_YIELD, CU_CTX_SCHED_BLOCKING_SYNC
def test_a_waiting_host_call_waits_as_the_process_chose(schedule):
    # page-locked buffers, so that the call's kernel has a word for the host: it is polled only where nothing was chosen
    import subprocess
    import sys

    out = subprocess.run([sys.executable, "-c", BLOCKING_CHILD, str(schedule)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    wall, cpu, right = out.stdout.split()
    assert right == "True" and float(wall) > 0.05
    if schedule == 4:
        assert float(cpu) < 0.2 * float(wall)  # (a poll takes all of it)
