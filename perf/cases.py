"""The work that users of this package have it do, as cases whose speed can be measured.

A case names one kind of call with its sizes and options:

  linear      ``Nf4Linear.forward`` / ``QloraLinear.forward``: one projection, at decode sizes (a few rows) and
              prefill sizes, in either weight orientation and tensor type
  block       the seven projections of a decoder layer for one decode step, those that share an input as one call
  host        the C ABI's host-pointer forward on a resident weight: what a host without device memory of its own calls
  backward    ``QloraLinear.backward``: an adapter's training step through a frozen weight
  round_trip  ``PackedNf4Tensor.quantize`` (and ``with_double_quantization``) and ``dequantize``
  checkpoint  ``Nf4Linear.from_checkpoint``: a checkpoint's matrix to the resident weight
  embedding   ``Nf4Embedding.forward``: the rows of a quantized table that token ids select

Everything goes through the package's public entry points.  ``listed`` holds the cases by name, ``draw`` gives more
of the same ranges.
"""
import ctypes
import math

import torch

from unifur_b200 import _lib
from unifur_b200._lib import LAYOUT_IN_OUT, LAYOUT_OUT_IN
from unifur_b200.quantize import PackedNf4Tensor, linear_forward, linear_forward_grouped
from unifur_b200.qwennet import Nf4Embedding, Nf4Linear, QloraLinear

DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}
LAYOUTS = {"out_in": LAYOUT_OUT_IN, "in_out": LAYOUT_IN_OUT}
BLOCK = 64                      # values per quantization block
MOST_MACS = 2048 * 4096 * 14336  # rows * d_in * d_out of the largest listed forward and backward


def linear(rows, d_in, d_out, rank, layout="out_in", dtype="bf16", double=False, bias=False):
    return {"kind": "linear", "rows": rows, "d_in": d_in, "d_out": d_out, "rank": rank, "layout": layout, "dtype": dtype,
            "double": double, "bias": bias}


def listed():
    return [
        # the smallest projection of a decode step: k or v of a grouped-query layer, one sequence
        dict(linear(1, 3584, 512, 16), name="decode_kv"),
        # the decode layer that bench.py's metric is quoted on, four sequences
        dict(linear(4, 4096, 11008, 16), name="decode_up"),
        # a decode step of eight sequences through the seven projections of the Qwen2-7B-shaped block
        {"name": "decode_block", "kind": "block", "rows": 8, "hidden": 3584, "kv": 512, "inter": 18944, "rank": 16},
        # the same decode layer as the reference stores and calls it: f32 tensors, W [d_in, d_out], u8 scales, no adapter
        dict(linear(1, 4096, 11008, 0, layout="in_out", dtype="f32", double=True), name="decode_reference"),
        # a host that holds host memory only: page-locked activations in, page-locked results out
        {"name": "decode_host", "kind": "host", "rows": 4, "d_in": 4096, "d_out": 11008, "rank": 16},
        # prefill of 2048 tokens, rank-64 adapter
        dict(linear(2048, 4096, 14336, 64), name="prefill_up"),
        # a short prompt: no multiple of any tile, u8 scales, a bias
        dict(linear(203, 3584, 18944, 16, double=True, bias=True), name="prefill_short"),
        # a prompt through a layer stored and called as the reference does it
        dict(linear(512, 4096, 4096, 16, layout="in_out", dtype="f32", double=True), name="prefill_reference"),
        # a training step's backward through the prefill layer
        {"name": "backward_up", "kind": "backward", "rows": 2048, "d_in": 4096, "d_out": 14336, "rank": 64, "layout": "out_in",
         "dtype": "bf16", "double": False},
        # one weight matrix quantized and reconstructed
        {"name": "round_trip", "kind": "round_trip", "len": 4096 * 4096, "double": False, "heavy": False},
        # loading: a checkpoint's bf16 matrix to a resident weight with double quantization
        {"name": "load_up", "kind": "checkpoint", "rows": 14336, "cols": 4096, "dtype": "bf16"},
        # 4096 token ids out of a vocabulary-sized table
        {"name": "embed_prompt", "kind": "embedding", "n": 151936, "d_model": 3584, "ids": 4096, "dtype": "bf16"},
    ]


def _spread(rng, low, high, step=1):
    """A size of [low, high], even over its logarithm, a multiple of `step`."""
    v = math.exp(rng.uniform(math.log(low), math.log(high)))
    return min(max(int(round(v / step)), -(-low // step)), high // step) * step


def _dim(rng, low=256, high=20480):
    """A model dimension: whole quantization blocks, most often a multiple of 256."""
    return _spread(rng, low, high, rng.choice((256, 256, 64)))


def draw(rng):
    kind = rng.choice(("decode", "decode", "prefill", "prefill", "block", "host", "backward", "round_trip", "checkpoint",
                       "embedding"))
    if kind in ("decode", "prefill"):
        layout, dtype = rng.choice((("out_in", "bf16"), ("out_in", "bf16"), ("in_out", "f32"), ("in_out", "bf16"),
                                    ("out_in", "f32")))
        d_in, d_out = _dim(rng), _dim(rng)
        most = max(17, min(4096, MOST_MACS // (d_in * d_out)))
        rows = rng.randint(1, 16) if kind == "decode" else _spread(rng, 17, most)
        return linear(rows, d_in, d_out, rng.choice((0, 8, 16, 32, 64)), layout, dtype, rng.random() < 0.5, rng.random() < 0.25)
    if kind == "block":
        hidden = _spread(rng, 1024, 5120, 256)
        return {"kind": "block", "rows": rng.randint(1, 16), "hidden": hidden, "kv": rng.choice((256, 512, 1024)),
                "inter": int(hidden * rng.uniform(2.6, 5.3)) // 256 * 256, "rank": rng.choice((8, 16, 32))}
    if kind == "host":
        return {"kind": "host", "rows": rng.randint(1, 16), "d_in": _dim(rng), "d_out": _dim(rng), "rank": rng.choice((0, 8, 16, 32))}
    if kind == "backward":
        d_in, d_out = _dim(rng), _dim(rng)
        layout, dtype = rng.choice((("out_in", "bf16"), ("in_out", "bf16"), ("in_out", "f32")))
        return {"kind": "backward", "rows": _spread(rng, 1, max(1, min(4096, MOST_MACS // (d_in * d_out)))), "d_in": d_in,
                "d_out": d_out, "rank": rng.choice((8, 16, 32, 64)), "layout": layout, "dtype": dtype, "double": rng.random() < 0.5}
    if kind == "round_trip":
        return {"kind": "round_trip", "len": _spread(rng, 4096, 14336 * 4096), "double": rng.random() < 0.5,
                "heavy": rng.random() < 0.5}
    if kind == "checkpoint":
        return {"kind": "checkpoint", "rows": _dim(rng, 256, 14336), "cols": _dim(rng, 256, 14336), "dtype": rng.choice(("bf16", "f32"))}
    return {"kind": "embedding", "n": _spread(rng, 32000, 151936), "d_model": _dim(rng, 512, 5120), "ids": _spread(rng, 1, 8192),
            "dtype": rng.choice(("bf16", "f32"))}


# ---- inputs -----------------------------------------------------------------------------------


class _Inputs:
    """Seeded tensors on the GPU with the distributions of bench.py's configurations."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, *shape, std=1.0, dtype=torch.float32):
        return (torch.randn(*shape, device="cuda", generator=self.gen) * std).to(dtype)

    def weights(self, *shape, heavy=False):
        """N(0, 0.02^2), or Student-t(4) * 0.02: outlier blocks."""
        z = self.normal(*shape, std=0.02)
        if heavy:
            chi = torch.zeros_like(z)
            for _ in range(4):
                chi += self.normal(*shape) ** 2
            z /= torch.sqrt(chi / 4)
        return z

    def packed(self, d_in, d_out, double):
        p = PackedNf4Tensor.quantize(self.weights(d_in * d_out))
        return p.with_double_quantization() if double else p

    def factors(self, d_in, d_out, rank, layout, dtype):
        a, b = ((rank, d_in), (d_out, rank)) if layout == "out_in" else ((d_in, rank), (rank, d_out))
        return self.normal(*a, std=0.01, dtype=DTYPES[dtype]), self.normal(*b, std=0.01, dtype=DTYPES[dtype])

    def layer(self, d_in, d_out, rank, layout, dtype, double=False, bias=False):
        base = Nf4Linear.from_packed(self.packed(d_in, d_out, double), d_in, d_out,
                                     self.normal(d_out) if bias else None, LAYOUTS[layout])
        return QloraLinear(base, *self.factors(d_in, d_out, rank, layout, dtype), 2.0) if rank else base


class _HostLayer:
    """A resident weight with its adapter and the host's page-locked buffers."""

    def __init__(self, inp, c):
        rows, d_in, d_out, rank = c["rows"], c["d_in"], c["d_out"], c["rank"]
        self.lib, self.rows = _lib.load(), rows
        p = inp.packed(d_in, d_out, False)
        codes, absmax = p.codes.cpu(), p.absmax.cpu()
        self.handle = ctypes.c_void_p()
        _lib.check(self.lib.nf4_weight_from_packed_host(codes.data_ptr(), absmax.data_ptr(), None, 0.0, d_in, d_out, LAYOUT_OUT_IN,
                                                        ctypes.byref(self.handle)))
        if rank:
            a, b = (t.cpu() for t in inp.factors(d_in, d_out, rank, "out_in", "bf16"))
            _lib.check(self.lib.nf4_weight_attach_lora_host(self.handle, a.data_ptr(), b.data_ptr(), rank, 2.0, _lib.DTYPE_BF16))
        self.x = inp.normal(rows, d_in, dtype=torch.bfloat16).cpu().pin_memory()
        self.y = torch.empty(rows, d_out, dtype=torch.bfloat16).pin_memory()

    def forward(self):
        _lib.check(self.lib.nf4_weight_linear_forward_host(self.handle, self.x.data_ptr(), self.rows, _lib.DTYPE_BF16, None, None,
                                                           None, 0, 0.0, self.y.data_ptr()))
        return self.y

    def __del__(self):
        self.lib.nf4_weight_free(self.handle)


def _block_shapes(c):
    h, kv, inter = c["hidden"], c["kv"], c["inter"]
    return {"q": (h, h), "k": (h, kv), "v": (h, kv), "o": (h, h), "gate": (h, inter), "up": (h, inter), "down": (inter, h)}


def prepare(case, seed):
    c, inp = case, _Inputs(seed)
    kind = c["kind"]
    if kind == "linear":
        return {"kind": kind, "layer": inp.layer(c["d_in"], c["d_out"], c["rank"], c["layout"], c["dtype"], c["double"], c["bias"]),
                "x": inp.normal(c["rows"], c["d_in"], dtype=DTYPES[c["dtype"]])}
    if kind == "block":
        s = {"kind": kind, "hidden": c["hidden"], "inter": c["inter"]}
        for name, (d_in, d_out) in _block_shapes(c).items():
            a, b = inp.factors(d_in, d_out, c["rank"], "out_in", "bf16")
            s[name] = {"packed": inp.packed(d_in, d_out, False), "d_out": d_out, "lora_a": a, "lora_b": b, "lora_scale": 2.0}
        for name, width in (("x", "hidden"), ("attn", "hidden"), ("x2", "hidden"), ("act", "inter")):
            s[name] = inp.normal(c["rows"], c[width], dtype=torch.bfloat16)
        return s
    if kind == "host":
        return {"kind": kind, "layer": _HostLayer(inp, c)}
    if kind == "backward":
        return {"kind": kind, "layer": inp.layer(c["d_in"], c["d_out"], c["rank"], c["layout"], c["dtype"], c["double"]),
                "x": inp.normal(c["rows"], c["d_in"], dtype=DTYPES[c["dtype"]]),
                "grad_y": inp.normal(c["rows"], c["d_out"], std=1e-3, dtype=DTYPES[c["dtype"]])}
    if kind == "round_trip":
        return {"kind": kind, "values": inp.weights(c["len"], heavy=c["heavy"]), "double": c["double"]}
    if kind == "checkpoint":
        return {"kind": kind, "weight": inp.weights(c["rows"], c["cols"]).to(DTYPES[c["dtype"]])}
    table = Nf4Embedding.from_values(inp.weights(c["n"] * c["d_model"]), c["n"], c["d_model"])
    ids = torch.randint(0, c["n"], (c["ids"],), device="cuda", generator=inp.gen)
    return {"kind": kind, "table": table, "ids": ids, "dtype": DTYPES[c["dtype"]]}


def _stored(p):
    return [p.codes, p.scale_codes, p.scale_of_scales] if p.is_double_quantized() else [p.codes, p.absmax]


def run(state):
    s, kind = state, state["kind"]
    if kind == "linear":
        return s["layer"].forward(s["x"])
    if kind == "block":
        h, out_in = s["hidden"], LAYOUT_OUT_IN
        q, k, v = linear_forward_grouped(s["x"], h, out_in, [s["q"], s["k"], s["v"]])
        o = linear_forward(s["attn"], s["o"]["packed"], h, s["o"]["d_out"], out_in, lora_a=s["o"]["lora_a"],
                           lora_b=s["o"]["lora_b"], lora_scale=s["o"]["lora_scale"])
        gate, up = linear_forward_grouped(s["x2"], h, out_in, [s["gate"], s["up"]])
        down = linear_forward(s["act"], s["down"]["packed"], s["inter"], s["down"]["d_out"], out_in, lora_a=s["down"]["lora_a"],
                              lora_b=s["down"]["lora_b"], lora_scale=s["down"]["lora_scale"])
        return [q, k, v, o, gate, up, down]
    if kind == "host":
        return s["layer"].forward()
    if kind == "backward":
        return list(s["layer"].backward(s["x"], s["grad_y"]))
    if kind == "round_trip":
        p = PackedNf4Tensor.quantize(s["values"])
        if s["double"]:
            p = p.with_double_quantization()
        return _stored(p) + [p.dequantize()]
    if kind == "checkpoint":
        return _stored(Nf4Linear.from_checkpoint(s["weight"]).packed())
    return s["table"].forward(s["ids"], s["dtype"])


# ---- what a pass cannot do without --------------------------------------------------------------


def _weight_bytes(n, double):
    blocks = -(-n // BLOCK)
    return -(-n // 2) + (blocks + 4 if double else 4 * blocks)


def _linear_work(rows, d_in, d_out, rank, esize, double=False, bias=False):
    return {"bytes": _weight_bytes(d_in * d_out, double) + esize * (rows * (d_in + d_out) + rank * (d_in + d_out)) + 4 * d_out * bias,
            "flops": 2 * rows * (d_in * d_out + rank * (d_in + d_out))}


def work(case):
    c, kind = case, case["kind"]
    esize = 4 if c.get("dtype") == "f32" else 2
    if kind == "linear":
        return _linear_work(c["rows"], c["d_in"], c["d_out"], c["rank"], esize, c["double"], c["bias"])
    if kind == "block":
        parts = [_linear_work(c["rows"], d_in, d_out, c["rank"], 2) for d_in, d_out in _block_shapes(c).values()]
        shared = 2 * c["rows"] * 3 * c["hidden"]  # k and v read q's input again, up gate's
        return {"bytes": sum(p["bytes"] for p in parts) - shared, "flops": sum(p["flops"] for p in parts)}
    if kind == "host":
        return _linear_work(c["rows"], c["d_in"], c["d_out"], c["rank"], 2)
    if kind == "backward":
        rows, d_in, d_out, r = c["rows"], c["d_in"], c["d_out"], c["rank"]
        # x, grad_y and the factors in, the three gradients out; grad_x, and the adapter's five rank-r products
        return {"bytes": _weight_bytes(d_in * d_out, c["double"]) + esize * (rows * (2 * d_in + d_out) + 2 * r * (d_in + d_out)),
                "flops": 2 * rows * (d_in * d_out + r * (3 * d_in + 2 * d_out))}
    if kind == "round_trip":
        return {"bytes": 8 * c["len"] + 2 * _weight_bytes(c["len"], c["double"]), "flops": 0}
    if kind == "checkpoint":
        n = c["rows"] * c["cols"]
        return {"bytes": esize * n + _weight_bytes(n, True), "flops": 0}
    n = c["ids"] * c["d_model"]
    return {"bytes": 8 * c["ids"] + _weight_bytes(n, True) + esize * n, "flops": 0}


def tolerance(case):
    c, kind = case, case["kind"]
    if kind in ("round_trip", "checkpoint", "embedding"):
        return "exact"
    if kind == "linear" and c["dtype"] == "f32":
        # up to 16 rows of the reference's orientation are f32 throughout; the other f32 paths multiply in f16 with
        # f32 sums, which the C header bounds by 1e-3
        return {"rel": 1e-5 if c["layout"] == "in_out" and c["rows"] <= 16 else 1e-3}
    if kind == "backward" and c["dtype"] == "f32":
        return {"rel": 1e-3}
    return {"rel": 5e-3}  # bf16 results
