// Host path of the Python mirror: the tensor side of one call (type conversions, outputs, workspace,
// argument block, current stream) in C++ over the C ABI.
//
// Why native.  A decode-sized forward is 5 to 10 us of GPU work; assembling its argument block from
// Python (two dozen ctypes fields, a device guard, three allocations and a fill kernel for the flag
// words) took 27 to 29 us, so every small call was bound by the interpreter (decode_block: 188 us of
// host work for 70 us of kernels).  Here a call costs about as much as its launch.
//
// Workspaces.  The decode and strip kernels meet on flag words at the start of the workspace that
// must be zero at first use and are left zero, by calls whose waits gave up too.  A fresh workspace would need a fill kernel in front
// of every call, which also breaks the overlap of a call's prologue with the call before it.  So a
// host thread keeps the last kKeptMost workspaces it used, of at most kKeptBytes each, by stream
// (calls on one stream are ordered; two threads never share one).  They live in torch's caching
// allocator and go back to it when others have been used since, when the thread ends, and by
// release_workspaces().  Larger workspaces, and calls under stream capture (whose replays may run on
// any stream later), are allocated per call.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/core/LegacyTypeDispatch.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cstring>
#include <optional>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../../include/nf4_b200.h"

namespace {

using at::Tensor;

// ---- errors ---------------------------------------------------------------------------------
struct PyFail {};  // a Python error has been set

[[noreturn]] void raise(PyObject *type, const char *msg) {
    PyErr_SetString(type, msg);
    throw PyFail{};
}

// A non-zero status becomes unifur_b200._lib.Nf4Error, as in the ctypes binding.
void check(int32_t status) {
    if (status == NF4_OK) return;
    PyObject *mod = PyImport_ImportModule("unifur_b200._lib");
    PyObject *cls = mod ? PyObject_GetAttrString(mod, "Nf4Error") : nullptr;
    PyObject *exc = cls ? PyObject_CallFunction(cls, "is", (int)status, nf4_last_error()) : nullptr;
    if (exc) PyErr_SetObject(cls, exc);
    Py_XDECREF(exc);
    Py_XDECREF(cls);
    Py_XDECREF(mod);
    throw PyFail{};
}

template <class F>
PyObject *guarded(F f) {
    try {
        // nothing here is differentiable: outputs are plain tensors, as the ctypes binding made them
        at::AutoDispatchBelowADInplaceOrView below_autograd;
        return f();
    } catch (const PyFail &) {
    } catch (const c10::Error &e) {
        const bool oom = dynamic_cast<const c10::OutOfMemoryError *>(&e) != nullptr;
        PyObject *type = PyExc_RuntimeError;
        if (oom) {
            PyObject *torch = PyImport_ImportModule("torch");
            PyObject *cls = torch ? PyObject_GetAttrString(torch, "OutOfMemoryError") : nullptr;
            if (cls) type = cls;
            PyErr_Clear();
            Py_XDECREF(torch);
        }
        PyErr_SetString(type, e.what_without_backtrace());
    } catch (const std::exception &e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}

// ---- arguments ------------------------------------------------------------------------------
const Tensor &tensor(PyObject *o) {
    if (!THPVariable_Check(o)) raise(PyExc_TypeError, "expected a torch tensor");
    return THPVariable_Unpack(o);
}
const Tensor *tensor_or_none(PyObject *o) { return o == Py_None ? nullptr : &tensor(o); }

uint64_t size_arg(PyObject *o) {
    const unsigned long long v = PyLong_AsUnsignedLongLong(o);
    if (v == (unsigned long long)-1 && PyErr_Occurred()) throw PyFail{};
    return v;
}
double float_arg(PyObject *o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw PyFail{};
    return v;
}
void expect(Py_ssize_t n, Py_ssize_t want) {
    if (n != want) raise(PyExc_TypeError, "wrong number of arguments");
}

int32_t io_dtype(at::ScalarType t) {
    if (t == at::kBFloat16) return NF4_DTYPE_BF16;
    if (t == at::kFloat) return NF4_DTYPE_F32;
    raise(PyExc_TypeError, (std::string("activations must be bf16 or f32, got ") + c10::toString(t)).c_str());
}

void require_cuda(const Tensor &t, const char *what) {
    if (!t.is_cuda())
        raise(PyExc_ValueError, (std::string(what) + " must live on a CUDA device (this package has no CPU path)").c_str());
}

Tensor as_type(const Tensor &t, at::ScalarType type) {
    return (t.scalar_type() == type ? t : t.to(type)).contiguous();
}

template <class T>
const T *ptr_as(const Tensor *t) { return t ? static_cast<const T *>(t->const_data_ptr()) : nullptr; }

// ---- device, stream, memory -----------------------------------------------------------------
struct Place {
    c10::cuda::CUDAGuard guard;
    c10::Device device;
    cudaStream_t stream;
    explicit Place(c10::Device d) : guard(d), device(d), stream(c10::cuda::getCurrentCUDAStream(d.index()).stream()) {}
};

Tensor empty(at::IntArrayRef shape, at::ScalarType type, const Place &at_) {
    return at::detail::empty_cuda(shape, type, at_.device, std::nullopt);
}

bool capturing(cudaStream_t s) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(s, &st) == cudaSuccess && st != cudaStreamCaptureStatusNone;
}

void zero_flags(const Tensor &ws, const Place &at_) {
    if (cudaMemsetAsync(ws.mutable_data_ptr(), 0, 256, at_.stream) != cudaSuccess)
        throw std::runtime_error("clearing the workspace's flag words failed");
}

constexpr size_t kKeptBytes = 16u << 20;
constexpr size_t kKeptMost = 16;
struct Kept {
    int device;
    cudaStream_t stream;
    uint32_t slot;
    Tensor ws;
};
thread_local std::vector<Kept> t_kept;  // most recently used last

// `bytes` of scratch whose first 256 bytes are zero.  `slot`: which of a call's workspaces (the
// projections of a grouped call have one each).
Tensor flagged_workspace(uint64_t bytes, const Place &at_, uint32_t slot) {
    if (bytes < 256) bytes = 256;
    if (bytes > kKeptBytes || capturing(at_.stream)) {
        Tensor ws = empty({(int64_t)bytes}, at::kByte, at_);
        zero_flags(ws, at_);
        return ws;
    }
    const int dev = at_.device.index();
    for (size_t i = t_kept.size(); i-- > 0;) {
        if (t_kept[i].device != dev || t_kept[i].stream != at_.stream || t_kept[i].slot != slot) continue;
        if ((uint64_t)t_kept[i].ws.numel() >= bytes) {
            std::rotate(t_kept.begin() + (long)i, t_kept.begin() + (long)i + 1, t_kept.end());
            return t_kept.back().ws;
        }
        t_kept.erase(t_kept.begin() + (long)i);  // too small: replaced by a larger one below
        break;
    }
    if (t_kept.size() >= kKeptMost) t_kept.erase(t_kept.begin());
    uint64_t cap = 1u << 16;
    while (cap < bytes) cap <<= 1;
    Tensor ws = empty({(int64_t)cap}, at::kByte, at_);
    zero_flags(ws, at_);
    t_kept.push_back(Kept{dev, at_.stream, slot, ws});
    return ws;
}

PyObject *pair(Tensor a, Tensor b) {
    return Py_BuildValue("NN", THPVariable_Wrap(std::move(a)), THPVariable_Wrap(std::move(b)));
}

// Runs one C-ABI call without the interpreter lock (a launch can wait for room in the queue).
template <class F>
int32_t unlocked(F f) {
    PyThreadState *st = PyEval_SaveThread();
    const int32_t rc = f();
    PyEval_RestoreThread(st);
    return rc;
}

// ---- forward --------------------------------------------------------------------------------
// One projection's operands as they come from Python; the converted ones are held until the launch
// is enqueued (torch's allocator keeps freed memory on the stream, so the kernels may still run).
struct Projection {
    const Tensor *codes, *absmax, *scale_codes, *scale_of_scales;
    uint64_t d_out;
    Tensor bias, a, b;
    float scale;
    bool just_written;  // the factors: by a conversion here, or perhaps by the optimizer that trains them
};

Projection projection(PyObject *const *v, at::ScalarType type) {
    // codes, absmax, scale_codes, scale_of_scales, d_out, bias, lora_a, lora_b, lora_scale
    Projection p;
    p.codes = &tensor(v[0]);
    p.scale_codes = tensor_or_none(v[2]);
    p.absmax = p.scale_codes ? nullptr : tensor_or_none(v[1]);
    p.scale_of_scales = tensor_or_none(v[3]);
    p.d_out = size_arg(v[4]);
    p.just_written = false;
    if (const Tensor *t = tensor_or_none(v[5])) p.bias = as_type(*t, at::kFloat);
    if (const Tensor *t = tensor_or_none(v[6])) {
        const Tensor &b = tensor(v[7]);
        p.a = as_type(*t, type);
        p.b = as_type(b, type);
        p.just_written = !p.a.is_same(*t) || !p.b.is_same(b) || t->requires_grad() || b.requires_grad();
    }
    p.scale = (float)float_arg(v[8]);
    return p;
}
constexpr Py_ssize_t kProjectionArgs = 9;

uint32_t rank_of(const Projection &p, int32_t layout) {
    return p.a.defined() ? (uint32_t)p.a.size(layout == NF4_LAYOUT_OUT_IN ? 0 : 1) : 0;
}

nf4_linear_args linear_args(const Tensor &x, uint64_t rows, uint64_t d_in, int32_t layout, const Projection &p) {
    nf4_linear_args a;
    std::memset(&a, 0, sizeof(a));
    a.struct_bytes = sizeof(a);
    a.layout = layout;
    a.io_dtype = io_dtype(x.scalar_type());
    a.rows = rows;
    a.d_in = d_in;
    a.d_out = p.d_out;
    a.x = x.const_data_ptr();
    a.packed = ptr_as<uint8_t>(p.codes);
    a.absmax = ptr_as<float>(p.absmax);
    a.scale_codes = ptr_as<uint8_t>(p.scale_codes);
    a.scale_of_scales = ptr_as<float>(p.scale_codes ? p.scale_of_scales : nullptr);
    a.bias = p.bias.defined() ? ptr_as<float>(&p.bias) : nullptr;
    if (p.a.defined()) {
        a.lora_a = p.a.const_data_ptr();
        a.lora_b = p.b.const_data_ptr();
        a.lora_rank = rank_of(p, layout);
    }
    a.lora_scale = p.scale;
    return a;
}

// x with its leading dimensions flattened (src/qwennet.rs:326-342)
struct Rows {
    Tensor x;
    uint64_t rows;
    std::vector<int64_t> shape;
    void widen(uint64_t from, uint64_t to) {  // the shape with its last dimension replaced
        if ((uint64_t)shape.back() != from) raise(PyExc_RuntimeError, "the last dimension of x is not d_in");
        shape.back() = (int64_t)to;
    }
};
Rows flatten(const Tensor &x, uint64_t d_in) {
    require_cuda(x, "x");
    Rows r{x.contiguous(), 0, x.sizes().vec()};
    if (d_in == 0 || r.shape.empty() || x.numel() % (int64_t)d_in != 0)
        raise(PyExc_RuntimeError, "x does not hold whole rows of d_in values");
    r.rows = (uint64_t)x.numel() / d_in;
    return r;
}

// `bytes` of scratch whose first `flags` bytes have to be zero.  The kernels that meet on flag words take the
// adapter's factors for constants, like the weight: they ask for them before the kernel ahead has completed.  One
// that has just written them would have to publish them for that, which torch's do not: a fill of the
// (zero) flag words between the two keeps them apart.
Tensor workspace(uint64_t bytes, uint64_t flags, const Projection &p, const Place &at_, uint32_t slot = 0) {
    if (!flags) return empty({(int64_t)(bytes < 256 ? 256 : bytes)}, at::kByte, at_);
    Tensor ws = flagged_workspace(bytes, at_, slot);
    if (p.just_written) zero_flags(ws, at_);
    return ws;
}
Tensor forward_workspace(const nf4_linear_args &a, const Projection &p, const Place &at_, uint32_t slot = 0) {
    return workspace(nf4_linear_workspace_bytes(a.rows, a.d_in, a.d_out, a.lora_rank), nf4_linear_flag_bytes(&a), p, at_, slot);
}

// linear_forward(x, d_in, layout, <projection>, out)
PyObject *linear_forward(PyObject *, PyObject *const *v, Py_ssize_t n) {
    return guarded([&]() -> PyObject * {
        expect(n, 3 + kProjectionArgs + 1);
        const uint64_t d_in = size_arg(v[1]);
        const int32_t layout = (int32_t)size_arg(v[2]);
        Rows r = flatten(tensor(v[0]), d_in);
        Place place(r.x.device());
        const Projection p = projection(v + 3, r.x.scalar_type());
        nf4_linear_args a = linear_args(r.x, r.rows, d_in, layout, p);
        const Tensor *out = tensor_or_none(v[3 + kProjectionArgs]);
        if (!out) r.widen(d_in, p.d_out);
        Tensor y = out ? *out : empty(r.shape, r.x.scalar_type(), place);
        a.y = y.mutable_data_ptr();
        a.ldy = out ? (uint64_t)out->stride(0) : p.d_out;
        const Tensor ws = forward_workspace(a, p, place);
        a.workspace = ws.mutable_data_ptr();
        a.workspace_bytes = (uint64_t)ws.numel();
        check(unlocked([&] { return nf4_linear_forward_dev(&a, place.stream); }));
        return THPVariable_Wrap(std::move(y));
    });
}

// linear_forward_grouped(x, d_in, layout, [<projection>, ...]) -> [y, ...]
PyObject *linear_forward_grouped(PyObject *, PyObject *const *v, Py_ssize_t n) {
    return guarded([&]() -> PyObject * {
        expect(n, 4);
        const uint64_t d_in = size_arg(v[1]);
        const int32_t layout = (int32_t)size_arg(v[2]);
        Rows r = flatten(tensor(v[0]), d_in);
        Place place(r.x.device());
        if (!PyList_Check(v[3])) raise(PyExc_TypeError, "expected a list of projections");
        const Py_ssize_t count = PyList_GET_SIZE(v[3]);
        std::vector<Projection> ps;
        std::vector<nf4_linear_args> as;
        std::vector<Tensor> ys, scratch;
        ps.reserve(count);
        as.reserve(count);
        for (Py_ssize_t i = 0; i < count; ++i) {
            PyObject *t = PyList_GET_ITEM(v[3], i);
            if (!PyTuple_Check(t) || PyTuple_GET_SIZE(t) != kProjectionArgs) raise(PyExc_TypeError, "bad projection");
            ps.push_back(projection(&PyTuple_GET_ITEM(t, 0), r.x.scalar_type()));
            as.push_back(linear_args(r.x, r.rows, d_in, layout, ps.back()));
            nf4_linear_args &a = as.back();
            r.widen(i == 0 ? d_in : as[i - 1].d_out, a.d_out);
            ys.push_back(empty(r.shape, r.x.scalar_type(), place));
            a.y = ys.back().mutable_data_ptr();
            a.ldy = a.d_out;
            scratch.push_back(forward_workspace(a, ps.back(), place, (uint32_t)i));
            a.workspace = scratch.back().mutable_data_ptr();
            a.workspace_bytes = (uint64_t)scratch.back().numel();
        }
        check(unlocked([&] { return nf4_linear_forward_grouped_dev(as.data(), (uint32_t)count, place.stream); }));
        PyObject *list = PyList_New(count);
        if (!list) throw PyFail{};
        for (Py_ssize_t i = 0; i < count; ++i) PyList_SET_ITEM(list, i, THPVariable_Wrap(std::move(ys[i])));
        return list;
    });
}

// ---- backward -------------------------------------------------------------------------------
// qlora_backward(x, grad_y, d_in, layout, <projection>) -> (grad_x, grad_a, grad_b)
PyObject *qlora_backward(PyObject *, PyObject *const *v, Py_ssize_t n) {
    return guarded([&]() -> PyObject * {
        expect(n, 4 + kProjectionArgs);
        const uint64_t d_in = size_arg(v[2]);
        const int32_t layout = (int32_t)size_arg(v[3]);
        Rows r = flatten(tensor(v[0]), d_in);
        Place place(r.x.device());
        const at::ScalarType type = r.x.scalar_type();
        const Projection p = projection(v + 4, type);
        const Tensor gy = as_type(tensor(v[1]), type);
        require_cuda(gy, "grad_y");
        if ((uint64_t)gy.numel() != r.rows * p.d_out) raise(PyExc_RuntimeError, "grad_y does not have x's rows of d_out values");
        nf4_linear_args a = linear_args(r.x, r.rows, d_in, layout, p);
        Tensor gx = empty(r.shape, type, place);
        Tensor ga = empty(p.a.sizes(), type, place), gb = empty(p.b.sizes(), type, place);
        void *px = gx.mutable_data_ptr(), *pa = ga.mutable_data_ptr(), *pb = gb.mutable_data_ptr();
        const void *pg = gy.const_data_ptr();
        const Tensor ws = workspace(nf4_qlora_backward_workspace_bytes(r.rows, d_in, p.d_out, a.lora_rank),
                                    nf4_qlora_backward_flag_bytes(&a, pg, px), p, place);
        a.workspace = ws.mutable_data_ptr();
        a.workspace_bytes = (uint64_t)ws.numel();
        check(unlocked([&] { return nf4_qlora_backward_dev(&a, pg, px, pa, pb, place.stream); }));
        return Py_BuildValue("NNN", THPVariable_Wrap(std::move(gx)), THPVariable_Wrap(std::move(ga)),
                             THPVariable_Wrap(std::move(gb)));
    });
}

// ---- quantize, dequantize, embedding ----------------------------------------------------------
constexpr int64_t kBlockValues = NF4_BLOCK_SIZE;
int64_t blocks_of(int64_t n) { return (n + kBlockValues - 1) / kBlockValues; }

Tensor flat_f32(const Tensor &t) {
    require_cuda(t, "values");
    return as_type(t, at::kFloat);
}

// quantize(values, one code per byte?) -> (codes, absmax)
PyObject *quantize(PyObject *, PyObject *const *v, Py_ssize_t n) {
    return guarded([&]() -> PyObject * {
        expect(n, 2);
        const Tensor x = flat_f32(tensor(v[0]));
        const bool unpacked = PyObject_IsTrue(v[1]) == 1;
        Place place(x.device());
        const int64_t len = x.numel();
        Tensor codes = empty({unpacked ? len : (len + 1) / 2}, at::kByte, place);
        Tensor absmax = empty({blocks_of(len)}, at::kFloat, place);
        const float *px = ptr_as<float>(&x);
        uint8_t *pc = static_cast<uint8_t *>(codes.mutable_data_ptr());
        float *pa = static_cast<float *>(absmax.mutable_data_ptr());
        check(unlocked([&] {
            return unpacked ? nf4_quantize_unpacked_dev(px, (uint64_t)len, pc, pa, place.stream)
                            : nf4_quantize_dev(px, (uint64_t)len, pc, pa, place.stream);
        }));
        return pair(std::move(codes), std::move(absmax));
    });
}

// quantize_transposed(weight) -> (codes, absmax); quantize_transposed_double(weight) -> (codes, scale_codes, scale_of_scales)
PyObject *quantize_transposed_as(PyObject *const *v, Py_ssize_t n, bool twice) {
    return guarded([&]() -> PyObject * {
        expect(n, 1);
        const Tensor &t = tensor(v[0]);
        require_cuda(t, "weight");
        if (t.dim() != 2 || (t.scalar_type() != at::kFloat && t.scalar_type() != at::kBFloat16))
            raise(PyExc_ValueError, "weight must be a 2-D float32 or bfloat16 tensor");
        const Tensor w = t.contiguous();
        Place place(w.device());
        const int64_t len = w.numel();
        const uint64_t rows = (uint64_t)w.size(0), cols = (uint64_t)w.size(1);
        Tensor codes = empty({(len + 1) / 2}, at::kByte, place);
        Tensor absmax = empty({blocks_of(len)}, at::kFloat, place);
        const uint64_t bytes = twice ? nf4_quantize_transposed_double_workspace_bytes(rows, cols) : nf4_quantize_transposed_workspace_bytes(rows, cols);
        Tensor ws;
        if (bytes) ws = empty({(int64_t)bytes}, at::kByte, place);
        const void *pw = w.const_data_ptr();
        uint8_t *pc = static_cast<uint8_t *>(codes.mutable_data_ptr());
        float *pa = static_cast<float *>(absmax.mutable_data_ptr());
        void *ps = bytes ? ws.mutable_data_ptr() : nullptr;
        const int32_t type = io_dtype(w.scalar_type());
        if (twice) {
            Tensor sc = empty({blocks_of(len)}, at::kByte, place), sos = empty({1}, at::kFloat, place);
            uint8_t *psc = static_cast<uint8_t *>(sc.mutable_data_ptr());
            float *psos = static_cast<float *>(sos.mutable_data_ptr());
            check(unlocked([&] {
                return nf4_quantize_transposed_double_dev(pw, type, rows, cols, pc, pa, psc, psos, ps, bytes, place.stream);
            }));
            return Py_BuildValue("NNN", THPVariable_Wrap(std::move(codes)), THPVariable_Wrap(std::move(sc)), THPVariable_Wrap(std::move(sos)));
        }
        check(unlocked([&] {
            return nf4_quantize_transposed_dev(pw, type, rows, cols, pc, pa, ps, bytes, place.stream);
        }));
        return pair(std::move(codes), std::move(absmax));
    });
}
PyObject *quantize_transposed(PyObject *, PyObject *const *v, Py_ssize_t n) { return quantize_transposed_as(v, n, false); }
PyObject *quantize_transposed_double(PyObject *, PyObject *const *v, Py_ssize_t n) { return quantize_transposed_as(v, n, true); }

// double_quantize(absmax, num_blocks) -> (scale_codes, scale_of_scales)
PyObject *double_quantize(PyObject *, PyObject *const *v, Py_ssize_t n) {
    return guarded([&]() -> PyObject * {
        expect(n, 2);
        const Tensor &absmax = tensor(v[0]);
        require_cuda(absmax, "absmax");
        const uint64_t nb = size_arg(v[1]);
        Place place(absmax.device());
        Tensor sc = empty({(int64_t)nb}, at::kByte, place), sos = empty({1}, at::kFloat, place);
        const float *pa = ptr_as<float>(&absmax);
        uint8_t *pc = nb ? static_cast<uint8_t *>(sc.mutable_data_ptr()) : nullptr;
        float *ps = static_cast<float *>(sos.mutable_data_ptr());
        check(unlocked([&] { return nf4_double_quantize_dev(pa, nb, pc, ps, place.stream); }));
        return pair(std::move(sc), std::move(sos));
    });
}

// dequantize(codes, len, absmax, scale_codes, scale_of_scales, one code per byte?) -> values
PyObject *dequantize(PyObject *, PyObject *const *v, Py_ssize_t n) {
    return guarded([&]() -> PyObject * {
        expect(n, 6);
        const Tensor &codes = tensor(v[0]);
        require_cuda(codes, "codes");
        const uint64_t len = size_arg(v[1]);
        const uint8_t *sc = ptr_as<uint8_t>(tensor_or_none(v[3]));
        const float *am = sc ? nullptr : ptr_as<float>(tensor_or_none(v[2]));
        const float *sos = sc ? ptr_as<float>(tensor_or_none(v[4])) : nullptr;
        const bool unpacked = PyObject_IsTrue(v[5]) == 1;
        Place place(codes.device());
        Tensor out = empty({(int64_t)len}, at::kFloat, place);
        const uint8_t *pc = ptr_as<uint8_t>(&codes);
        float *po = static_cast<float *>(out.mutable_data_ptr());
        check(unlocked([&] {
            return unpacked ? nf4_dequantize_unpacked_dev(pc, len, am, sc, sos, po, place.stream)
                            : nf4_dequantize_dev(pc, len, am, sc, sos, po, place.stream);
        }));
        return THPVariable_Wrap(std::move(out));
    });
}

// quantize_dequantize(values, double_quantization) -> values on the NF4 grid, same shape
PyObject *quantize_dequantize(PyObject *, PyObject *const *v, Py_ssize_t n) {
    return guarded([&]() -> PyObject * {
        expect(n, 2);
        const Tensor x = flat_f32(tensor(v[0]));
        const int32_t dq = PyObject_IsTrue(v[1]) == 1;
        Place place(x.device());
        const uint64_t len = (uint64_t)x.numel(), bytes = nf4_quantize_dequantize_workspace_bytes(len);
        Tensor out = empty(x.sizes(), at::kFloat, place), ws = empty({(int64_t)bytes}, at::kByte, place);
        const float *px = ptr_as<float>(&x);
        float *po = static_cast<float *>(out.mutable_data_ptr());
        void *pw = ws.mutable_data_ptr();
        check(unlocked([&] { return nf4_quantize_dequantize_dev(px, len, dq, po, pw, bytes, place.stream); }));
        return THPVariable_Wrap(std::move(out));
    });
}

// embedding(ids, codes, absmax, scale_codes, scale_of_scales, n_embedding, d_model, bf16?) -> rows
PyObject *embedding(PyObject *, PyObject *const *v, Py_ssize_t n) {
    return guarded([&]() -> PyObject * {
        expect(n, 8);
        const Tensor &codes = tensor(v[1]);
        require_cuda(codes, "codes");
        Place place(codes.device());
        const Tensor &given = tensor(v[0]);
        const Tensor ids = (given.device() == place.device && given.scalar_type() == at::kLong ? given : given.to(place.device, at::kLong)).contiguous();
        const float *am = ptr_as<float>(tensor_or_none(v[2])), *sos = ptr_as<float>(tensor_or_none(v[4]));
        const uint8_t *sc = ptr_as<uint8_t>(tensor_or_none(v[3])), *pc = ptr_as<uint8_t>(&codes);
        const uint64_t rows = size_arg(v[5]), width = size_arg(v[6]), count = (uint64_t)ids.numel();
        const bool bf16 = PyObject_IsTrue(v[7]) == 1;
        std::vector<int64_t> shape = given.sizes().vec();
        shape.push_back((int64_t)width);
        Tensor out = empty(shape, bf16 ? at::kBFloat16 : at::kFloat, place);
        const int64_t *pi = ptr_as<int64_t>(&ids);
        void *po = out.mutable_data_ptr();
        check(unlocked([&] {
            return nf4_embedding_gather_dev(pc, am, sc, sos, rows, width, pi, count, po,
                                            bf16 ? NF4_DTYPE_BF16 : NF4_DTYPE_F32, place.stream);
        }));
        return THPVariable_Wrap(std::move(out));
    });
}

PyObject *release_workspaces(PyObject *, PyObject *) {
    t_kept.clear();
    Py_RETURN_NONE;
}

#define FAST(name) \
    { #name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(name)), METH_FASTCALL, nullptr }
PyMethodDef kMethods[] = {
    FAST(linear_forward), FAST(linear_forward_grouped), FAST(qlora_backward), FAST(quantize), FAST(quantize_transposed),
    FAST(quantize_transposed_double),
    FAST(double_quantize), FAST(dequantize), FAST(quantize_dequantize), FAST(embedding),
    {"release_workspaces", release_workspaces, METH_NOARGS, "Give the calling thread's kept workspaces back."},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&kModule); }
