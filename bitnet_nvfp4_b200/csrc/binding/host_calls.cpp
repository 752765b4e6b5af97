// The per-call path of host.py in C: argument conversion, output allocation and the library call of the entry points that a token loop
// issues dozens of times per token. Such a call is a few microseconds of GPU work; through ctypes its host side (three allocations, ten
// to twelve argument conversions, a stream query) took longer than the kernel, so the GPU waited for Python.
// host.py keeps the signatures and passes its arguments on by position.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Device.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>
#include <vector>

#include "bnf4.h"

namespace {

PyObject* g_error = nullptr;  // the package's exception class

struct Failed {};  // a Python exception is set

void* raw_stream() { return reinterpret_cast<void*>(c10::cuda::getCurrentCUDAStream().stream()); }

// Positional arguments, converted as the ctypes prototypes convert them.
struct Args {
    PyObject* const* a;
    Py_ssize_t n, i = 0;
    PyObject* next() {
        if (i >= n) {
            PyErr_Format(PyExc_TypeError, "expected more than %zd arguments", n);
            throw Failed{};
        }
        return a[i++];
    }
    at::Tensor tensor() {
        PyObject* o = next();
        return THPVariable_Check(o) ? THPVariable_Unpack(o) : described(o);
    }
    at::Tensor matrix() {
        at::Tensor t = tensor();
        if (t.dim() != 2) {
            PyErr_Format(PyExc_ValueError, "argument %zd must have two dimensions, not %lld", i, static_cast<long long>(t.dim()));
            throw Failed{};
        }
        return t;
    }
    at::Tensor described(PyObject* o);
    void* ptr();
    int integer();
    float real();
};

// the Python value of a ctypes number or pointer, which the fields of a ctypes structure take (a new reference); nullptr for other objects
PyObject* ctypes_value(PyObject* o) {
    if (PyIndex_Check(o) || PyFloat_Check(o)) return nullptr;
    static PyObject* simple = [] {
        PyObject* m = PyImport_ImportModule("ctypes");
        PyObject* c = m ? PyObject_GetAttrString(m, "_SimpleCData") : nullptr;
        Py_XDECREF(m);
        return c;
    }();
    if (!simple || PyObject_IsInstance(o, simple) != 1) {
        PyErr_Clear();
        return nullptr;
    }
    return PyObject_GetAttrString(o, "value");
}
float to_real(PyObject* o) {
    PyObject* held = PyFloat_Check(o) ? nullptr : ctypes_value(o);
    const double v = PyFloat_AsDouble(held ? held : o);
    Py_XDECREF(held);
    if (v == -1.0 && PyErr_Occurred()) throw Failed{};
    return static_cast<float>(v);
}
long long to_integer(PyObject* o) {
    if (PyLong_Check(o)) {
        const unsigned long long v = PyLong_AsUnsignedLongLongMask(o);
        if (v == ~0ull && PyErr_Occurred()) throw Failed{};
        return static_cast<long long>(v);
    }
    PyObject* held = ctypes_value(o);
    PyObject* l = PyNumber_Index(held ? held : o);
    Py_XDECREF(held);
    if (!l) throw Failed{};
    const unsigned long long v = PyLong_AsUnsignedLongLongMask(l);
    Py_DECREF(l);
    if (v == ~0ull && PyErr_Occurred()) throw Failed{};
    return static_cast<long long>(v);
}
void* to_pointer(PyObject* o) {
    if (o == Py_None) return nullptr;
    if (THPVariable_Check(o)) return THPVariable_Unpack(o).data_ptr();
    if (PyLong_Check(o)) return reinterpret_cast<void*>(to_integer(o));
    PyObject* r = PyObject_HasAttrString(o, "data_ptr") ? PyObject_CallMethod(o, "data_ptr", nullptr) : ctypes_value(o);
    if (!r) {
        if (!PyErr_Occurred()) PyErr_Format(PyExc_TypeError, "%s is no pointer", Py_TYPE(o)->tp_name);
        throw Failed{};
    }
    void* p = r == Py_None ? nullptr : PyLong_AsVoidPtr(r);
    Py_DECREF(r);
    if (!p && PyErr_Occurred()) throw Failed{};
    return p;
}
void* Args::ptr() { return to_pointer(next()); }
// An object that is no tensor but has data_ptr() and, where they are asked for, shape and device. (Bytes without an owner: the element type does
// not matter, the entry points know it.)
at::Tensor Args::described(PyObject* o) {
    if (!PyObject_HasAttrString(o, "data_ptr")) {
        PyErr_Format(PyExc_TypeError, "argument %zd must be a tensor, not %s", i, Py_TYPE(o)->tp_name);
        throw Failed{};
    }
    void* p = to_pointer(o);
    at::globalContext().lazyInitDevice(at::kCUDA);  // (the outputs are allocated by torch)
    std::vector<int64_t> sizes;
    if (PyObject* shape = PyObject_GetAttrString(o, "shape")) {
        PyObject* seq = PySequence_Tuple(shape);
        Py_DECREF(shape);
        if (!seq) throw Failed{};
        for (Py_ssize_t d = 0; d < PyTuple_GET_SIZE(seq); ++d) {
            const Py_ssize_t n = PyNumber_AsSsize_t(PyTuple_GET_ITEM(seq, d), PyExc_OverflowError);
            if (n == -1 && PyErr_Occurred()) {
                Py_DECREF(seq);
                throw Failed{};
            }
            sizes.push_back(n);
        }
        Py_DECREF(seq);
    } else PyErr_Clear();
    at::Device device(at::kCUDA, c10::cuda::current_device());
    if (PyObject* dev = PyObject_GetAttrString(o, "device")) {
        if (THPDevice_Check(dev)) device = reinterpret_cast<THPDevice*>(dev)->device;
        Py_DECREF(dev);
        if (device.is_cuda() && !device.has_index()) device.set_index(c10::cuda::current_device());
    } else PyErr_Clear();
    return at::for_blob(p, sizes).options(at::TensorOptions().dtype(at::kByte).device(device)).target_device(device).make_tensor();
}
float Args::real() { return to_real(next()); }
int Args::integer() { return static_cast<int>(to_integer(next())); }

// Uncleared bytes on a device, straight from the caching allocator, and a tensor on a part of them.
c10::Storage device_bytes(const at::Device& device, int64_t bytes) {
    c10::cuda::OptionalCUDAGuard guard;
    if (device.index() != c10::cuda::current_device()) guard.set_device(device);
    c10::Allocator* from = c10::cuda::CUDACachingAllocator::get();
    return c10::Storage(c10::make_intrusive<c10::StorageImpl>(c10::StorageImpl::use_byte_size_t(), bytes, from->allocate(static_cast<size_t>(bytes)), from, /*resizable=*/true));
}
at::Tensor part(c10::Storage storage, int64_t offset, at::IntArrayRef sizes, at::ScalarType dtype) {  // offset in elements
    at::Tensor t = at::detail::make_tensor<c10::TensorImpl>(std::move(storage), c10::DispatchKeySet(c10::DispatchKey::CUDA), c10::scalarTypeToTypeMeta(dtype));
    t.unsafeGetTensorImpl()->set_storage_offset(offset);
    t.unsafeGetTensorImpl()->set_sizes_contiguous(sizes);
    return t;
}
at::Tensor empty_like_device(const at::Tensor& like, at::IntArrayRef sizes, at::ScalarType dtype) {
    int64_t n = 1;
    for (const int64_t d : sizes) n = d < 0 || n < 0 ? -1 : n * d;
    if (!like.is_cuda() || n < 0) return at::empty(sizes, like.options().dtype(dtype));  // (with its errors)
    return part(device_bytes(like.device(), n * static_cast<int64_t>(c10::elementSize(dtype))), 0, sizes, dtype);
}
// Outputs of a quantiser: the int8 values, and the operand of a GEMM, whose codes and scale bytes share a storage (an allocation is half a
// microsecond, a seventh of the call). Nothing is cleared: the library writes every value, code and scale byte, padding included.
struct Quantised {
    at::Tensor q, codes, sf;
    Quantised(const at::Tensor& like, int64_t rows, int64_t cols, bool want_q) {
        const int64_t nc = (rows * cols * 4 + 7) / 8, ns = (rows + 127) / 128 * 128 * (((cols + 15) / 16 + 3) / 4 * 4);
        if (want_q) q = empty_like_device(like, {rows, cols}, at::kChar);
        if (!like.is_cuda() || rows < 0 || cols < 0) {
            codes = empty_like_device(like, {nc}, at::kByte);
            sf = empty_like_device(like, {ns}, at::kByte);
            return;
        }
        const int64_t at = (nc + 511) / 512 * 512;
        c10::Storage operand = device_bytes(like.device(), at + ns);
        codes = part(operand, 0, {nc}, at::kByte);
        sf = part(std::move(operand), at, {ns}, at::kByte);
    }
    template <typename T>
    T* values() { return static_cast<T*>(q.data_ptr()); }
    PyObject* result() {
        PyObject* parts[3];
        int n = 0;
        if (q.defined()) parts[n++] = THPVariable_Wrap(std::move(q));
        parts[n++] = THPVariable_Wrap(std::move(codes));
        parts[n++] = THPVariable_Wrap(std::move(sf));
        PyObject* t = PyTuple_New(n);
        for (int i = 0; i < n; ++i) PyTuple_SET_ITEM(t, i, parts[i]);
        return t;
    }
};

// The library call itself, without the interpreter lock (as ctypes makes it).
template <typename F>
void call(F&& f) {
    int rc;
    {
        PyThreadState* save = PyEval_SaveThread();
        rc = f();
        PyEval_RestoreThread(save);
    }
    if (rc != 0) {
        PyErr_Format(g_error, "libbnf4 error %d: %s", rc, bnf4_last_error());
        throw Failed{};
    }
}

template <typename T>
T* as(void* p) { return static_cast<T*>(p); }

#define ENTRY(name)                                                            \
    PyObject* name##_body(Args& x);                                            \
    PyObject* name(PyObject*, PyObject* const* args, Py_ssize_t nargs) {       \
        HANDLE_TH_ERRORS                                                       \
        Args x{args, nargs};                                                   \
        try {                                                                  \
            return name##_body(x);                                             \
        } catch (const Failed&) {                                              \
            return nullptr;                                                    \
        }                                                                      \
        END_HANDLE_TH_ERRORS                                                   \
    }                                                                          \
    PyObject* name##_body(Args& x)

ENTRY(quantize_a) {  // x, k_out
    const at::Tensor t = x.matrix();
    const int m = static_cast<int>(t.size(0)), k = static_cast<int>(t.size(1)), k_out = x.integer();
    Quantised o(t, m, k_out, false);
    const void* in = t.data_ptr();
    void* s = raw_stream();
    call([&] { return bnf4_nvfp4_quantize_a(static_cast<const int8_t*>(in), m, 1, k, k_out, as<uint8_t>(o.codes.data_ptr()), as<uint8_t>(o.sf.data_ptr()), s); });
    return o.result();
}

ENTRY(embedding_lookup_noise_quantize) {  // tokens, token_stride, emb_w, emb_noise, hidden, batch, noise_scale, anti_sign
    void* tokens = x.ptr();
    const int stride = x.integer();
    const at::Tensor emb = x.tensor();
    void* noise = x.ptr();
    const int hidden = x.integer(), batch = x.integer();
    const float scale = x.real();
    const int anti = x.integer();
    Quantised o(emb, batch, hidden, true);
    void *w = emb.data_ptr(), *s = raw_stream();
    call([&] {
        return bnf4_embedding_lookup_noise_quantize_nvfp4(as<uint8_t>(tokens), stride, as<int8_t>(w), as<int8_t>(noise), hidden, batch, scale, anti,
                                                          o.values<int8_t>(), as<uint8_t>(o.codes.data_ptr()), as<uint8_t>(o.sf.data_ptr()), s);
    });
    return o.result();
}

ENTRY(add_pos_gelu_quantize) {  // x, pos, act_scale
    const at::Tensor t = x.matrix();
    const int batch = static_cast<int>(t.size(0)), hidden = static_cast<int>(t.size(1));
    void* pos = x.ptr();
    const float act = x.real();
    Quantised o(t, batch, hidden, true);
    void *in = t.data_ptr(), *s = raw_stream();
    call([&] {
        return bnf4_add_pos_gelu_quantize_nvfp4(as<float>(in), as<float>(pos), hidden, batch, act, o.values<int8_t>(), as<uint8_t>(o.codes.data_ptr()),
                                                as<uint8_t>(o.sf.data_ptr()), s);
    });
    return o.result();
}

ENTRY(absmean_norm_q) {  // x8, scale
    const at::Tensor t = x.matrix();
    const int batch = static_cast<int>(t.size(0)), hidden = static_cast<int>(t.size(1));
    const float scale = x.real();
    Quantised o(t, batch, hidden, true);
    void *in = t.data_ptr(), *s = raw_stream();
    call([&] {
        return bnf4_absmean_norm_q_nvfp4(as<int8_t>(in), hidden, batch, hidden, scale, o.values<int8_t>(), as<uint8_t>(o.codes.data_ptr()),
                                         as<uint8_t>(o.sf.data_ptr()), s);
    });
    return o.result();
}

ENTRY(add_scaled_absmean_norm_q) {  // x8_inout, y, add_scale, norm_scale
    const at::Tensor t = x.matrix();
    const int batch = static_cast<int>(t.size(0)), hidden = static_cast<int>(t.size(1));
    const at::Tensor y = x.tensor();
    const float add = x.real(), norm = x.real();
    Quantised o(y, batch, hidden, true);
    void *inout = t.data_ptr(), *yp = y.data_ptr(), *s = raw_stream();
    call([&] {
        return bnf4_add_scaled_to_int8_absmean_norm_q_nvfp4(as<int8_t>(inout), as<float>(yp), hidden, batch, hidden, add, norm, o.values<int8_t>(),
                                                            as<uint8_t>(o.codes.data_ptr()), as<uint8_t>(o.sf.data_ptr()), s);
    });
    return o.result();
}

ENTRY(gemm) {  // a, b, sfa, sfb, m, n, k, alpha, beta, c, d
    const at::Tensor a = x.tensor();
    void *b = x.ptr(), *sfa = x.ptr(), *sfb = x.ptr();
    const int m = x.integer(), n = x.integer(), k = x.integer();
    const float alpha = x.real(), beta = x.real();
    void* c = x.ptr();
    PyObject* given = x.next();
    at::Tensor made;
    if (given == Py_None) made = empty_like_device(a, {m, n}, at::kFloat);
    void *d = given == Py_None ? made.data_ptr() : to_pointer(given), *ap = a.data_ptr(), *s = raw_stream();
    call([&] {
        return bnf4_gemm_ternary_f_nvfp4(as<uint8_t>(ap), as<uint8_t>(b), as<uint8_t>(sfa), as<uint8_t>(sfb), m, n, k, alpha, beta, as<float>(c), as<float>(d), s);
    });
    if (given == Py_None) return THPVariable_Wrap(std::move(made));
    Py_INCREF(given);
    return given;
}

ENTRY(gemm_gelu_i8) {  // a, b, sfa, sfb, m, n, k, alpha, beta, c, act_scale
    const at::Tensor a = x.tensor();
    void *b = x.ptr(), *sfa = x.ptr(), *sfb = x.ptr();
    const int m = x.integer(), n = x.integer(), k = x.integer();
    const float alpha = x.real(), beta = x.real();
    void* c = x.ptr();
    const float act = x.real();
    at::Tensor d = empty_like_device(a, {m, n}, at::kChar);
    void *dp = d.data_ptr(), *ap = a.data_ptr(), *s = raw_stream();
    call([&] {
        return bnf4_gemm_ternary_f_nvfp4_gelu_i8(as<uint8_t>(ap), as<uint8_t>(b), as<uint8_t>(sfa), as<uint8_t>(sfb), m, n, k, alpha, beta, as<float>(c), act,
                                                 as<int8_t>(dp), s);
    });
    return THPVariable_Wrap(std::move(d));
}

ENTRY(efla_step_half) {  // S, qkv, fused_cols, beta_bias, hidden, batch, method, eps
    void* S = x.ptr();
    const at::Tensor qkv = x.tensor();
    const int fused = x.integer();
    const float bias = x.real();
    const int hidden = x.integer(), batch = x.integer(), method = x.integer();
    const float eps = x.real();
    if (at::isFloatingType(qkv.scalar_type()) && qkv.scalar_type() != at::kFloat) {  // (raw bytes of floats are a caller's business)
        PyErr_Format(PyExc_TypeError, "qkv must be float32, not %s", at::toString(qkv.scalar_type()));
        throw Failed{};
    }
    at::Tensor out = empty_like_device(qkv, {batch, hidden}, at::kFloat);
    void *in = qkv.data_ptr(), *o = out.data_ptr(), *s = raw_stream();
    call([&] { return bnf4_efla_step_half_qkv_fused(as<uint16_t>(S), as<float>(in), fused, bias, hidden, batch, method, eps, as<float>(o), s); });
    return THPVariable_Wrap(std::move(out));
}

ENTRY(cross_entropy) {  // logits, bias, bias_noise, bias_noise_scale, targets, token_stride, loss
    const at::Tensor logits = x.matrix();
    const int batch = static_cast<int>(logits.size(0)), vocab = static_cast<int>(logits.size(1));
    void *bias = x.ptr(), *noise = x.ptr();
    const float scale = x.real();
    void* targets = x.ptr();
    const int stride = x.integer();
    void *loss = x.ptr(), *in = logits.data_ptr(), *s = raw_stream();
    call([&] { return bnf4_cross_entropy_loss(as<float>(in), as<float>(bias), as<float>(noise), scale, as<uint8_t>(targets), stride, vocab, batch, as<float>(loss), s); });
    Py_RETURN_NONE;
}

// ---- descriptor calls: the fields of the ctypes structures, registered once ----
struct Field {
    int offset;
    char code;  // 'P' pointer, 'i' int, 'f' float, 'q' long long
};
struct Desc {
    size_t size = 0;
    std::vector<Field> fields;
    PyObject* index = nullptr;  // name -> position in fields
};
Desc g_desc[3];  // row quantiser, GEMM, scan

ENTRY(register_desc) {  // kind, size, [(name, offset, code), ...]
    Desc& d = g_desc[x.integer()];
    d.size = static_cast<size_t>(x.integer());
    PyObject* list = x.next();
    d.fields.clear();
    Py_XDECREF(d.index);
    d.index = PyDict_New();
    for (Py_ssize_t i = 0; i < PyList_Size(list); ++i) {
        const char *name, *code;
        int offset;
        if (!PyArg_ParseTuple(PyList_GetItem(list, i), "sis", &name, &offset, &code)) throw Failed{};
        PyObject* pos = PyLong_FromLong(static_cast<long>(i));
        PyDict_SetItemString(d.index, name, pos);
        Py_DECREF(pos);
        d.fields.push_back({offset, code[0]});
    }
    Py_RETURN_NONE;
}

ENTRY(desc_call) {  // kind, front end (row quantiser), {field: value}
    const int kind = x.integer(), front_end = x.integer();
    PyObject* kw = x.next();
    const Desc& d = g_desc[kind];
    alignas(16) unsigned char buf[512] = {};
    if (d.index == nullptr || d.size > sizeof(buf)) {
        PyErr_SetString(PyExc_RuntimeError, "descriptor is not registered");
        throw Failed{};
    }
    PyObject *key, *value;
    Py_ssize_t at = 0;
    while (PyDict_Next(kw, &at, &key, &value)) {
        PyObject* pos = PyDict_GetItemWithError(d.index, key);
        if (!pos) {
            if (PyErr_Occurred()) throw Failed{};
            continue;  // not a field: ignored
        }
        const Field f = d.fields[static_cast<size_t>(PyLong_AsLong(pos))];
        if (f.code == 'f') {
            const float fv = to_real(value);
            std::memcpy(buf + f.offset, &fv, 4);
        } else if (f.code == 'P') {
            void* p = to_pointer(value);
            std::memcpy(buf + f.offset, &p, sizeof(p));
        } else {
            const long long v = to_integer(value);
            std::memcpy(buf + f.offset, &v, f.code == 'q' ? 8 : 4);  // little endian: the low half
        }
    }
    void* s = raw_stream();
    call([&] {
        if (kind == 0) return bnf4_rowquant(front_end, reinterpret_cast<const bnf4_rowquant_desc*>(buf), s);
        if (kind == 1) return bnf4_gemm_nvfp4_ex(reinterpret_cast<const bnf4_gemm_desc*>(buf), s);
        return bnf4_efla_scan(reinterpret_cast<const bnf4_efla_desc*>(buf), s);
    });
    Py_RETURN_NONE;
}

ENTRY(set_error_class) {
    PyObject* e = x.next();
    Py_INCREF(e);
    Py_XSETREF(g_error, e);
    Py_RETURN_NONE;
}

#define METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {METHOD(quantize_a), METHOD(embedding_lookup_noise_quantize), METHOD(add_pos_gelu_quantize), METHOD(absmean_norm_q),
                         METHOD(add_scaled_absmean_norm_q), METHOD(gemm), METHOD(gemm_gelu_i8), METHOD(efla_step_half), METHOD(cross_entropy),
                         METHOD(register_desc), METHOD(desc_call), METHOD(set_error_class), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", "Per-call path of the kernel-entry functions.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module_def); }
