// The Python face of the hot calls (module `_call`): linear, the routed chain and the plugin table's matmul on host arrays,
// argument checks, output and workspace allocation and the launch in one native call. Through ctypes a one-row linear spent
// 15 us on the host around a 7 us kernel (attribute reads, argument conversion, two Python-level allocations).
//
// Every function returns None when an argument is not what the engine takes: the Python side then names the refusal. A
// status of the C ABI other than T3_OK comes back as an int.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/t3.h"
#include "../../include/t3_table.h"

namespace {

PyObject *s_trellis, *s_suh, *s_svh, *s_gate, *s_up, *s_down, *s_codebook, *s_window_bits;

// an attribute whose holder keeps it alive (instances of the package's dataclasses)
struct Attr {
    PyObject* p;
    Attr(PyObject* o, PyObject* name) : p(PyObject_GetAttr(o, name)) {}
    ~Attr() { Py_XDECREF(p); }
};

const at::Tensor* tensor(PyObject* o) {
    if (!THPVariable_Check(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    return t.is_cuda() && t.is_contiguous() ? &t : nullptr;
}

int act_dtype(const at::Tensor& t) {
    switch (t.scalar_type()) {
        case at::kFloat: return T3_F32;
        case at::kHalf: return T3_F16;
        case at::kBFloat16: return T3_BF16;
        default: return -1;
    }
}
bool is_codes(const at::Tensor& t) { return t.scalar_type() == at::kUInt16 || t.scalar_type() == at::kShort; }
bool is_half(const at::Tensor& t) { return t.scalar_type() == at::kHalf; }
bool is_index(const at::Tensor& t) { return t.scalar_type() == at::kInt || t.scalar_type() == at::kUInt32; }

bool decode_of(PyObject* o, t3_decode& dec) {
    Attr cb(o, s_codebook), wb(o, s_window_bits);
    if (!cb.p || !wb.p) return false;
    dec.codebook = (int)PyLong_AsLong(cb.p);
    dec.window_bits = (int)PyLong_AsLong(wb.p);
    return !PyErr_Occurred();
}

at::Tensor empty(at::IntArrayRef sizes, at::ScalarType type, const at::Tensor& like) {
    return at::Tensor(at::detail::empty_cuda(sizes, type, like.device(), std::nullopt));
}

void* stream_of(const at::Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

PyObject* finish(int status, at::Tensor& y) {
    if (status != T3_OK) return PyLong_FromLong(status);
    return THPVariable_Wrap(std::move(y));
}

// linear(x, trellis, suh, svh, dec)
PyObject* call_linear(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    if (nargs != 5) Py_RETURN_NONE;
    const at::Tensor *x = tensor(args[0]), *t = tensor(args[1]), *suh = tensor(args[2]), *svh = tensor(args[3]);
    if (!x || !t || !suh || !svh || x->dim() < 1 || t->dim() != 3) Py_RETURN_NONE;
    const int64_t in = t->size(0) * 16, out = t->size(1) * 16, n = t->size(2);
    const int dt = act_dtype(*x);
    if (x->size(-1) != in || suh->numel() != in || svh->numel() != out || dt < 0 || !is_codes(*t) || !is_half(*suh) || !is_half(*svh) ||
        in == 0 || in > INT32_MAX || out > INT32_MAX)
        Py_RETURN_NONE;
    const int64_t rows = x->numel() / in;
    t3_decode dec;
    if (rows < 1 || !decode_of(args[4], dec)) {
        if (PyErr_Occurred()) return nullptr;
        Py_RETURN_NONE;
    }
    c10::SmallVector<int64_t, 5> shape(x->sizes().begin(), x->sizes().end());
    shape.back() = out;
    at::Tensor y = empty(shape, x->scalar_type(), *x), ws;
    const size_t bytes = t3_linear_workspace_bytes((size_t)rows, (int)in, (int)out, (int)n);
    if (bytes) ws = empty({(int64_t)bytes}, at::kByte, *x);
    void* stream = stream_of(*x);
    int status;
    Py_BEGIN_ALLOW_THREADS
    status = t3_linear(x->data_ptr(), dt, (size_t)rows, t->data_ptr(), suh->data_ptr(), svh->data_ptr(), (int)in, (int)out, (int)n, dec,
                       y.data_ptr(), bytes ? ws.data_ptr() : nullptr, bytes, stream);
    Py_END_ALLOW_THREADS
    return finish(status, y);
    END_HANDLE_TH_ERRORS
}

// One projection of a bank: trellis [E, in / 16, out / 16, n], suh [E, in], svh [E, out]
bool proj_of(PyObject* bank, PyObject* name, t3_proj& p, int64_t (&dims)[4]) {
    Attr proj(bank, name);
    if (!proj.p) return false;
    Attr to(proj.p, s_trellis), so(proj.p, s_suh), vo(proj.p, s_svh);
    if (!to.p || !so.p || !vo.p) return false;
    const at::Tensor *t = tensor(to.p), *suh = tensor(so.p), *svh = tensor(vo.p);
    if (!t || !suh || !svh || t->dim() != 4 || suh->dim() != 2 || svh->dim() != 2 || !is_codes(*t) || !is_half(*suh) || !is_half(*svh))
        return false;
    for (int i = 0; i < 4; ++i) dims[i] = t->size(i);
    dims[1] *= 16, dims[2] *= 16;
    if (suh->size(0) != dims[0] || suh->size(1) != dims[1] || svh->size(0) != dims[0] || svh->size(1) != dims[2]) return false;
    p = {t->data_ptr(), suh->data_ptr(), svh->data_ptr()};
    return true;
}

// moe(x, bank, inds, scores, dec, limit, clamp_at, shared or None, event handle or 0)
PyObject* call_moe(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    if (nargs != 9) Py_RETURN_NONE;
    const at::Tensor *x = tensor(args[0]), *inds = tensor(args[2]), *scores = tensor(args[3]);
    if (!x || !inds || !scores || x->dim() != 3 || inds->dim() != 3 || x->size(0) != inds->size(0) || x->size(1) != inds->size(1) ||
        !inds->sizes().equals(scores->sizes()))
        Py_RETURN_NONE;
    const int64_t topk = inds->size(2), hidden = x->size(2), rows = x->size(0) * x->size(1);
    const int dt = act_dtype(*x), sdt = act_dtype(*scores);
    if (topk <= 0 || topk > T3_REDUCE_MAX_TOPK || hidden % 128 || dt < 0 || sdt < 0 || !is_index(*inds)) Py_RETURN_NONE;
    t3_bank bank = {};
    int64_t g[4], u[4], d[4];
    if (!proj_of(args[1], s_gate, bank.gate, g) || !proj_of(args[1], s_up, bank.up, u) || !proj_of(args[1], s_down, bank.down, d)) {
        PyErr_Clear();
        Py_RETURN_NONE;
    }
    const int64_t inter = g[2];
    if (g[1] != hidden || u[1] != hidden || u[2] != inter || d[1] != inter || d[2] != hidden || u[0] != g[0] || d[0] != g[0] || inter % 128)
        Py_RETURN_NONE;
    bank.experts = (int)g[0], bank.hidden = (int)hidden, bank.inter = (int)inter;
    bank.n_gate = (int)g[3], bank.n_up = (int)u[3], bank.n_down = (int)d[3];
    t3_decode dec;
    if (!decode_of(args[4], dec)) return nullptr;
    const long limit = PyLong_AsLong(args[5]), clamp_at = PyLong_AsLong(args[6]);
    const at::Tensor* shared = nullptr;
    if (args[7] != Py_None) {
        shared = tensor(args[7]);
        if (!shared || shared->scalar_type() != x->scalar_type() || shared->numel() != x->numel()) Py_RETURN_NONE;
    }
    void* event = PyLong_AsVoidPtr(args[8]);
    if (PyErr_Occurred()) return nullptr;
    const size_t bytes = t3_moe_workspace_bytes((size_t)rows, (int)topk, &bank);
    at::Tensor ws = empty({(int64_t)(bytes ? bytes : 1)}, at::kByte, *x), y = empty(x->sizes(), x->scalar_type(), *x);
    void* stream = stream_of(*x);
    int status;
    Py_BEGIN_ALLOW_THREADS
    if (shared && event)
        status = t3_moe_with_shared_after(x->data_ptr(), dt, (size_t)rows, &bank, inds->data_ptr(), scores->data_ptr(), sdt, (int)topk, dec,
                                          shared->data_ptr(), event, y.data_ptr(), ws.data_ptr(), bytes, stream);
    else if (shared)
        status = t3_moe_with_shared(x->data_ptr(), dt, (size_t)rows, &bank, inds->data_ptr(), scores->data_ptr(), sdt, (int)topk, dec,
                                    shared->data_ptr(), y.data_ptr(), ws.data_ptr(), bytes, stream);
    else
        status = t3_moe_swiglu(x->data_ptr(), dt, (size_t)rows, &bank, inds->data_ptr(), scores->data_ptr(), sdt, (int)topk, dec,
                               (uint32_t)limit, (int)clamp_at, y.data_ptr(), ws.data_ptr(), bytes, stream);
    Py_END_ALLOW_THREADS
    return finish(status, y);
    END_HANDLE_TH_ERRORS
}

struct Buffer {
    Py_buffer view = {};
    bool held = false;
    bool get(PyObject* o, int flags) { return held = PyObject_GetBuffer(o, &view, flags) == 0; }
    ~Buffer() {
        if (held) PyBuffer_Release(&view);
    }
};

// table_matmul(weight, x, y, stream, dtype): the plugin table's matmul on two host buffers. True, or None where the caller has
// to take the general path (other dtypes, a refusal to be named).
PyObject* call_table_matmul(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    if (nargs != 5) Py_RETURN_NONE;
    Buffer w, x, y;
    if (!w.get(args[0], PyBUF_SIMPLE) || w.view.len != (Py_ssize_t)sizeof(t3_weight) || !x.get(args[1], PyBUF_ND) ||
        !y.get(args[2], PyBUF_ND | PyBUF_WRITABLE) || x.view.ndim < 1 || x.view.ndim > 8 || y.view.ndim != x.view.ndim) {
        PyErr_Clear();
        Py_RETURN_NONE;
    }
    void* stream = PyLong_AsVoidPtr(args[3]);
    const int dtype = (int)PyLong_AsLong(args[4]);
    if (PyErr_Occurred()) return nullptr;
    t3_array xa = {}, ya = {};
    for (int k = 0; k < 2; ++k) {
        t3_array& a = k ? ya : xa;
        const Py_buffer& v = k ? y.view : x.view;
        a.data = v.buf;
        a.dtype = dtype;
        a.ndim = v.ndim;
        for (int i = 0; i < v.ndim; ++i) a.shape[i] = v.shape[i];
    }
    static const auto matmul = t3_table()->matmul;
    t3_verdict verdict;
    Py_BEGIN_ALLOW_THREADS
    verdict = matmul(static_cast<const t3_weight*>(w.view.buf), &xa, stream, &ya);
    Py_END_ALLOW_THREADS
    if (verdict.kind != T3_VERDICT_OK) Py_RETURN_NONE;
    Py_RETURN_TRUE;
}

PyMethodDef methods[] = {
    {"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(call_linear)), METH_FASTCALL, nullptr},
    {"moe", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(call_moe)), METH_FASTCALL, nullptr},
    {"table_matmul", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(call_table_matmul)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_call", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__call(void) {
    s_trellis = PyUnicode_InternFromString("trellis"), s_suh = PyUnicode_InternFromString("suh"), s_svh = PyUnicode_InternFromString("svh");
    s_gate = PyUnicode_InternFromString("gate"), s_up = PyUnicode_InternFromString("up"), s_down = PyUnicode_InternFromString("down");
    s_codebook = PyUnicode_InternFromString("codebook"), s_window_bits = PyUnicode_InternFromString("window_bits");
    return PyModule_Create(&module);
}
