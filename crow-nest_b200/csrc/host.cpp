// Host side of the small operators as a Python extension: argument checks, output allocation, the current stream and the call into the
// C ABI in one native call. A decode host makes these calls once per matrix and token; through ctypes and torch's Python layer a
// 4096 x 4096 GEMV cost 13 us of host time (3.3 for the current stream, 2.5 for the output, 1 for the view, 1.5 for the arguments) beside
// a kernel of 4.6.
//
// The extension is not linked against the library: the package loads that (the product build, or the diagnostic one) and hands its entry
// points over (`bind`). A non-zero status becomes the package's own exception (`raise_status`, given to `bind`).
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>
#include <string>

namespace {

struct Api {
    int (*gemv)(const void*, const void*, const void*, void*, int, int, int, int, int, void*);
    int (*gemv_gu)(const void*, const void*, const void*, const void*, const void*, void*, int, int, int, int, float, int, void*);
    int (*gemm)(const void*, const void*, const void*, void*, int, int, int, int, int, void*, size_t, void*);
    size_t (*gemm_ws)(int, int, int);
    int (*bs_gemm)(const void*, const void*, const void*, void*, int, int, int, int, int, void*, size_t, void*);
    size_t (*bs_ws)(int, int, int);
    int (*fp8)(const void*, const void*, const void*, void*, int, int, int, int, int, void*);
    int (*head)(const void*, const void*, const void*, void*, void*, int, int, int, int, void*);
    int (*softmax)(const void*, void*, void*, int, int, int, void*);
    int (*sigmoid)(const void*, const void*, void*, void*, int, int, int, float, void*);
} api;
PyObject* g_raise = nullptr;  // raise_status(status or message)

struct Failed {};  // a Python exception is set
[[noreturn]] void raise_with(PyObject* arg) {  // takes arg over
    PyObject* r = arg && g_raise ? PyObject_CallFunctionObjArgs(g_raise, arg, nullptr) : nullptr;
    Py_XDECREF(arg);
    Py_XDECREF(r);
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "crownest_b200: call failed");
    throw Failed();
}
[[noreturn]] void raise(const std::string& s) { raise_with(PyUnicode_FromString(s.c_str())); }
// The call itself runs without the interpreter lock, as through ctypes: a launch may wait for room in the stream.
template <typename F>
void call(F f) {
    int status;
    Py_BEGIN_ALLOW_THREADS;
    status = f();
    Py_END_ALLOW_THREADS;
    if (status != 0) raise_with(PyLong_FromLong(status));
}

const at::Tensor& tensor(PyObject* o) {
    if (!THPVariable_Check(o)) {
        PyErr_Format(PyExc_TypeError, "expected a tensor, got %s", Py_TYPE(o)->tp_name);
        throw Failed();
    }
    return THPVariable_Unpack(o);
}
void* ptr(PyObject* o) { return tensor(o).data_ptr(); }
long integer(PyObject* o) {
    const long v = PyLong_AsLong(o);
    if (v == -1 && PyErr_Occurred()) throw Failed();
    return v;
}
float real(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw Failed();
    return (float)v;
}
int dtype_code(const at::Tensor& t, PyObject* o) {
    if (t.scalar_type() == at::kBFloat16) return 1;
    if (t.scalar_type() == at::kFloat) return 0;
    PyObject* d = PyObject_GetAttrString(o, "dtype");
    PyObject* s = d ? PyObject_Str(d) : nullptr;
    const char* name = s ? PyUnicode_AsUTF8(s) : nullptr;
    const std::string text = std::string("activations must be bf16 or f32, got ") + (name ? name : "?");
    Py_XDECREF(s);
    Py_XDECREF(d);
    PyErr_Clear();
    raise(text);
}
// the rows of x as [m][k], one after another: x itself where it has that form
at::Tensor rows_of(const at::Tensor& x, long k) { return x.dim() == 2 && x.size(1) == k && x.is_contiguous() ? x : x.reshape({-1, k}).contiguous(); }
void* stream() { return (void*)c10::cuda::getCurrentCUDAStream().stream(); }
int i32(long v) { return (int)v; }  // C ints, as the ctypes binding passes them

template <typename F>
PyObject* guarded(F f) {
    try {
        return f();
    } catch (const Failed&) {
    } catch (const c10::Error& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}
bool argc(Py_ssize_t n, Py_ssize_t want) {
    if (n == want) return true;
    PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, n);
    return false;
}
// the caller's output, or the tensor made for it
PyObject* result(PyObject* given, at::Tensor&& made) { return given != Py_None ? Py_NewRef(given) : THPVariable_Wrap(std::move(made)); }

// gemv(w, gs, rows, cols, x, y | None, ldy | None) -> y
PyObject* py_gemv(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!argc(n, 7)) return nullptr;
    return guarded([&]() -> PyObject* {
        const long rows = integer(a[2]), k = integer(a[3]);
        const at::Tensor& x = tensor(a[4]);
        const at::Tensor x2 = rows_of(x, k);
        const long m = x2.size(0);
        at::Tensor y = a[5] == Py_None ? at::empty({m, rows}, x.options()) : tensor(a[5]);
        const long ld = a[6] != Py_None ? integer(a[6]) : (y.dim() == 2 ? y.stride(0) : rows);
        const int dt = dtype_code(x, a[4]);
        void *w = ptr(a[0]), *gs = ptr(a[1]), *px = x2.data_ptr(), *py = y.data_ptr(), *st = stream();
        call([&] { return api.gemv(w, gs, px, py, i32(rows), i32(k), i32(m), i32(ld), dt, st); });
        return result(a[5], std::move(y));
    });
}

// gemv_gu(gate w, up w, gate gs, up gs, rows, cols, x, h | None, limit) -> h
PyObject* py_gemv_gu(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!argc(n, 9)) return nullptr;
    return guarded([&]() -> PyObject* {
        const long rows = integer(a[4]), k = integer(a[5]);
        const at::Tensor& x = tensor(a[6]);
        const at::Tensor x2 = rows_of(x, k);
        const long m = x2.size(0);
        at::Tensor h = a[7] == Py_None ? at::empty({m, rows}, x.options()) : tensor(a[7]);
        const long ld = h.dim() == 2 ? h.stride(0) : rows;
        const float limit = real(a[8]);
        const int dt = dtype_code(x, a[6]);
        void *wg = ptr(a[0]), *wu = ptr(a[1]), *gg = ptr(a[2]), *gu = ptr(a[3]), *px = x2.data_ptr(), *ph = h.data_ptr(), *st = stream();
        call([&] { return api.gemv_gu(wg, wu, gg, gu, px, ph, i32(rows), i32(k), i32(m), i32(ld), limit, dt, st); });
        return result(a[7], std::move(h));
    });
}

// gemm / bs_gemm(w, gs, rows, cols, x, y | None, workspace | None) -> y
template <bool BS>
PyObject* py_gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!argc(n, 7)) return nullptr;
    return guarded([&]() -> PyObject* {
        const long rows = integer(a[2]), k = integer(a[3]);
        const at::Tensor& x = tensor(a[4]);
        const at::Tensor x2 = rows_of(x, k);
        const long m = x2.size(0);
        at::Tensor y = a[5] == Py_None ? at::empty({m, rows}, x.options()) : tensor(a[5]);
        at::Tensor ws = a[6] != Py_None ? tensor(a[6])
                                        : at::empty({(long)(BS ? api.bs_ws : api.gemm_ws)(i32(rows), i32(k), i32(m))}, x.options().dtype(at::kByte));
        const long ld = y.stride(0);
        const int dt = dtype_code(x, a[4]);
        const size_t bytes = (size_t)ws.numel();
        void *w = ptr(a[0]), *gs = ptr(a[1]), *px = x2.data_ptr(), *py = y.data_ptr(), *pw = ws.data_ptr(), *st = stream();
        call([&] { return (BS ? api.bs_gemm : api.gemm)(w, gs, px, py, i32(rows), i32(k), i32(m), i32(ld), dt, pw, bytes, st); });
        return result(a[5], std::move(y));
    });
}

// fp8(w, scale, rows, cols, x, y | None) -> y
PyObject* py_fp8(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!argc(n, 6)) return nullptr;
    return guarded([&]() -> PyObject* {
        const long rows = integer(a[2]), k = integer(a[3]);
        const at::Tensor &w = tensor(a[0]), &scale = tensor(a[1]), &x = tensor(a[4]);
        const at::Tensor x2 = rows_of(x, k);
        const long m = x2.size(0), sr = (rows + 127) / 128, sc = (k + 127) / 128;
        const std::string shape = "[" + std::to_string(rows) + ", " + std::to_string(k) + "]";
        if (w.numel() != rows * k) raise("fp8: " + std::to_string(w.numel()) + " FP8 bytes for shape " + shape);
        if (scale.numel() != sr * sc)
            raise("fp8: " + std::to_string(scale.numel()) + " scales, the 128x128 grid of " + shape + " needs [" + std::to_string(sr) + ", " + std::to_string(sc) +
                  "] = " + std::to_string(sr * sc));
        at::Tensor y = a[5] == Py_None ? at::empty({m, rows}, x.options()) : tensor(a[5]);
        const long ld = y.stride(0);
        const int dt = dtype_code(x, a[4]);
        void *pw = w.data_ptr(), *ps = scale.data_ptr(), *px = x2.data_ptr(), *py = y.data_ptr(), *st = stream();
        call([&] { return api.fp8(pw, ps, px, py, i32(rows), i32(k), i32(m), i32(ld), dt, st); });
        return result(a[5], std::move(y));
    });
}

// head(w, gs, rows, cols, x, logits | None) -> (tokens, logits)
PyObject* py_head(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!argc(n, 6)) return nullptr;
    return guarded([&]() -> PyObject* {
        const long rows = integer(a[2]), k = integer(a[3]);
        const at::Tensor& x = tensor(a[4]);
        const at::Tensor x2 = rows_of(x, k);
        const long m = x2.size(0);
        at::Tensor logits = a[5] == Py_None ? at::empty({m, rows}, x.options()) : tensor(a[5]);
        at::Tensor tokens = at::empty({m}, x.options().dtype(at::kInt));
        const int dt = dtype_code(x, a[4]);
        void *w = ptr(a[0]), *gs = ptr(a[1]), *px = x2.data_ptr(), *pl = logits.data_ptr(), *pt = tokens.data_ptr(), *st = stream();
        call([&] { return api.head(w, gs, px, pl, pt, i32(rows), i32(k), i32(m), dt, st); });
        return Py_BuildValue("(NN)", THPVariable_Wrap(std::move(tokens)), result(a[5], std::move(logits)));
    });
}

// route_softmax(logits, k) / route_sigmoid(logits, bias | None, k, scale) -> (ids, weights)
template <bool SIGMOID>
PyObject* py_route(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!argc(n, SIGMOID ? 4 : 2)) return nullptr;
    return guarded([&]() -> PyObject* {
        const at::Tensor& logits = tensor(a[0]);
        if (logits.dim() != 2) {
            PyErr_Format(PyExc_ValueError, "logits must be [tokens][experts], got %zd dimensions", (Py_ssize_t)logits.dim());
            throw Failed();
        }
        const long k = integer(a[SIGMOID ? 2 : 1]), t = logits.size(0), e = logits.size(1);
        at::Tensor ids = at::empty({t, k}, logits.options().dtype(at::kInt)), wts = at::empty({t, k}, logits.options().dtype(at::kFloat));
        const float scale = SIGMOID ? real(a[3]) : 1.0f;
        void *pl = logits.data_ptr(), *pb = SIGMOID && a[1] != Py_None ? ptr(a[1]) : nullptr, *pi = ids.data_ptr(), *pw = wts.data_ptr(), *st = stream();
        call([&] { return SIGMOID ? api.sigmoid(pl, pb, pi, pw, i32(t), i32(e), i32(k), scale, st) : api.softmax(pl, pi, pw, i32(t), i32(e), i32(k), st); });
        return Py_BuildValue("(NN)", THPVariable_Wrap(std::move(ids)), THPVariable_Wrap(std::move(wts)));
    });
}

// the current stream of the current device, as an address
PyObject* py_stream(PyObject*, PyObject*) {
    return guarded([&]() -> PyObject* { return PyLong_FromVoidPtr(stream()); });
}

// bind({entry point: address}, raise_status)
PyObject* py_bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!argc(n, 2)) return nullptr;
    const struct {
        const char* name;
        void* slot;
    } table[] = {{"cn_nvfp4_gemv", &api.gemv},
                 {"cn_nvfp4_gemv_gu", &api.gemv_gu},
                 {"cn_nvfp4_gemm", &api.gemm},
                 {"cn_nvfp4_gemm_workspace_bytes_of", &api.gemm_ws},
                 {"cn_nvfp4_bs_gemm", &api.bs_gemm},
                 {"cn_nvfp4_bs_workspace_bytes", &api.bs_ws},
                 {"cn_fp8_gemv", &api.fp8},
                 {"cn_lm_head_argmax", &api.head},
                 {"cn_route_softmax_topk", &api.softmax},
                 {"cn_route_sigmoid_topk", &api.sigmoid}};
    for (const auto& t : table) {
        PyObject* v = PyDict_GetItemString(a[0], t.name);
        void* p = v ? PyLong_AsVoidPtr(v) : nullptr;
        if (!p) {
            if (!PyErr_Occurred()) PyErr_Format(PyExc_KeyError, "%s", t.name);
            return nullptr;
        }
        memcpy(t.slot, &p, sizeof p);
    }
    Py_XSETREF(g_raise, Py_NewRef(a[1]));
    Py_RETURN_NONE;
}

#define CN_FAST(name, f) {name, (PyCFunction)(void (*)(void))f, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {CN_FAST("gemv", py_gemv),
                         CN_FAST("gemv_gu", py_gemv_gu),
                         CN_FAST("gemm", py_gemm<false>),
                         CN_FAST("bs_gemm", py_gemm<true>),
                         CN_FAST("fp8", py_fp8),
                         CN_FAST("head", py_head),
                         CN_FAST("route_softmax", py_route<false>),
                         CN_FAST("route_sigmoid", py_route<true>),
                         CN_FAST("bind", py_bind),
                         {"stream", py_stream, METH_NOARGS, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }
