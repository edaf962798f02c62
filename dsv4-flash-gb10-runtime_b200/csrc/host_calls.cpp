// dsv4_host.so - the Python operators' call path in C++: argument checks, output allocation and the call of the C ABI
// entry, for the common case of well-formed CUDA tensors on the current stream.
//
// A call through ctypes with its checks in Python took 17 us of host time, more than the kernel of every dense operator;
// this takes about 3 (most of it the launch itself).  A function returns None when anything is out of the ordinary (tensors of
// several devices or of one that is not current, a stride, a shape that does not fit, an explicit stream): the caller then goes
// through the checks in Python, which name what is wrong, copy what may be copied, or make the device current.  Entry addresses come from the ctypes-loaded libraries (bind), so the
// environment overrides of the library paths hold here too.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <cstring>

namespace {

using at::ScalarType;
using at::Tensor;
typedef const void* P;

struct Entries {
    void *mxfp4_gemv_m1, *fp8_e4m3_gemv_m1, *fp8_e4m3_gemv_m1_f32scale, *fp8_e4m3_gemv_batched, *fp8_e4m3_shared_swiglu_m1,
        *fp8_e4m3_shared_swiglu_workspace_bytes, *mxfp4_grouped_gemv_topk, *mxfp4_grouped_workspace_bytes,
        *mxfp4_grouped_gemv_topk_ids_stages, *mxfp4_moe_route_topk, *mxfp4_moe_decode_layer, *mxfp4_moe_decode_workspace_bytes,
        *mxfp4_moe_forward, *mxfp4_moe_forward_path, *mxfp4_moe_forward_workspace_bytes;
} entry = {};
const struct { const char* name; void** slot; } kEntries[] = {
#define DSV4_ENTRY(n) {#n, &entry.n}
    DSV4_ENTRY(mxfp4_gemv_m1), DSV4_ENTRY(fp8_e4m3_gemv_m1), DSV4_ENTRY(fp8_e4m3_gemv_m1_f32scale),
    DSV4_ENTRY(fp8_e4m3_gemv_batched), DSV4_ENTRY(fp8_e4m3_shared_swiglu_m1),
    DSV4_ENTRY(fp8_e4m3_shared_swiglu_workspace_bytes), DSV4_ENTRY(mxfp4_grouped_gemv_topk),
    DSV4_ENTRY(mxfp4_grouped_workspace_bytes), DSV4_ENTRY(mxfp4_grouped_gemv_topk_ids_stages), DSV4_ENTRY(mxfp4_moe_route_topk),
    DSV4_ENTRY(mxfp4_moe_decode_layer), DSV4_ENTRY(mxfp4_moe_decode_workspace_bytes), DSV4_ENTRY(mxfp4_moe_forward),
    DSV4_ENTRY(mxfp4_moe_forward_path), DSV4_ENTRY(mxfp4_moe_forward_workspace_bytes),
#undef DSV4_ENTRY
};
template <class F>
F fn(void* p) { return reinterpret_cast<F>(p); }
// The C entry, called as ctypes calls it: other Python threads go on meanwhile (a launch blocks while its queue is full).  The
// arguments are evaluated before the lock is given up.
struct Unlocked {
    PyThreadState* const state = PyEval_SaveThread();
    ~Unlocked() { PyEval_RestoreThread(state); }
};
template <class... Params, class... Args>
int call(int (*f)(Params...), Args... args) {
    Unlocked unlocked;
    return f(args...);
}

// A CUDA tensor of the given type, or nullptr.
const Tensor* cuda(PyObject* o, ScalarType type) {
    if (!o || !THPVariable_Check(o)) return nullptr;
    const Tensor& t = THPVariable_Unpack(o);
    return t.is_cuda() && t.scalar_type() == type ? &t : nullptr;
}
const Tensor* dense(PyObject* o, ScalarType type) {
    const Tensor* t = cuda(o, type);
    return t && t->is_contiguous() ? t : nullptr;
}
bool shape(const Tensor& t, std::initializer_list<int64_t> want) {
    return t.sizes() == at::IntArrayRef(want);
}
// All on one device.
bool together(std::initializer_list<const Tensor*> tensors) {
    const auto device = (*tensors.begin())->device();
    for (const Tensor* t : tensors)
        if (t->device() != device) return false;
    return true;
}
// That device is the current one, which allocation, stream and launch are meant for.  (A guard that makes it so cost every call
// about 0.1 us.)
bool current(const Tensor* t) { return c10::cuda::current_device() == t->device().index(); }
// An optional output or workspace: on that device, or not on a GPU at all (mapped host memory, where an operator takes it).
bool reachable(PyObject* given, const Tensor* like) {
    if (given == Py_None) return true;
    if (!THPVariable_Check(given)) return false;
    const Tensor& t = THPVariable_Unpack(given);
    return !t.is_cuda() || t.device() == like->device();
}
P ptr(const Tensor* t) { return t->const_data_ptr(); }
void* stream_of(const Tensor* t) { return c10::cuda::getCurrentCUDAStream(t->device().index()).stream(); }
Tensor empty(at::IntArrayRef size, ScalarType type, const Tensor* like) {
    return at::detail::empty_cuda(size, type, like->device(), std::nullopt);
}
PyObject* failed(const char* what, int rc) {
    PyErr_Format(PyExc_RuntimeError, "%s returned %d", what, rc);
    return nullptr;
}
// The caller's output (any object it passed), or the one made here.
PyObject* result(PyObject* given, Tensor&& made) {
    if (given != Py_None) { Py_INCREF(given); return given; }
    return THPVariable_Wrap(std::move(made));
}
constexpr ScalarType kByte = ScalarType::Byte, kBf16 = ScalarType::BFloat16, kF32 = ScalarType::Float, kI32 = ScalarType::Int;
PyObject* kKeys[12] = {};      // interned dictionary keys
enum { kW1p, kW3p, kW2p, kW1s, kW3s, kW2s, kW1, kW3, kW2, kPacked, kScale };
PyObject* get(PyObject* dict, int key) { return PyDict_Check(dict) ? PyDict_GetItem(dict, kKeys[key]) : nullptr; }

#define FAST(name) PyObject* name(PyObject*, PyObject* const* a, Py_ssize_t n)
#define ORDINARY(cond) do { if (!(cond)) { PyErr_Clear(); Py_RETURN_NONE; } } while (0)      // (an integer beyond 64 bits is an error that is pending)
// C++ exceptions become the Python ones that torch raises for them (torch.OutOfMemoryError for an allocation).
#define GUARD(...) try { __VA_ARGS__ } catch (...) { torch::translate_exception_to_python(std::current_exception()); return nullptr; }

FAST(bind) {
    if (n != 2) { PyErr_SetString(PyExc_TypeError, "bind(name, address)"); return nullptr; }
    const char* name = PyUnicode_AsUTF8(a[0]);
    void* p = PyLong_AsVoidPtr(a[1]);
    if (!name || PyErr_Occurred()) return nullptr;
    for (const auto& e : kEntries)
        if (!std::strcmp(e.name, name)) *e.slot = p;
    Py_RETURN_NONE;
}

// A caller's optional output vector of `rows` bf16 values: None, or one that fits.
bool good_out(PyObject* o, std::initializer_list<int64_t> want, const Tensor* like) {
    if (o == Py_None) return true;
    const Tensor* t = dense(o, kBf16);
    return t && shape(*t, want) && t->device() == like->device();
}

PyObject* dense_gemv(void* f, const char* what, PyObject* const* a, Py_ssize_t n, int64_t per_block_k, int64_t tile, ScalarType scale_type) {
    ORDINARY(n == 5 && f && a[4] == Py_None);
    const Tensor *w = cuda(a[0], kByte), *s = cuda(a[1], scale_type), *x = dense(a[2], kBf16);
    ORDINARY(w && s && x && x->dim() == 1 && w->dim() == 2 && s->dim() == 2);
    const int64_t K = x->size(0), N = w->size(0);
    const bool fp4 = tile == 1;
    ORDINARY(K % per_block_k == 0 && N % tile == 0 && w->size(1) == (fp4 ? K / 2 : K) && s->size(0) == N / tile &&
             s->size(1) == K / per_block_k && w->stride(1) == 1 && s->stride(1) == 1 && together({x, w, s}) && good_out(a[3], {N}, x));
    ORDINARY(current(x));
    Tensor made;
    void* y;
    if (a[3] == Py_None) { made = empty({N}, kBf16, x); y = made.mutable_data_ptr(); }
    else y = THPVariable_Unpack(a[3]).mutable_data_ptr();
    const int rc = call(fn<int (*)(P, P, P, int, int, int64_t, int64_t, void*, void*)>(f),
        ptr(x), ptr(w), ptr(s), (int)K, (int)N, w->stride(0), s->stride(0) * (int64_t)s->element_size(), y, stream_of(x));
    if (rc != 0) return failed(what, rc);
    return result(a[3], std::move(made));
}
FAST(mxfp4_gemv) { GUARD(return dense_gemv(entry.mxfp4_gemv_m1, "mxfp4_gemv_m1", a, n, 32, 1, kByte);) }
FAST(fp8_gemv) { GUARD(return dense_gemv(entry.fp8_e4m3_gemv_m1, "fp8_e4m3_gemv_m1", a, n, 128, 128, kByte);) }
FAST(fp8_gemv_f32scale) { GUARD(return dense_gemv(entry.fp8_e4m3_gemv_m1_f32scale, "fp8_e4m3_gemv_m1_f32scale", a, n, 128, 128, kF32);) }

// (W_fp8, W_scale, x, n_groups, out, stream)
FAST(fp8_gemv_batched) { GUARD(
    ORDINARY(n == 6 && entry.fp8_e4m3_gemv_batched && a[5] == Py_None && PyLong_Check(a[3]));
    const Tensor *w = cuda(a[0], kByte), *s = cuda(a[1], kByte), *x = cuda(a[2], kBf16);
    ORDINARY(w && s && x && w->dim() == 2 && s->dim() == 2 && (x->dim() == 1 || x->dim() == 2));
    const int64_t G = PyLong_AsLong(a[3]), K = w->size(1), rows = w->size(0);
    const bool single = x->dim() == 1;
    const int64_t S = single ? 1 : x->size(0), row = single ? x->size(0) : x->size(1);
    ORDINARY(G >= 1 && row == G * K && rows % G == 0 && K % 128 == 0 && (rows / G) % 128 == 0 && s->size(0) == rows / 128 &&
             s->size(1) == K / 128 && w->stride(1) == 1 && s->stride(1) == 1 && x->stride(-1) == 1 && a[4] == Py_None && together({x, w, s}));
    ORDINARY(current(x));
    Tensor y = single ? empty({rows}, kBf16, x) : empty({S, rows}, kBf16, x);
    const int rc = call(fn<int (*)(P, P, P, int, int, int64_t, int64_t, int, int, int64_t, int64_t, void*, void*)>(entry.fp8_e4m3_gemv_batched),
        ptr(x), ptr(w), ptr(s), (int)K, (int)(rows / G), w->stride(0), s->stride(0), (int)G, (int)S,
        S > 1 ? x->stride(0) : G * K, rows, y.mutable_data_ptr(), stream_of(x));
    if (rc != 0) return failed("fp8_e4m3_gemv_batched", rc);
    return THPVariable_Wrap(std::move(y));
) }

// (shared, x, limit_gate, limit_up, out, workspace, stream)
FAST(fp8_shared_swiglu) { GUARD(
    ORDINARY(n == 7 && entry.fp8_e4m3_shared_swiglu_m1 && entry.fp8_e4m3_shared_swiglu_workspace_bytes && a[6] == Py_None);
    const Tensor *w1 = dense(get(a[0], kW1), kByte), *w3 = dense(get(a[0], kW3), kByte), *w2 = dense(get(a[0], kW2), kByte);
    const Tensor *s1 = dense(get(a[0], kW1s), kByte), *s3 = dense(get(a[0], kW3s), kByte), *s2 = dense(get(a[0], kW2s), kByte);
    const Tensor* x = dense(a[1], kBf16);
    ORDINARY(w1 && w3 && w2 && s1 && s3 && s2 && x && x->dim() == 1 && w1->dim() == 2 && w2->dim() == 2);
    const int64_t K = x->size(0), H = w1->size(0), O = w2->size(0);
    ORDINARY(shape(*w1, {H, K}) && shape(*w3, {H, K}) && shape(*w2, {O, H}) && shape(*s1, {H / 128, K / 128}) &&
             shape(*s3, {H / 128, K / 128}) && shape(*s2, {O / 128, H / 128}) && together({x, w1, w3, w2, s1, s3, s2}) && good_out(a[4], {O}, x) && reachable(a[5], x));
    ORDINARY(current(x));
    const double lg = PyFloat_AsDouble(a[2]), lu = PyFloat_AsDouble(a[3]);
    if (PyErr_Occurred()) return nullptr;
    const size_t need = fn<size_t (*)(int)>(entry.fp8_e4m3_shared_swiglu_workspace_bytes)((int)H);
    Tensor ws, made;
    if (a[5] == Py_None) {
        ws = empty({(int64_t)need}, kByte, x);
    } else {
        ws = THPVariable_Unpack(a[5]);
        ORDINARY(ws.is_cuda() && ws.nbytes() >= need);
    }
    void* y;
    if (a[4] == Py_None) { made = empty({O}, kBf16, x); y = made.mutable_data_ptr(); }
    else y = THPVariable_Unpack(a[4]).mutable_data_ptr();
    const int rc = call(fn<int (*)(P, P, P, P, P, P, P, int, int, int, float, float, void*, void*, void*)>(entry.fp8_e4m3_shared_swiglu_m1),
        ptr(x), ptr(w1), ptr(s1), ptr(w3), ptr(s3), ptr(w2), ptr(s2), (int)K, (int)H, (int)O, (float)lg, (float)lu, y,
        ws.mutable_data_ptr(), stream_of(x));
    if (rc != 0) return failed("fp8_e4m3_shared_swiglu_m1", rc);
    return result(a[4], std::move(made));
) }

struct Experts {
    const Tensor *p1, *p3, *p2, *s1, *s3, *s2;
    int64_t E, H, O;
    bool ok(const Tensor* x, int64_t K) {
        if (!p1 || !p3 || !p2 || !s1 || !s3 || !s2 || p1->dim() != 3 || p2->dim() != 3 || !together({x, p1, p3, p2, s1, s3, s2})) return false;
        E = p1->size(0); H = p1->size(1); O = p2->size(1);
        return shape(*p1, {E, H, K / 2}) && shape(*p3, {E, H, K / 2}) && shape(*s1, {E, H, K / 32}) && shape(*s3, {E, H, K / 32}) &&
               shape(*p2, {E, O, H / 2}) && shape(*s2, {E, O, H / 32});
    }
};
Experts bank_of(PyObject* d) {
    return {dense(get(d, kW1p), kByte), dense(get(d, kW3p), kByte), dense(get(d, kW2p), kByte), dense(get(d, kW1s), kByte),
            dense(get(d, kW3s), kByte), dense(get(d, kW2s), kByte), 0, 0, 0};
}
// Output and workspace as the operators take them: None = allocate; a given (reachable) tensor is used as it is.
void* take(PyObject* o, int64_t n, ScalarType type, const Tensor* like, Tensor& keep) {
    keep = o == Py_None ? empty({n}, type, like) : THPVariable_Unpack(o);
    return keep.mutable_data_ptr();
}
int score_of(PyObject* o) {
    if (!PyUnicode_Check(o)) return -1;
    return PyUnicode_CompareWithASCIIString(o, "softmax") == 0 ? 0 : PyUnicode_CompareWithASCIIString(o, "sqrt_softplus") == 0 ? 1 : -1;
}

// (W1, W3, W2, x, r, out, workspace)
FAST(grouped_gemv) { GUARD(
    ORDINARY(n == 7 && entry.mxfp4_grouped_gemv_topk && entry.mxfp4_grouped_workspace_bytes);
    Experts e = {dense(get(a[0], kPacked), kByte), dense(get(a[1], kPacked), kByte), dense(get(a[2], kPacked), kByte),
                 dense(get(a[0], kScale), kByte), dense(get(a[1], kScale), kByte), dense(get(a[2], kScale), kByte), 0, 0, 0};
    const Tensor *x = dense(a[3], kBf16), *r = dense(a[4], kF32);
    ORDINARY(x && r && e.ok(x, x->numel()) && shape(*r, {e.E}) && together({x, r}) && reachable(a[5], x) && reachable(a[6], x));
    ORDINARY(current(x));
    Tensor out, ws;
    void* y = take(a[5], e.O, kBf16, x, out);
    void* w = take(a[6], (int64_t)fn<size_t (*)(int, int, int)>(entry.mxfp4_grouped_workspace_bytes)((int)e.E, (int)e.H, (int)e.O), kByte, x, ws);
    const int rc = call(fn<int (*)(P, P, P, P, P, P, P, P, int, int, int, int, void*, void*, void*)>(entry.mxfp4_grouped_gemv_topk),
        ptr(x), ptr(e.p1), ptr(e.p3), ptr(e.p2), ptr(e.s1), ptr(e.s3), ptr(e.s2), ptr(r), (int)x->numel(), (int)e.H, (int)e.O,
        (int)e.E, y, w, stream_of(x));
    if (rc != 0) return failed("mxfp4_grouped_gemv_topk", rc);
    return result(a[5], std::move(out));
) }

// (bank, ids, x, r, out, workspace, stage_mask)
FAST(grouped_gemv_ids) { GUARD(
    ORDINARY(n == 7 && entry.mxfp4_grouped_gemv_topk_ids_stages && entry.mxfp4_grouped_workspace_bytes && PyLong_Check(a[6]));
    Experts e = bank_of(a[0]);
    const Tensor *ids = dense(a[1], kI32), *x = dense(a[2], kBf16), *r = dense(a[3], kF32);
    ORDINARY(ids && x && r && e.ok(x, x->numel()) && shape(*r, {ids->numel()}) && together({x, ids, r}) && reachable(a[4], x) && reachable(a[5], x));
    ORDINARY(current(x));
    Tensor out, ws;
    const int k = (int)ids->numel();
    void* y = take(a[4], e.O, kBf16, x, out);
    void* w = take(a[5], (int64_t)fn<size_t (*)(int, int, int)>(entry.mxfp4_grouped_workspace_bytes)(k, (int)e.H, (int)e.O), kByte, x, ws);
    const int rc = call(fn<int (*)(P, P, P, P, P, P, P, P, P, int, int, int, int, void*, void*, int, void*)>(entry.mxfp4_grouped_gemv_topk_ids_stages),
        ptr(x), ptr(e.p1), ptr(e.p3), ptr(e.p2), ptr(e.s1), ptr(e.s3), ptr(e.s2), ptr(ids), ptr(r), (int)x->numel(), (int)e.H,
        (int)e.O, k, y, w, (int)PyLong_AsLong(a[6]), stream_of(x));
    if (rc != 0) return failed("mxfp4_grouped_gemv_topk_ids", rc);
    return result(a[4], std::move(out));
) }

// (logits, k, score_func, eps, scaling, ids_out, w_out)
FAST(route_topk) { GUARD(
    ORDINARY(n == 7 && entry.mxfp4_moe_route_topk && PyLong_Check(a[1]));
    const Tensor* l = dense(a[0], kF32);
    const int func = score_of(a[2]);
    ORDINARY(l && func >= 0 && (l->dim() == 1 || l->dim() == 2));
    const int64_t T = l->dim() == 1 ? 1 : l->size(0), E = l->size(-1), k = PyLong_AsLong(a[1]);
    ORDINARY(k > 0);
    const double eps = PyFloat_AsDouble(a[3]), scaling = PyFloat_AsDouble(a[4]);
    if (PyErr_Occurred()) return nullptr;
    Tensor ids; Tensor w;
    ORDINARY(reachable(a[5], l) && reachable(a[6], l));
    ORDINARY(current(l));
    ids = a[5] == Py_None ? empty({T, k}, kI32, l) : THPVariable_Unpack(a[5]);
    w = a[6] == Py_None ? empty({T, k}, kF32, l) : THPVariable_Unpack(a[6]);
    const int rc = call(fn<int (*)(P, int, int, int, int, float, float, void*, void*, void*)>(entry.mxfp4_moe_route_topk),
        ptr(l), (int)T, (int)E, (int)k, func, (float)eps, (float)scaling, ids.mutable_data_ptr(), w.mutable_data_ptr(), stream_of(l));
    if (rc != 0) return failed("mxfp4_moe_route_topk", rc);
    PyObject* pair = PyTuple_New(2);
    PyTuple_SET_ITEM(pair, 0, result(a[5], std::move(ids)));
    PyTuple_SET_ITEM(pair, 1, result(a[6], std::move(w)));
    return pair;
) }

// (bank, logits, x, k, score_func, eps, scaling, out, workspace)
FAST(decode_layer) { GUARD(
    ORDINARY(n == 9 && entry.mxfp4_moe_decode_layer && entry.mxfp4_moe_decode_workspace_bytes && PyLong_Check(a[3]));
    Experts e = bank_of(a[0]);
    const Tensor *l = dense(a[1], kF32), *x = dense(a[2], kBf16);
    const int func = score_of(a[4]);
    ORDINARY(l && x && func >= 0 && e.ok(x, x->numel()) && l->numel() == e.E && together({x, l}) && reachable(a[7], x) && reachable(a[8], x));
    const int k = (int)PyLong_AsLong(a[3]);
    const double eps = PyFloat_AsDouble(a[5]), scaling = PyFloat_AsDouble(a[6]);
    if (PyErr_Occurred()) return nullptr;
    ORDINARY(k > 0);
    ORDINARY(current(x));
    Tensor out, ws;
    void* y = take(a[7], e.O, kBf16, x, out);
    void* w = take(a[8], (int64_t)fn<size_t (*)(int, int, int)>(entry.mxfp4_moe_decode_workspace_bytes)(k, (int)e.H, (int)e.O), kByte, x, ws);
    const int rc = call(fn<int (*)(P, P, P, P, P, P, P, P, int, int, float, float, int, int, int, int, void*, void*, void*)>(entry.mxfp4_moe_decode_layer),
        ptr(x), ptr(e.p1), ptr(e.p3), ptr(e.p2), ptr(e.s1), ptr(e.s3), ptr(e.s2), ptr(l), (int)e.E, func, (float)eps, (float)scaling,
        (int)x->numel(), (int)e.H, (int)e.O, k, y, w, stream_of(x));
    if (rc != 0) return failed("mxfp4_moe_decode_layer", rc);
    return result(a[7], std::move(out));
) }

// (bank, x, ids, weights, out, workspace, path: -1 = the library's default)
FAST(moe_forward) { GUARD(
    ORDINARY(n == 7 && entry.mxfp4_moe_forward && entry.mxfp4_moe_forward_path && entry.mxfp4_moe_forward_workspace_bytes && PyLong_Check(a[6]));
    Experts e = bank_of(a[0]);
    const Tensor *x = dense(a[1], kBf16), *ids = dense(a[2], kI32), *w = dense(a[3], kF32);
    ORDINARY(x && ids && w && x->dim() == 2 && ids->dim() == 2 && e.ok(x, x->size(1)) && together({x, ids, w}) && reachable(a[4], x) && reachable(a[5], x));
    ORDINARY(current(x));
    const int64_t T = x->size(0), K = x->size(1), k = ids->size(1);
    ORDINARY(shape(*ids, {T, k}) && shape(*w, {T, k}));
    Tensor out, ws;
    void *y, *wp;
    if (a[4] == Py_None) { out = empty({T, e.O}, kBf16, x); y = out.mutable_data_ptr(); }
    else y = THPVariable_Unpack(a[4]).mutable_data_ptr();
    if (a[5] == Py_None) {
        const size_t need = fn<size_t (*)(int, int, int, int, int, int)>(entry.mxfp4_moe_forward_workspace_bytes)((int)T, (int)k, (int)K, (int)e.H, (int)e.O, (int)e.E);
        ws = empty({(int64_t)need}, kByte, x);
    } else {
        ws = THPVariable_Unpack(a[5]);
    }
    wp = ws.mutable_data_ptr();
    const int path = (int)PyLong_AsLong(a[6]);
    int rc;
    if (path < 0)
        rc = call(fn<int (*)(P, P, P, P, P, P, P, P, P, int, int, int, int, int, int, void*, void*, void*)>(entry.mxfp4_moe_forward),
            ptr(x), ptr(e.p1), ptr(e.p3), ptr(e.p2), ptr(e.s1), ptr(e.s3), ptr(e.s2), ptr(ids), ptr(w), (int)T, (int)e.E, (int)K,
            (int)e.H, (int)e.O, (int)k, y, wp, stream_of(x));
    else
        rc = call(fn<int (*)(int, P, P, P, P, P, P, P, P, P, int, int, int, int, int, int, void*, void*, void*)>(entry.mxfp4_moe_forward_path),
            path, ptr(x), ptr(e.p1), ptr(e.p3), ptr(e.p2), ptr(e.s1), ptr(e.s3), ptr(e.s2), ptr(ids), ptr(w), (int)T, (int)e.E,
            (int)K, (int)e.H, (int)e.O, (int)k, y, wp, stream_of(x));
    if (rc != 0) return failed("mxfp4_moe_forward", rc);
    return result(a[4], std::move(out));
) }

PyMethodDef kMethods[] = {
#define DSV4_METHOD(n) {#n, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(n)), METH_FASTCALL, nullptr}
    DSV4_METHOD(bind), DSV4_METHOD(mxfp4_gemv), DSV4_METHOD(fp8_gemv), DSV4_METHOD(fp8_gemv_f32scale),
    DSV4_METHOD(fp8_gemv_batched), DSV4_METHOD(fp8_shared_swiglu), DSV4_METHOD(grouped_gemv), DSV4_METHOD(grouped_gemv_ids),
    DSV4_METHOD(route_topk), DSV4_METHOD(decode_layer), DSV4_METHOD(moe_forward), {nullptr, nullptr, 0, nullptr}
#undef DSV4_METHOD
};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "dsv4_host", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_dsv4_host(void) {
    const char* keys[] = {"w1p", "w3p", "w2p", "w1s", "w3s", "w2s", "w1", "w3", "w2", "packed", "scale"};
    for (int i = 0; i < 11; ++i) kKeys[i] = PyUnicode_InternFromString(keys[i]);
    return PyModule_Create(&kModule);
}
