// The operators of mimir_b200/tensor.py for the calls that programs are made of: contiguous CUDA tensors of the right shapes and
// element types. A call is taken from the Python arguments to the C ABI here, about 3 us of host time instead of 9 through ctypes.
//
// Every function returns the result, or None for any call it is not made for (another type or subclass, layout, device or shape, a dispatch mode
// or a transform that is active, a status that is not OK): the caller then takes the general path, which makes copies and raises errors.
// tensor.py alone says what an operator means; nothing is accepted here that it would refuse.
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "mimk.h"

namespace {

using at::Tensor;

// No transform or mode wants to see the operations (functorch, tracing, fake tensors ...), nor __torch_function__. Inference mode,
// which takes one key from the default set, does not: what is allocated in it becomes an inference tensor by itself.
bool nothing_watches() {
    const auto tls = c10::impl::tls_local_dispatch_key_set();
    return tls.included_.add(c10::DispatchKey::ADInplaceOrView) == c10::default_included_set && !c10::impl::TorchDispatchModeTLS::any_modes_set() && !at::impl::torch_function_mode_enabled();
}

int dtype_of(at::ScalarType t) { return t == at::kFloat ? MIMK_F32 : t == at::kBFloat16 ? MIMK_BF16 : -1; }

PyTypeObject* parameter_type;  // torch.nn.Parameter, for the life of the module

// A torch.Tensor or torch.nn.Parameter proper, dense and row-major on a CUDA device, of F32 or BF16 elements; null if not.
const Tensor* dense(PyObject* o, bool any_strides = false) {
    if (Py_TYPE(o) != reinterpret_cast<PyTypeObject*>(THPVariableClass) && Py_TYPE(o) != parameter_type) return nullptr;
    const Tensor& t = THPVariable_Unpack(o);
    if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || !t.has_storage() || t.is_neg() || dtype_of(t.scalar_type()) < 0) return nullptr;
    if (t.key_set().has_any(c10::DispatchKeySet({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                                 c10::DispatchKey::Functionalize, c10::DispatchKey::ZeroTensor})))
        return nullptr;
    if (t.numel() == 0 || (!any_strides && !t.is_contiguous())) return nullptr;
    return &t;
}

bool is_int(PyObject* o, int64_t& v) {
    if (!PyLong_CheckExact(o)) return false;
    v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    return true;
}
// None: `plain`; a dtype of F32 or BF16: that one
bool out_type(PyObject* o, at::ScalarType plain, at::ScalarType& t) {
    if (o == Py_None) {
        t = plain;
        return true;
    }
    if (!THPDtype_Check(o)) return false;
    t = reinterpret_cast<THPDtype*>(o)->scalar_type;
    return dtype_of(t) >= 0;
}

Tensor empty(at::IntArrayRef shape, at::ScalarType t, const Tensor& like) { return at::detail::empty_cuda(shape, t, like.device(), std::nullopt); }
// The call into the library, f(stream), without the interpreter's lock: it may wait, for the device where a cached buffer grows, or for room
// in a launch queue, and what it waits for may be another Python thread's to issue.
template <class F>
int unlocked(F&& f) {
    void* stream         = c10::cuda::getCurrentCUDAStream().stream();
    PyThreadState* state = PyEval_SaveThread();
    const int status     = f(stream);
    PyEval_RestoreThread(state);
    return status;
}
PyObject* result(int status, Tensor&& out) {
    if (status != MIMK_OK) Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(out));
}

// B of a product, [..., k, n]: row-major, or a transposed view of a row-major [..., n, k].
int b_layout(const Tensor& b) {
    if (b.is_contiguous()) return MIMK_B_KN;
    const int64_t r = b.dim(), k = b.size(r - 2), n = b.size(r - 1);
    if ((k != 1 && b.stride(r - 2) != 1) || (n != 1 && b.stride(r - 1) != k)) return -1;
    if (r == 3 && b.size(0) != 1 && b.stride(0) != k * n) return -1;
    return MIMK_B_NK;
}

struct View3 {  // the axes before, at and behind `ax`
    int64_t outer = 1, len = 1, inner = 1;
    int64_t ax;
    View3(const Tensor& x, int64_t axis) : ax(axis < 0 ? axis + x.dim() : axis) {
        for (int64_t i = 0; i < x.dim(); ++i) (i < ax ? outer : i == ax ? len : inner) *= x.size(i);
    }
    bool good(const Tensor& x) const { return ax >= 0 && ax < x.dim(); }
};
std::vector<int64_t> without(const Tensor& x, int64_t ax) {
    std::vector<int64_t> s(x.sizes().begin(), x.sizes().end());
    s.erase(s.begin() + ax);
    return s;
}

#define OP(NAME, N)                                                                   \
    PyObject* NAME(PyObject*, PyObject* const* a, Py_ssize_t n) {                     \
        HANDLE_TH_ERRORS                                                              \
        if (n != N || !nothing_watches()) Py_RETURN_NONE;
#define END_OP          \
    Py_RETURN_NONE;     \
    END_HANDLE_TH_ERRORS \
    }

// a, b, post id, bias, out dtype
OP(product_2d, 5)
    const Tensor *x = dense(a[0]), *w = dense(a[1], true), *bias = a[3] == Py_None ? nullptr : dense(a[3]);
    int64_t post;
    at::ScalarType t;
    if (!x || !w || (!bias && a[3] != Py_None) || !is_int(a[2], post) || x->dim() != 2 || w->dim() != 2 || x->scalar_type() != w->scalar_type()) Py_RETURN_NONE;
    const int64_t m = x->size(0), k = x->size(1), cols = w->size(1);
    const int layout = b_layout(*w);
    if (k != w->size(0) || layout < 0 || !out_type(a[4], x->scalar_type(), t)) Py_RETURN_NONE;
    if (bias && (bias->scalar_type() != at::kFloat || bias->numel() != cols)) Py_RETURN_NONE;
    Tensor out = empty({m, cols}, t, *x);
    mimk_gemm_desc d = {};
    d.batch = 1, d.m = m, d.n = cols, d.k = k, d.stride_c = m * cols;
    d.a = x->data_ptr(), d.b = w->data_ptr(), d.c = out.data_ptr();
    d.in_dtype = dtype_of(x->scalar_type()), d.out_dtype = dtype_of(t), d.b_layout = layout, d.post = int(post);
    d.post_row = bias ? bias->data_ptr() : nullptr;
    return result(unlocked([&](void* stream) { return mimk_gemm(&d, stream); }), std::move(out));
END_OP

// a, b, out dtype
OP(bmm, 3)
    const Tensor *x = dense(a[0]), *w = dense(a[1], true);
    at::ScalarType t;
    if (!x || !w || x->dim() != 3 || w->dim() != 3 || x->scalar_type() != w->scalar_type()) Py_RETURN_NONE;
    const int64_t batch = x->size(0), m = x->size(1), k = x->size(2), cols = w->size(2);
    const int layout = b_layout(*w);
    if (batch != w->size(0) || k != w->size(1) || layout < 0 || !out_type(a[2], x->scalar_type(), t)) Py_RETURN_NONE;
    Tensor out = empty({batch, m, cols}, t, *x);
    mimk_gemm_desc d = {};
    d.batch = batch, d.m = m, d.n = cols, d.k = k, d.stride_a = m * k, d.stride_b = k * cols, d.stride_c = m * cols;
    d.a = x->data_ptr(), d.b = w->data_ptr(), d.c = out.data_ptr();
    d.in_dtype = dtype_of(x->scalar_type()), d.out_dtype = dtype_of(t), d.b_layout = layout, d.post = MIMK_POST_ID;
    return result(unlocked([&](void* stream) { return mimk_gemm(&d, stream); }), std::move(out));
END_OP

// monoid id, axis, x
OP(reduce, 3)
    const Tensor* x = dense(a[2]);
    int64_t monoid, ax;
    if (!x || !is_int(a[0], monoid) || !is_int(a[1], ax)) Py_RETURN_NONE;
    const View3 v(*x, ax);
    if (!v.good(*x)) Py_RETURN_NONE;
    Tensor out = empty(without(*x, v.ax), x->scalar_type(), *x);
    return result(unlocked([&](void* stream) { return mimk_reduce(x->data_ptr(), out.data_ptr(), dtype_of(x->scalar_type()), v.outer, v.len, v.inner, int(monoid), stream); }), std::move(out));
END_OP

// monoid id, axis, x, unary inner id, unary outer id
OP(reduce_of_unary, 5)
    const Tensor* x = dense(a[2]);
    int64_t monoid, ax, inner, outer;
    if (!x || !is_int(a[0], monoid) || !is_int(a[1], ax) || !is_int(a[3], inner) || !is_int(a[4], outer)) Py_RETURN_NONE;
    const View3 v(*x, ax);
    if (!v.good(*x)) Py_RETURN_NONE;
    mimk_producer pre = {};
    pre.inner_op = int32_t(inner), pre.outer_op = int32_t(outer), pre.y_mode = 3;
    Tensor out = empty(without(*x, v.ax), x->scalar_type(), *x);
    return result(unlocked([&](void* stream) { return mimk_reduce_fused(x->data_ptr(), &pre, out.data_ptr(), dtype_of(x->scalar_type()), v.outer, v.len, v.inner, int(monoid), stream); }),
                  std::move(out));
END_OP

// axis, x, out dtype
OP(softmax, 3)
    const Tensor* x = dense(a[1]);
    int64_t ax;
    at::ScalarType t;
    if (!x || !is_int(a[0], ax) || !out_type(a[2], x->scalar_type(), t)) Py_RETURN_NONE;
    const View3 v(*x, ax);
    if (!v.good(*x)) Py_RETURN_NONE;
    Tensor out = empty(x->sizes(), t, *x);
    return result(unlocked([&](void* stream) { return mimk_softmax(x->data_ptr(), out.data_ptr(), dtype_of(x->scalar_type()), dtype_of(t), v.outer, v.len, v.inner, stream); }), std::move(out));
END_OP

// x, gamma, eps, out dtype
OP(rmsnorm, 4)
    const Tensor *x = dense(a[0]), *gamma = dense(a[1]);
    at::ScalarType t;
    if (!x || !gamma || x->dim() < 1 || gamma->scalar_type() != at::kFloat || !PyFloat_CheckExact(a[2]) || !out_type(a[3], x->scalar_type(), t)) Py_RETURN_NONE;
    const int64_t cols = x->size(x->dim() - 1);
    if (gamma->numel() != cols) Py_RETURN_NONE;
    Tensor out = empty(x->sizes(), t, *x);
    return result(unlocked([&](void* stream) { return mimk_rmsnorm(x->data_ptr(), gamma->data_ptr(), out.data_ptr(), dtype_of(x->scalar_type()), dtype_of(t), x->numel() / cols, cols,
                               float(PyFloat_AS_DOUBLE(a[2])), stream); }),
                  std::move(out));
END_OP

// op id, x, out dtype
OP(unary, 3)
    const Tensor* x = dense(a[1]);
    int64_t op;
    at::ScalarType t;
    if (!x || !is_int(a[0], op) || !out_type(a[2], x->scalar_type(), t)) Py_RETURN_NONE;
    Tensor out = empty(x->sizes(), t, *x);
    return result(unlocked([&](void* stream) { return mimk_map_t(int(op), x->data_ptr(), nullptr, out.data_ptr(), dtype_of(x->scalar_type()), dtype_of(t), 1, x->numel(), 1, 3, stream); }),
                  std::move(out));
END_OP

// op id, x, y, out dtype
OP(binary, 4)
    const Tensor *x = dense(a[1]), *y = dense(a[2]);
    int64_t op;
    at::ScalarType t;
    if (!x || !y || !is_int(a[0], op) || x->scalar_type() != y->scalar_type() || x->sizes() != y->sizes() || !out_type(a[3], x->scalar_type(), t)) Py_RETURN_NONE;
    Tensor out = empty(x->sizes(), t, *x);
    return result(unlocked([&](void* stream) { return mimk_map_t(int(op), x->data_ptr(), y->data_ptr(), out.data_ptr(), dtype_of(x->scalar_type()), dtype_of(t), 1, x->numel(), 1, 0, stream); }),
                  std::move(out));
END_OP

// op id, axis, x, y, out dtype
OP(binary_ax, 5)
    const Tensor *x = dense(a[2]), *y = dense(a[3]);
    int64_t op, ax;
    at::ScalarType t;
    if (!x || !y || !is_int(a[0], op) || !is_int(a[1], ax) || x->scalar_type() != y->scalar_type() || !out_type(a[4], x->scalar_type(), t)) Py_RETURN_NONE;
    const View3 v(*x, ax);
    if (!v.good(*x) || y->sizes() != at::IntArrayRef(without(*x, v.ax))) Py_RETURN_NONE;
    Tensor out = empty(x->sizes(), t, *x);
    return result(unlocked([&](void* stream) { return mimk_map_t(int(op), x->data_ptr(), y->data_ptr(), out.data_ptr(), dtype_of(x->scalar_type()), dtype_of(t), v.outer, v.len, v.inner, 1, stream); }),
                  std::move(out));
END_OP

// q, k, v, scale, causal
OP(attention, 5)
    const Tensor *q = dense(a[0]), *k = dense(a[1]), *v = dense(a[2]);
    if (!q || !k || !v || !PyFloat_CheckExact(a[3]) || !PyBool_Check(a[4])) Py_RETURN_NONE;
    const int64_t r = q->dim();
    if (r < 2 || k->dim() != r || k->sizes() != v->sizes() || q->size(r - 1) != k->size(r - 1)) Py_RETURN_NONE;
    if (q->scalar_type() != k->scalar_type() || q->scalar_type() != v->scalar_type()) Py_RETURN_NONE;
    mimk_attn_desc d = {};
    d.batch_heads = 1;
    for (int64_t i = 0; i < r - 2; ++i) {
        if (q->size(i) != k->size(i)) Py_RETURN_NONE;
        d.batch_heads *= q->size(i);
    }
    Tensor out = empty(q->sizes(), q->scalar_type(), *q);
    d.seq_q = q->size(r - 2), d.seq_k = k->size(r - 2), d.head_dim = q->size(r - 1);
    d.q = q->data_ptr(), d.k = k->data_ptr(), d.v = v->data_ptr(), d.o = out.data_ptr();
    d.scale = float(PyFloat_AS_DOUBLE(a[3])), d.causal = a[4] == Py_True, d.dtype = dtype_of(q->scalar_type());
    return result(unlocked([&](void* stream) { return mimk_attn_fwd(&d, stream); }), std::move(out));
END_OP

// x, w1, w3, w2
OP(mlp_gated, 4)
    const Tensor *x = dense(a[0]), *w1 = dense(a[1], true), *w3 = dense(a[2], true), *w2 = dense(a[3], true);
    if (!x || !w1 || !w3 || !w2 || x->dim() != 2 || w1->dim() != 2 || w2->dim() != 2 || w1->sizes() != w3->sizes()) Py_RETURN_NONE;
    const at::ScalarType t = x->scalar_type();
    if (w1->scalar_type() != t || w3->scalar_type() != t || w2->scalar_type() != t) Py_RETURN_NONE;
    const int layout = b_layout(*w1);
    if (layout < 0 || b_layout(*w3) != layout || b_layout(*w2) != layout || x->size(1) != w1->size(0) || w1->size(1) != w2->size(0)) Py_RETURN_NONE;
    mimk_mlp_desc d = {};
    d.m = x->size(0), d.k = x->size(1), d.f = w1->size(1), d.n = w2->size(1);
    Tensor out = empty({d.m, d.n}, t, *x);
    d.x = x->data_ptr(), d.w1 = w1->data_ptr(), d.w3 = w3->data_ptr(), d.w2 = w2->data_ptr(), d.y = out.data_ptr();
    d.dtype = dtype_of(t), d.b_layout = layout;
    return result(unlocked([&](void* stream) { return mimk_mlp_gated(&d, stream); }), std::move(out));
END_OP

// x, perm (a tuple of ints): the copy-style map_reduce_post that tensor.py's transpose spells
OP(transpose, 2)
    const Tensor* x = dense(a[0]);
    if (!x || !PyTuple_CheckExact(a[1]) || PyTuple_GET_SIZE(a[1]) != x->dim() || x->dim() > MIMK_MRP_MAX_RANK) Py_RETURN_NONE;
    const int r = int(x->dim());
    mimk_mrp_desc d = {};
    std::vector<int64_t> shape(r);
    bool seen[MIMK_MRP_MAX_RANK] = {};
    d.ro = d.rn = r, d.nis = 1;
    d.in_map[0].rows = d.map_out.rows = r;
    for (int i = 0; i < r; ++i) {
        int64_t p;
        if (!is_int(PyTuple_GET_ITEM(a[1], i), p) || p < 0 || p >= r || seen[p]) Py_RETURN_NONE;
        seen[p] = true, shape[i] = d.sr[i] = d.so[i] = x->size(p);
        d.in_map[0].coef[p][i] = 1, d.map_out.coef[i][i] = 1, d.in_shape[0][i] = x->size(i);
    }
    Tensor out = empty(shape, x->scalar_type(), *x);
    d.in[0] = x->data_ptr(), d.in_dtype[0] = d.out_dtype = dtype_of(x->scalar_type()), d.acc_dtype = MIMK_F32;
    d.comb = MIMK_F_FIRST, d.post = MIMK_P_ID, d.out = out.data_ptr();
    return result(unlocked([&](void* stream) { return mimk_map_reduce_post(&d, stream); }), std::move(out));
END_OP

PyMethodDef methods[] = {
#define ENTRY(NAME) {#NAME, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(NAME)), METH_FASTCALL, nullptr}
    ENTRY(product_2d), ENTRY(bmm), ENTRY(reduce), ENTRY(reduce_of_unary), ENTRY(softmax), ENTRY(rmsnorm), ENTRY(unary), ENTRY(binary), ENTRY(binary_ax),
    ENTRY(attention), ENTRY(mlp_gated), ENTRY(transpose), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__native() {
    PyObject* nn = PyImport_ImportModule("torch.nn.parameter");
    if (!nn) return nullptr;
    parameter_type = reinterpret_cast<PyTypeObject*>(PyObject_GetAttrString(nn, "Parameter"));
    Py_DECREF(nn);
    return parameter_type ? PyModule_Create(&module) : nullptr;
}
