// CPython entry points of the op front-ends: from tensors to the C ABI without a Python frame of checks.
//
// A small kernel of this library runs for 2-20 us; assembling its parameter block in Python (some
// forty attribute reads through ctypes) took 16-30 us per call on the host, so an eager call was bound
// by its own front-end. Each function here takes the arguments of one front-end in order, does the
// same checks on the C++ tensors, allocates the result and launches:
//   * it returns the result when the operands can go to the kernel as they are;
//   * it returns None, having launched nothing, for whatever needs a conversion, a copy or an error
//     message (autocast, odd alignments, ragged K, wrong shapes): the Python front-end then takes
//     its general path, which is the only place where those cases are handled.
// Measured (128 x 768 LayerNorm called back to back): 16.2 us per call through ctypes before.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/kernl_b200.h"

namespace {

bool is_none(PyObject* o) { return o == Py_None; }

// A CUDA tensor argument, or nullptr.
const at::Tensor* cuda_tensor(PyObject* o) {
    if (!THPVariable_Check(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    return t.is_cuda() ? &t : nullptr;
}

bool aligned16(const at::Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; }
bool is_16bit(at::ScalarType s) { return s == at::kHalf || s == at::kBFloat16; }
int32_t dtype_code(at::ScalarType s) { return s == at::kHalf ? KB_F16 : s == at::kBFloat16 ? KB_BF16 : KB_F32; }
bool like(const at::Tensor& t, const at::Tensor& ref) { return t.scalar_type() == ref.scalar_type() && t.device() == ref.device(); }
bool autocast_on() { return at::autocast::is_autocast_enabled(at::kCUDA); }

at::Tensor empty(at::IntArrayRef sizes, const at::Tensor& ref) {
    return at::detail::empty_cuda(sizes, ref.scalar_type(), ref.device(), c10::nullopt);
}

void* stream_of(const at::Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

PyObject* failed(const char* what, int status) {
    PyErr_Format(PyExc_RuntimeError, "kernl_b200: %s failed: %s (status %d)", what, kb_status_str(status), status);
    return nullptr;
}

// The GIL is given up around allocation and launch: a launch into a full queue blocks until the GPU has caught up, and a
// cudaMalloc for seconds, and a serving process has other threads to run meanwhile.
struct WithoutGil {
    PyThreadState* const state = PyEval_SaveThread();
    WithoutGil() = default;
    WithoutGil(const WithoutGil&) = delete;
    ~WithoutGil() { PyEval_RestoreThread(state); }
};

bool arity(Py_ssize_t got, Py_ssize_t want, const char* name) {
    if (got == want) return true;
    PyErr_Format(PyExc_TypeError, "%s takes %zd arguments, got %zd", name, want, got);
    return false;
}

// linear(x, weight, bias, activation_code, act_inputs, out) -> result or None
PyObject* linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (!arity(n, 6, "linear")) return nullptr;
    const at::Tensor *x = cuda_tensor(a[0]), *w = cuda_tensor(a[1]);
    const int act = (int)PyLong_AsLong(a[3]);
    if (act == -1 && PyErr_Occurred()) return nullptr;
    if (x == nullptr || w == nullptr || act < 0 || autocast_on()) Py_RETURN_NONE;
    const int64_t dim = x->dim();
    if (!is_16bit(x->scalar_type()) || !like(*w, *x) || w->dim() != 2 || (dim != 2 && dim != 3)) Py_RETURN_NONE;
    if (dim == 3 && !x->is_contiguous()) Py_RETURN_NONE;
    const int64_t K = x->size(dim - 1), M = dim == 2 ? x->size(0) : x->size(0) * x->size(1), N = w->size(0);
    const int64_t x_stride = dim == 2 ? x->stride(0) : K;
    if (M == 0 || K % 8 != 0 || x_stride % 8 != 0 || x->stride(dim - 1) != 1 || w->size(1) != K || !w->is_contiguous() ||
        !aligned16(*x) || !aligned16(*w))
        Py_RETURN_NONE;
    const at::Tensor* bias = nullptr;
    if (!is_none(a[2])) {
        bias = cuda_tensor(a[2]);
        if (bias == nullptr || !like(*bias, *x) || bias->dim() != 1 || bias->size(0) != N || !bias->is_contiguous() || !aligned16(*bias))
            Py_RETURN_NONE;
    }
    const bool gated = act == KB_ACT_SWIGLU;
    const int64_t n_out = gated ? N / 2 : N;
    const at::Tensor* pre = nullptr;
    if (!is_none(a[4])) {
        pre = cuda_tensor(a[4]);
        if (pre == nullptr || gated || !like(*pre, *x) || pre->dim() != 2 || pre->size(0) != M || pre->size(1) != N || !pre->is_contiguous())
            Py_RETURN_NONE;
    }
    if (gated && N % 16 != 0) Py_RETURN_NONE;
    at::Tensor y;
    if (!is_none(a[5])) {
        const at::Tensor* out = cuda_tensor(a[5]);
        if (out == nullptr || dim != 2 || !like(*out, *x) || out->dim() != 2 || out->size(0) != M || out->size(1) != n_out || out->stride(1) != 1)
            Py_RETURN_NONE;
        y = *out;
    }
    kb_linear_params p{};
    p.x = x->data_ptr();
    p.w = w->data_ptr();
    p.bias = bias != nullptr ? bias->data_ptr() : nullptr;
    p.act_inputs = pre != nullptr ? pre->data_ptr() : nullptr;
    p.M = M;
    p.N = N;
    p.K = K;
    p.x_row_stride = x_stride;
    p.activation = act;
    p.dtype = dtype_code(x->scalar_type());
    int st;
    {
        const WithoutGil unlocked;
        const c10::cuda::CUDAGuard guard(x->device());
        if (!y.defined()) y = dim == 2 ? empty({M, n_out}, *x) : empty({x->size(0), x->size(1), n_out}, *x);
        p.y = y.data_ptr();
        p.y_row_stride = dim == 2 ? y.stride(0) : n_out;
        st = kb_linear_fwd(&p, stream_of(*x));
    }
    if (st != KB_OK) return failed("linear_layer", st);
    return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

// layer_norm(x, weight, bias, eps, use_rms_norm, residual, out, with_sum) -> result, (result, sum) or None;
// with_sum false: the sum of x and the residual is normalised but not stored, and only the result is returned
PyObject* layer_norm(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (!arity(n, 8, "layer_norm")) return nullptr;
    const at::Tensor *x = cuda_tensor(a[0]), *w = cuda_tensor(a[1]);
    const double eps = PyFloat_AsDouble(a[3]);
    if (eps == -1.0 && PyErr_Occurred()) return nullptr;
    const int rms = PyObject_IsTrue(a[4]), with_sum = PyObject_IsTrue(a[7]);
    if (rms < 0 || with_sum < 0) return nullptr;
    if (x == nullptr || w == nullptr || autocast_on() || x->dim() == 0) Py_RETURN_NONE;
    const int64_t dim = x->dim(), cols = x->size(dim - 1);
    if (!is_16bit(x->scalar_type()) || !like(*w, *x) || w->numel() != cols || w->dim() != 1 || !w->is_contiguous() || !aligned16(*w) ||
        !x->is_contiguous() || x->numel() == 0)
        Py_RETURN_NONE;
    const at::Tensor *bias = nullptr, *residual = nullptr;
    if (!is_none(a[2])) {
        bias = cuda_tensor(a[2]);
        if (bias == nullptr || !like(*bias, *x) || bias->numel() != cols || !bias->is_contiguous() || !aligned16(*bias)) Py_RETURN_NONE;
    }
    if (!is_none(a[5])) {
        residual = cuda_tensor(a[5]);
        if (residual == nullptr || !like(*residual, *x) || !residual->sizes().equals(x->sizes()) || !residual->is_contiguous() ||
            !aligned16(*residual))
            Py_RETURN_NONE;
    }
    at::Tensor y, sum;
    if (!is_none(a[6])) {
        const at::Tensor* out = cuda_tensor(a[6]);
        if (out == nullptr || !like(*out, *x) || !out->sizes().equals(x->sizes()) || !out->is_contiguous()) Py_RETURN_NONE;
        y = *out;
    }
    kb_norm_params p{};
    p.x = x->data_ptr();
    p.gamma = w->data_ptr();
    p.beta = bias != nullptr ? bias->data_ptr() : nullptr;
    p.rows = x->numel() / cols;
    p.cols = cols;
    p.x_row_stride = p.y_row_stride = cols;
    p.x_col_stride = p.y_col_stride = 1;
    p.eps = (float)(x->scalar_type() == at::kHalf && eps < 1.6e-5 ? 1.6e-5 : eps);
    p.is_rms = rms;
    p.dtype = dtype_code(x->scalar_type());
    p.residual = residual != nullptr ? residual->data_ptr() : nullptr;
    int st;
    {
        const WithoutGil unlocked;
        const c10::cuda::CUDAGuard guard(x->device());
        if (!y.defined()) y = empty(x->sizes(), *x);
        if (residual != nullptr && with_sum) sum = empty(x->sizes(), *x);
        p.y = y.data_ptr();
        p.sum_out = sum.defined() ? sum.data_ptr() : nullptr;
        st = kb_norm_fwd(&p, stream_of(*x));
    }
    if (st != KB_OK) return failed("layer_norm", st);
    if (!sum.defined()) return THPVariable_Wrap(std::move(y));
    PyObject* pair = PyTuple_New(2);
    if (pair == nullptr) return nullptr;
    PyTuple_SET_ITEM(pair, 0, THPVariable_Wrap(std::move(y)));
    PyTuple_SET_ITEM(pair, 1, THPVariable_Wrap(std::move(sum)));
    return pair;
    END_HANDLE_TH_ERRORS
}

// Fills the parameters shared by the two attention entries from (q, k, v, output, sm_scale, is_causal,
// mask). 1: filled, 0: not a case for this path, -1: a Python error is set.
int attention_params(PyObject* const* a, kb_attn_params& p, const at::Tensor*& q) {
    q = cuda_tensor(a[0]);
    const at::Tensor *k = cuda_tensor(a[1]), *v = cuda_tensor(a[2]), *o = cuda_tensor(a[3]);
    const double scale = PyFloat_AsDouble(a[4]);
    if (scale == -1.0 && PyErr_Occurred()) return -1;
    const int causal = PyObject_IsTrue(a[5]);
    if (causal < 0) return -1;
    if (q == nullptr || k == nullptr || v == nullptr || o == nullptr || autocast_on()) return 0;
    if (!is_16bit(q->scalar_type()) || !like(*k, *q) || !like(*v, *q) || !like(*o, *q)) return 0;
    if (q->dim() != 4 || k->dim() != 4 || v->dim() != 4 || !o->sizes().equals(q->sizes()) || !v->sizes().equals(k->sizes())) return 0;
    const int64_t B = q->size(0), H = q->size(1), M = q->size(2), D = q->size(3), HK = k->size(1), N = k->size(2);
    if (k->size(0) != B || k->size(3) != D || HK <= 0 || H % HK != 0) return 0;
    p.q = q->data_ptr();
    p.k = k->data_ptr();
    p.v = v->data_ptr();
    p.o = o->data_ptr();
    p.B = B;
    p.H = H;
    p.M = M;
    p.N = N;
    p.D = D;
    p.kv_group = (int32_t)(H / HK);
    for (int i = 0; i < 4; ++i) {
        p.q_strides[i] = q->stride(i);
        p.k_strides[i] = k->stride(i);
        p.v_strides[i] = v->stride(i);
        p.o_strides[i] = o->stride(i);
    }
    p.mask_dtype = KB_F32;
    if (!is_none(a[6])) {
        const at::Tensor* m = cuda_tensor(a[6]);
        if (m == nullptr || m->device() != q->device() || m->dim() != 4 || (!is_16bit(m->scalar_type()) && m->scalar_type() != at::kFloat)) return 0;
        const int64_t full[4] = {B, H, M, N};
        for (int i = 0; i < 4; ++i) {
            if (m->size(i) != full[i] && (i == 3 || m->size(i) != 1)) return 0;
            p.mask_strides[i] = m->size(i) > 1 ? m->stride(i) : 0;  // a broadcast dimension never advances
        }
        p.mask = m->data_ptr();
        p.mask_dtype = dtype_code(m->scalar_type());
    }
    p.sm_scale = (float)scale;
    p.is_causal = causal;
    p.dtype = dtype_code(q->scalar_type());
    return 1;
}

// attention(q, k, v, output, sm_scale, is_causal, mask) -> output or None
PyObject* attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (!arity(n, 7, "attention")) return nullptr;
    kb_attn_params p{};
    const at::Tensor* q;
    const int filled = attention_params(a, p, q);
    if (filled < 0) return nullptr;
    if (filled == 0 || p.D % 8 != 0 || p.D > 128) Py_RETURN_NONE;
    // tensor maps: unit stride on the head dimension, 16-byte aligned rows and base
    const int64_t* strides[3] = {p.q_strides, p.k_strides, p.v_strides};
    const void* bases[3] = {p.q, p.k, p.v};
    for (int t = 0; t < 3; ++t) {
        const int64_t sizes[3] = {p.B, t == 0 ? p.H : p.H / p.kv_group, t == 0 ? p.M : p.N};
        if (strides[t][3] != 1 || (reinterpret_cast<uintptr_t>(bases[t]) & 15) != 0) Py_RETURN_NONE;
        for (int i = 0; i < 3; ++i)
            if (sizes[i] > 1 && strides[t][i] % 8 != 0) Py_RETURN_NONE;
    }
    int st;
    {
        const WithoutGil unlocked;
        const c10::cuda::CUDAGuard guard(q->device());
        st = kb_attention_fwd(&p, stream_of(*q));
    }
    if (st != KB_OK) return failed("attention_forward", st);
    Py_INCREF(a[3]);
    return a[3];
    END_HANDLE_TH_ERRORS
}

// decode_attention(q, k, v, output, sm_scale, is_causal, mask, kv_len) -> output or None
PyObject* decode_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (!arity(n, 8, "decode_attention")) return nullptr;
    kb_attn_params p{};
    const at::Tensor* q;
    const int filled = attention_params(a, p, q);
    if (filled < 0) return nullptr;
    if (filled == 0 || p.D > 256) Py_RETURN_NONE;
    if (!is_none(a[7])) {
        const at::Tensor* len = cuda_tensor(a[7]);
        if (len == nullptr || len->scalar_type() != at::kLong || len->numel() != 1 || len->device() != q->device()) Py_RETURN_NONE;
        p.kv_len_dev = len->data_ptr<int64_t>();
    }
    int st;
    {
        const WithoutGil unlocked;
        const c10::cuda::CUDAGuard guard(q->device());
        st = kb_attention_decode_fwd(&p, nullptr, 0, stream_of(*q));
    }
    if (st == KB_ERR_BAD_ARG) Py_RETURN_NONE;  // a layout that needs scratch, which the general path allocates
    if (st != KB_OK) return failed("skinny_attention_forward", st);
    Py_INCREF(a[3]);
    return a[3];
    END_HANDLE_TH_ERRORS
}

// The caches, tables and position of a rotary embedding with cache write: false for what the Python front-end has to look at.
// a: k_cache, v_cache, cos, sin, pos, batch, seq
bool rope_args(PyObject* const* a, const at::Tensor& like_this, kb_rope_params& p) {
    const at::Tensor* t[4];
    for (int i = 0; i < 4; ++i)
        if ((t[i] = cuda_tensor(a[i])) == nullptr || t[i]->device() != like_this.device() || !t[i]->is_contiguous()) return false;
    const at::Tensor &kc = *t[0], &vc = *t[1], &cos = *t[2], &sin = *t[3];
    if (!is_16bit(like_this.scalar_type()) || !like(kc, like_this) || !like(vc, like_this) || cos.scalar_type() != at::kFloat ||
        sin.scalar_type() != at::kFloat)
        return false;
    p.B = PyLong_AsLongLong(a[5]);
    p.S = PyLong_AsLongLong(a[6]);
    if (PyErr_Occurred()) return false;
    if (kc.dim() != 4 || kc.size(0) != p.B || !vc.sizes().equals(kc.sizes())) return false;
    p.H = kc.size(1);
    p.max_seq = kc.size(2);
    p.D = kc.size(3);
    if (!cos.sizes().equals({p.max_seq, p.D / 2}) || !sin.sizes().equals(cos.sizes())) return false;
    if (PyLong_Check(a[4])) {
        p.pos_host = PyLong_AsLongLong(a[4]);
        if (p.pos_host == -1 && PyErr_Occurred()) return false;
    } else {
        const at::Tensor* pos = cuda_tensor(a[4]);
        if (pos == nullptr || pos->scalar_type() != at::kLong || pos->numel() != 1 || pos->device() != like_this.device()) return false;
        p.pos_dev = pos->data_ptr<int64_t>();
    }
    p.k_cache = kc.data_ptr();
    p.v_cache = vc.data_ptr();
    p.cos = cos.data_ptr<float>();
    p.sin = sin.data_ptr<float>();
    p.dtype = dtype_code(like_this.scalar_type());
    return true;
}

// rope_kv_write(qkv, k_cache, v_cache, cos, sin, pos, batch, seq) -> rotated q or None
PyObject* rope_kv_write(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (!arity(n, 8, "rope_kv_write")) return nullptr;
    const at::Tensor* qkv = cuda_tensor(a[0]);
    kb_rope_params p{};
    if (qkv == nullptr || !qkv->is_contiguous() || !rope_args(a + 1, *qkv, p)) {
        if (PyErr_Occurred()) return nullptr;
        Py_RETURN_NONE;
    }
    if (qkv->dim() != 2 || qkv->size(0) != p.B * p.S || qkv->size(1) != 3 * p.H * p.D) Py_RETURN_NONE;
    p.qkv = qkv->data_ptr();
    at::Tensor q;
    int st;
    {
        const WithoutGil unlocked;
        const c10::cuda::CUDAGuard guard(qkv->device());
        q = empty({p.B, p.S, p.H, p.D}, *qkv);
        p.q_out = q.data_ptr();
        st = kb_rope_kv_write(&p, stream_of(*qkv));
    }
    if (st != KB_OK) return failed("rope_kv_write", st);
    return THPVariable_Wrap(std::move(q));
    END_HANDLE_TH_ERRORS
}

// linear_rope_kv_write(x, weight, k_cache, v_cache, cos, sin, pos, batch, seq) -> rotated q or None
PyObject* linear_rope_kv_write(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (!arity(n, 9, "linear_rope_kv_write")) return nullptr;
    const at::Tensor *x = cuda_tensor(a[0]), *w = cuda_tensor(a[1]);
    kb_rope_params p{};
    if (x == nullptr || w == nullptr || autocast_on() || !rope_args(a + 2, *x, p)) {
        if (PyErr_Occurred()) return nullptr;
        Py_RETURN_NONE;
    }
    if (!like(*w, *x) || w->dim() != 2 || x->dim() != 2) Py_RETURN_NONE;
    const int64_t M = x->size(0), K = x->size(1), N = w->size(0);
    if (M == 0 || K % 8 != 0 || x->stride(0) % 8 != 0 || x->stride(1) != 1 || w->size(1) != K || !w->is_contiguous() || !aligned16(*x) ||
        !aligned16(*w) || M != p.B * p.S || N != 3 * p.H * p.D)
        Py_RETURN_NONE;
    kb_linear_params l{};
    l.x = x->data_ptr();
    l.w = w->data_ptr();
    l.M = M;
    l.N = N;
    l.K = K;
    l.x_row_stride = x->stride(0);
    l.y_row_stride = N;
    l.dtype = p.dtype;
    at::Tensor q;
    int st;
    {
        const WithoutGil unlocked;
        const c10::cuda::CUDAGuard guard(x->device());
        q = empty({p.B, p.S, p.H, p.D}, *x);
        const at::Tensor qkv = empty({M, N}, *x);  // (on this stream: given back to it when the launches are queued)
        p.q_out = q.data_ptr();
        l.y = qkv.data_ptr();
        st = kb_linear_rope_kv_write(&l, &p, stream_of(*x));
    }
    if (st != KB_OK) return failed("linear_rope_kv_write", st);
    return THPVariable_Wrap(std::move(q));
    END_HANDLE_TH_ERRORS
}

#define KB_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {KB_METHOD(linear), KB_METHOD(layer_norm), KB_METHOD(attention),
                         KB_METHOD(decode_attention), KB_METHOD(rope_kv_write), KB_METHOD(linear_rope_kv_write), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host_ops", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host_ops() { return PyModule_Create(&module); }
