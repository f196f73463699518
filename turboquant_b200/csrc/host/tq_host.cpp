// Host side of the calls a decode step makes, as a CPython extension.
//
// A decode step is two or three kernel launches of a few microseconds each; the same step driven through
// torch slicing, ctypes argument structures and per-step length tensors costs 20-80 us of Python.  The
// functions here take the tensors as they are, check what the Python wrappers checked, fill the C argument
// block and launch: about 1 us of their own per call.
//
// Every function is a fast path: what it does not take (another device, another layout, a shape the
// wrappers refuse with a message) it answers with None / NotImplemented-like results BEFORE anything is
// launched, and the Python wrapper goes its general way.  Status codes of the library come back as ints.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <vector>

#include "turboquant_b200.h"

namespace {

// ------------------------------------------------------------------ argument helpers

inline const at::Tensor* tensor_or_null(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }
template <class T>
inline T* address(PyObject* o) { return reinterpret_cast<T*>(PyLong_AsUnsignedLongLong(o)); }
inline int dtype_code(at::ScalarType t) {
    return t == at::kBFloat16 ? TQ_BF16 : t == at::kHalf ? TQ_F16 : t == at::kFloat ? TQ_F32 : -1;
}
inline void* stream_of(const at::Tensor& t) {
    return reinterpret_cast<void*>(c10::cuda::getCurrentCUDAStream(t.get_device()).stream());
}
// A captured launch keeps its arguments: lengths that the host knows would stay those of the capture, where the general way's
// are read on the device at every replay.  The legacy default stream cannot be captured and need not be asked (0.2 us).
inline bool capturing(const at::Tensor& t) {
    return stream_of(t) != nullptr && c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None;
}
// (n, heads, dim) rows the kernels can read in place: CUDA, `dim` contiguous
inline bool rows_ok(const at::Tensor& t, int64_t heads, int64_t dim) {
    return t.is_cuda() && t.dim() == 3 && t.size(1) == heads && t.size(2) == dim && t.stride(2) == 1;
}
// The first n rows of t as a contiguous (n, width) block, whatever its shape (rows, heads, dim) or (rows, width)
inline bool block_ok(const at::Tensor& t, int64_t n, int64_t heads, int64_t dim) {
    return t.is_cuda() && t.is_contiguous() && (t.dim() == 3 ? t.size(1) == heads && t.size(2) == dim : t.dim() == 2 && t.size(1) == heads * dim) &&
           t.size(0) >= n;
}
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Workspace (a Python object with .buf and .ensure(nbytes)): pointer and size once it holds `need` bytes.
bool workspace(PyObject* ws, size_t need, void** ptr, size_t* bytes) {
    static PyObject* name = PyUnicode_InternFromString("buf");
    for (int pass = 0; pass < 2; ++pass) {
        PyObject* buf = PyObject_GetAttr(ws, name);
        if (buf == nullptr) return false;
        const at::Tensor* t = tensor_or_null(buf);
        const bool fits = t != nullptr && (size_t)t->numel() >= need;
        if (fits) {
            *ptr = t->data_ptr();
            *bytes = (size_t)t->numel();
        }
        Py_DECREF(buf);   // the workspace object keeps it
        if (fits) return true;
        PyObject* r = PyObject_CallMethod(ws, "ensure", "n", (Py_ssize_t)need);
        if (r == nullptr) return false;
        Py_DECREF(r);
    }
    PyErr_SetString(PyExc_RuntimeError, "the workspace did not grow");
    return false;
}

// Fills what every decode call shares; false with a Python error set when the workspace cannot be had.
// *rc is the library's answer to the planning calls.
bool plan(tq_decode_args& a, const tq_consts* c, const tq_pool* pool, PyObject* ws, int batch, int q_heads, int max_seq,
          int max_ring, int* rc) {
    size_t need = 0;
    a.batch = batch;
    a.num_q_heads = q_heads;
    a.max_seq_len = max_seq;
    a.num_splits = tq_decode_splits(batch, pool->num_kv_heads, max_seq, max_ring, 0);
    *rc = tq_decode_workspace_bytes(&c->cfg, batch, q_heads, pool->num_kv_heads, a.num_splits, &need);
    if (*rc != TQ_OK) return true;
    return workspace(ws, need, &a.workspace, &a.workspace_bytes);
}

#define ARGS(n)                                                                              \
    if (nargs != (n)) {                                                                      \
        PyErr_Format(PyExc_TypeError, "%s takes %d arguments, got %zd", __func__, n, nargs); \
        return nullptr;                                                                      \
    }

// ------------------------------------------------------------------ ring

// ring_write(ring_k, ring_v, key, value, position, n) -> status, or None: not a case for the kernel
PyObject* ring_write(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    ARGS(6);
    const at::Tensor *rk = tensor_or_null(args[0]), *rv = tensor_or_null(args[1]), *k = tensor_or_null(args[2]),
                     *v = tensor_or_null(args[3]);
    const int64_t pos = PyLong_AsLongLong(args[4]), n = PyLong_AsLongLong(args[5]);
    if (!rk || !rv || !k || !v || !rk->is_cuda() || n < 1 || pos < 0 || rk->dim() != 3 || pos + n > rk->size(0)) Py_RETURN_NONE;
    const int64_t h = rk->size(1), d = rk->size(2);
    if (!rows_ok(*k, h, d) || !rows_ok(*v, h, d) || k->size(0) < n || v->size(0) < n || k->scalar_type() != rk->scalar_type() ||
        v->scalar_type() != rk->scalar_type() || k->get_device() != rk->get_device() || v->get_device() != rk->get_device() ||
        k->stride(0) != v->stride(0) || k->stride(1) != v->stride(1) || !rk->is_contiguous() || !rv->is_contiguous())
        Py_RETURN_NONE;
    const int dt = dtype_code(rk->scalar_type());
    if (dt < 0) Py_RETURN_NONE;
    const int rc = tq_ring_write(k->data_ptr(), v->data_ptr(), (tq_dtype)dt, n, (int32_t)h, (int32_t)d, k->stride(0), k->stride(1),
                                 rk->data_ptr(), rv->data_ptr(), h * d, pos, stream_of(*rk));
    if (rc == TQ_ERR_ALIGN || rc == TQ_ERR_UNSUPPORTED) Py_RETURN_NONE;
    return PyLong_FromLong(rc);
    END_HANDLE_TH_ERRORS
}

// ------------------------------------------------------------------ store

// store(consts, pool, key, value, head_dim, block_table | None, slots | None, start_pos, n) -> status or None
PyObject* store(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    ARGS(9);
    const tq_consts* c = address<const tq_consts>(args[0]);
    const tq_pool* pool = address<const tq_pool>(args[1]);
    const at::Tensor *k = tensor_or_null(args[2]), *v = tensor_or_null(args[3]);
    const int64_t d = PyLong_AsLongLong(args[4]), start = PyLong_AsLongLong(args[7]), n = PyLong_AsLongLong(args[8]);
    const at::Tensor *bt = tensor_or_null(args[5]), *slots = tensor_or_null(args[6]);
    if (PyErr_Occurred()) return nullptr;
    if (!k || !v || n < 1 || !rows_ok(*k, pool->num_kv_heads, d) || !rows_ok(*v, pool->num_kv_heads, d) || k->size(0) != n ||
        v->size(0) != n || k->stride(0) != v->stride(0) || k->stride(1) != v->stride(1) || k->scalar_type() != v->scalar_type() ||
        k->get_device() != v->get_device())
        Py_RETURN_NONE;
    if (slots && (slots->scalar_type() != at::kLong || slots->numel() < n || !slots->is_contiguous() || !slots->is_cuda())) Py_RETURN_NONE;
    const int dt = dtype_code(k->scalar_type());
    if (dt < 0 || (!bt && !slots)) Py_RETURN_NONE;
    return PyLong_FromLong(tq_store(c, k->data_ptr(), v->data_ptr(), (tq_dtype)dt, n, pool->num_kv_heads, k->stride(0), k->stride(1),
                                    slots ? slots->data_ptr<int64_t>() : nullptr, bt ? bt->data_ptr<int32_t>() : nullptr, start,
                                    pool, stream_of(*k)));
    END_HANDLE_TH_ERRORS
}

// ------------------------------------------------------------------ decode

// hybrid(consts, pool, workspace, block_table, head_dim, n_history, query, n_queries, q_heads, recent_k | None,
//        recent_v | None, n_recent | None, scale | None, min_history, out | None) -> out tensor, status int on failure, or None
// The first n_recent rows of recent_k / recent_v are attended to (None: all of them); a caller that has a ring passes its
// storage and fill instead of slicing both tensors, 3 us of a 20 us step.
// One sequence: every query attends to the whole history and all recent tokens.  `query` may be
// (n, q_heads, head_dim) or (n, q_heads * head_dim); with `out` (same dtype, contiguous, at least as long) the
// result is written there.
PyObject* hybrid(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    ARGS(15);
    const tq_consts* c = address<const tq_consts>(args[0]);
    const tq_pool* pool = address<const tq_pool>(args[1]);
    const at::Tensor* bt = tensor_or_null(args[3]);
    const int64_t d = PyLong_AsLongLong(args[4]), n = PyLong_AsLongLong(args[5]), t = PyLong_AsLongLong(args[7]),
                  qh = PyLong_AsLongLong(args[8]), min_history = PyLong_AsLongLong(args[13]);
    const at::Tensor *q = tensor_or_null(args[6]), *rk = tensor_or_null(args[9]), *rv = tensor_or_null(args[10]),
                     *out = tensor_or_null(args[14]);
    const double scale = args[12] == Py_None ? 1.0 / std::sqrt((double)d) : PyFloat_AsDouble(args[12]);
    const int64_t n_recent = args[11] == Py_None ? -1 : PyLong_AsLongLong(args[11]);
    if (PyErr_Occurred()) return nullptr;
    const int64_t h = pool->num_kv_heads;
    if (!bt || !q || t < 1 || qh < 1 || qh % h != 0 || !block_ok(*q, t, qh, d) || q->get_device() != bt->get_device()) Py_RETURN_NONE;
    const int dt = dtype_code(q->scalar_type());
    if (dt < 0 || (out && (!block_ok(*out, t, qh, d) || out->scalar_type() != q->scalar_type() || !aligned16(out->data_ptr()))))
        Py_RETURN_NONE;
    tq_decode_args a = {};
    const int64_t r = !rk ? 0 : n_recent >= 0 ? n_recent : rk->size(0);
    if (n < min_history && r == 0) Py_RETURN_NONE;
    if (r > 0) {
        if (!rv || !rows_ok(*rk, h, d) || !rows_ok(*rv, h, d) || rk->stride(1) != d || rv->stride(1) != d ||
            rk->stride(0) != rv->stride(0) || rk->size(0) < r || rv->size(0) != rk->size(0) || rk->scalar_type() != rv->scalar_type() || r > 256)
            Py_RETURN_NONE;
        const int rdt = dtype_code(rk->scalar_type());
        if (rdt < 0 || !aligned16(rk->data_ptr()) || !aligned16(rv->data_ptr()) || (r > 1 && rk->stride(0) * rk->element_size() % 16 != 0))
            Py_RETURN_NONE;
        a.ring_k = rk->data_ptr();
        a.ring_v = rv->data_ptr();
        a.ring_dtype = (tq_dtype)rdt;
        a.max_ring_len = (int32_t)r;
        a.ring_stride_token = rk->stride(0);
    }
    if (capturing(*q)) Py_RETURN_NONE;
    int rc = TQ_OK;
    if (!plan(a, c, pool, args[2], (int)t, (int)qh, (int)n, (int)r, &rc)) return nullptr;
    if (rc != TQ_OK) return PyLong_FromLong(rc);
    a.query = q->data_ptr();
    a.q_dtype = (tq_dtype)dt;
    a.block_table = bt->data_ptr<int32_t>();
    a.block_table_stride = (int32_t)bt->numel();
    a.min_history = (int32_t)min_history;
    a.scale = (float)scale;
    a.flags = TQ_DECODE_HOST_LENS | TQ_DECODE_SHARED_TABLE;
    at::Tensor res;
    if (!out) {
        res = at::empty({t, qh, d}, q->options());
        out = &res;
    }
    a.out = out->data_ptr();
    rc = tq_decode(c, pool, &a, stream_of(*q));
    if (rc != TQ_OK) return PyLong_FromLong(rc);
    if (!res.defined()) {
        Py_INCREF(args[14]);
        return args[14];
    }
    return THPVariable_Wrap(std::move(res));
    END_HANDLE_TH_ERRORS
}

// step(consts, pool, workspace, block_table, head_dim, n_history, query, key, value, q_heads, ring_k, ring_v, ring_fill,
//      scale | None, min_history, out | None) -> out tensor, status int, or None
// One new token of one sequence: appended to the ring by the launch that prepares the query, then attended.
PyObject* step(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    ARGS(16);
    const tq_consts* c = address<const tq_consts>(args[0]);
    const tq_pool* pool = address<const tq_pool>(args[1]);
    const at::Tensor* bt = tensor_or_null(args[3]);
    const int64_t d = PyLong_AsLongLong(args[4]), n = PyLong_AsLongLong(args[5]), qh = PyLong_AsLongLong(args[9]),
                  fill = PyLong_AsLongLong(args[12]), min_history = PyLong_AsLongLong(args[14]);
    const at::Tensor *q = tensor_or_null(args[6]), *k = tensor_or_null(args[7]), *v = tensor_or_null(args[8]),
                     *rk = tensor_or_null(args[10]), *rv = tensor_or_null(args[11]), *out = tensor_or_null(args[15]);
    const double scale = args[13] == Py_None ? 1.0 / std::sqrt((double)d) : PyFloat_AsDouble(args[13]);
    if (PyErr_Occurred()) return nullptr;
    const int64_t h = pool->num_kv_heads;
    if (!bt || !q || !k || !v || !rk || !rv || qh < 1 || qh % h != 0 || q->dim() != 3 || q->size(0) != 1 || q->size(1) != qh ||
        q->size(2) != d || !q->is_cuda() || !q->is_contiguous() || k->numel() != h * d || v->numel() != h * d || !k->is_contiguous() ||
        !v->is_contiguous() || k->size(0) != 1 || v->size(0) != 1 || !k->is_cuda() || !v->is_cuda() ||
        k->scalar_type() != rk->scalar_type() || v->scalar_type() != rk->scalar_type() ||
        q->get_device() != bt->get_device() || fill < 0 || fill >= rk->size(0) || fill >= 256 || !rk->is_contiguous() || !rv->is_contiguous())
        Py_RETURN_NONE;
    const int dt = dtype_code(q->scalar_type()), rdt = dtype_code(rk->scalar_type());
    if (dt < 0 || rdt < 0 || !aligned16(k->data_ptr()) || !aligned16(v->data_ptr())) Py_RETURN_NONE;
    if (out && (!block_ok(*out, 1, qh, d) || out->scalar_type() != q->scalar_type() || !aligned16(out->data_ptr()))) Py_RETURN_NONE;
    if (capturing(*q)) Py_RETURN_NONE;
    tq_decode_args a = {};
    int rc = TQ_OK;
    if (!plan(a, c, pool, args[2], 1, (int)qh, (int)n, (int)fill + 1, &rc)) return nullptr;
    if (rc != TQ_OK) return PyLong_FromLong(rc);
    a.query = q->data_ptr();
    a.q_dtype = (tq_dtype)dt;
    a.block_table = bt->data_ptr<int32_t>();
    a.block_table_stride = (int32_t)bt->numel();
    a.min_history = (int32_t)min_history;
    a.ring_k = rk->data_ptr();
    a.ring_v = rv->data_ptr();
    a.ring_dtype = (tq_dtype)rdt;
    a.max_ring_len = (int32_t)fill + 1;
    a.ring_stride_token = h * d;
    a.append_k = k->data_ptr();
    a.append_v = v->data_ptr();
    a.ring_capacity = (int32_t)rk->size(0);
    a.scale = (float)scale;
    a.flags = TQ_DECODE_HOST_LENS;
    at::Tensor res;
    if (!out) {
        res = at::empty({1, qh, d}, q->options());
        out = &res;
    }
    a.out = out->data_ptr();
    rc = tq_decode(c, pool, &a, stream_of(*q));
    if (rc != TQ_OK) return PyLong_FromLong(rc);
    if (!res.defined()) {
        Py_INCREF(args[15]);
        return args[15];
    }
    return THPVariable_Wrap(std::move(res));
    END_HANDLE_TH_ERRORS
}

// batch(consts, pool, workspace, head_dim, query, block_tables, seq_lens, max_seq_len, scale | None, min_history, out | None)
// -> out tensor, status int, or None.  One decode token per sequence of a paged batch, no exact tokens.
PyObject* batch(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    ARGS(11);
    const tq_consts* c = address<const tq_consts>(args[0]);
    const tq_pool* pool = address<const tq_pool>(args[1]);
    const int64_t d = PyLong_AsLongLong(args[3]), max_seq = PyLong_AsLongLong(args[7]), min_history = PyLong_AsLongLong(args[9]);
    const at::Tensor *q = tensor_or_null(args[4]), *bt = tensor_or_null(args[5]), *lens = tensor_or_null(args[6]),
                     *out = tensor_or_null(args[10]);
    const double scale = args[8] == Py_None ? 1.0 / std::sqrt((double)d) : PyFloat_AsDouble(args[8]);
    if (PyErr_Occurred()) return nullptr;
    if (!q || !bt || !lens || q->dim() != 3 || q->size(0) < 1 || q->size(2) != d || !q->is_cuda() || !q->is_contiguous() ||
        bt->dim() != 2 || bt->scalar_type() != at::kInt || bt->stride(1) != 1 || !bt->is_cuda() || lens->scalar_type() != at::kInt ||
        !lens->is_contiguous() || !lens->is_cuda() || bt->size(0) < q->size(0) || lens->numel() < q->size(0))
        Py_RETURN_NONE;
    const int64_t b = q->size(0), qh = q->size(1);
    const int dt = dtype_code(q->scalar_type());
    if (dt < 0 || (out && (!out->is_cuda() || !out->is_contiguous() || out->sizes() != q->sizes() || out->scalar_type() != q->scalar_type()))) Py_RETURN_NONE;
    tq_decode_args a = {};
    int rc = TQ_OK;
    if (!plan(a, c, pool, args[2], (int)b, (int)qh, (int)max_seq, 0, &rc)) return nullptr;
    if (rc != TQ_OK) return PyLong_FromLong(rc);
    a.query = q->data_ptr();
    a.q_dtype = (tq_dtype)dt;
    a.block_table = bt->data_ptr<int32_t>();
    a.block_table_stride = (int32_t)bt->stride(0);
    a.seq_lens = lens->data_ptr<int32_t>();
    a.min_history = (int32_t)min_history;
    a.scale = (float)scale;
    at::Tensor res;
    if (!out) {
        res = at::empty_like(*q);
        out = &res;
    }
    a.out = out->data_ptr();
    rc = tq_decode(c, pool, &a, stream_of(*q));
    if (rc != TQ_OK) return PyLong_FromLong(rc);
    if (!res.defined()) {
        Py_INCREF(args[10]);
        return args[10];
    }
    return THPVariable_Wrap(std::move(res));
    END_HANDLE_TH_ERRORS
}

// ------------------------------------------------------------------ the quantiser objects on plain rows

// sizes of `t` without its last dimension, then `tail`
inline std::vector<int64_t> lead_shape(const at::Tensor& t, std::initializer_list<int64_t> tail) {
    std::vector<int64_t> s(t.sizes().begin(), t.sizes().end() - 1);
    s.insert(s.end(), tail);
    return s;
}
inline bool rows_tensor(const at::Tensor* t) { return t && t->is_cuda() && t->is_contiguous() && t->dim() >= 1 && t->numel() > 0; }
inline bool declined(int rc) { return rc == TQ_ERR_UNSUPPORTED || rc == TQ_ERR_ALIGN || rc == TQ_ERR_SHAPE; }
PyObject* tuple_of(std::initializer_list<at::Tensor> ts) {
    PyObject* r = PyTuple_New((Py_ssize_t)ts.size());
    Py_ssize_t i = 0;
    for (const at::Tensor& t : ts) PyTuple_SET_ITEM(r, i++, THPVariable_Wrap(t));
    return r;
}

// quantize_keys(consts, x (..., D)) -> (codes, sign bits, norms, residual norms), status, or None
PyObject* quantize_keys(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    ARGS(2);
    const tq_consts* c = address<const tq_consts>(args[0]);
    const at::Tensor* x = tensor_or_null(args[1]);
    if (PyErr_Occurred()) return nullptr;
    const int64_t d = c->cfg.head_dim;
    if (!rows_tensor(x) || x->size(-1) != d) Py_RETURN_NONE;
    const int dt = dtype_code(x->scalar_type());
    if (dt != TQ_F32 && dt != TQ_F16) Py_RETURN_NONE;
    const auto bytes = x->options().dtype(at::kByte);
    at::Tensor codes = at::empty(lead_shape(*x, {c->cfg.key_bits == 3 ? d / 4 : d / 2}), bytes), signs = at::empty(lead_shape(*x, {d / 8}), bytes),
               norms = at::empty(lead_shape(*x, {}), x->options()), rnorms = at::empty(lead_shape(*x, {}), x->options().dtype(at::kFloat));
    const int rc = tq_rows_quantize_keys(c, x->data_ptr(), (tq_dtype)dt, x->numel() / d, d, codes.data_ptr<uint8_t>(), signs.data_ptr<uint8_t>(),
                                         norms.data_ptr(), (tq_dtype)dt, rnorms.data_ptr(), TQ_F32, stream_of(*x));
    if (declined(rc)) Py_RETURN_NONE;
    if (rc != TQ_OK) return PyLong_FromLong(rc);
    return tuple_of({codes, signs, norms, rnorms});
    END_HANDLE_TH_ERRORS
}

// dequantize_keys(consts, codes, sign bits | None, norms, residual norms | None) -> rows fp32, status, or None
PyObject* dequantize_keys(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    ARGS(5);
    const tq_consts* c = address<const tq_consts>(args[0]);
    const at::Tensor *codes = tensor_or_null(args[1]), *signs = tensor_or_null(args[2]), *norms = tensor_or_null(args[3]), *rn = tensor_or_null(args[4]);
    if (PyErr_Occurred()) return nullptr;
    if (!rows_tensor(codes) || !rows_tensor(norms) || (signs && !rows_tensor(signs)) || (rn && !rows_tensor(rn)) || (signs != nullptr) != (rn != nullptr))
        Py_RETURN_NONE;
    const int64_t d = c->cfg.head_dim, n = norms->numel(), row = c->cfg.key_bits == 3 ? d / 4 : d / 2;
    const int dn = dtype_code(norms->scalar_type()), dr = rn ? dtype_code(rn->scalar_type()) : TQ_F32;
    if (dn < 0 || dr < 0 || codes->scalar_type() != at::kByte || codes->numel() != n * row || (signs && (signs->scalar_type() != at::kByte ||
        signs->numel() != n * (d / 8) || rn->numel() != n)))
        Py_RETURN_NONE;
    std::vector<int64_t> shape(norms->sizes().begin(), norms->sizes().end());
    shape.push_back(d);
    at::Tensor out = at::empty(shape, norms->options().dtype(at::kFloat));
    const int rc = tq_rows_dequantize_keys(c, codes->data_ptr<uint8_t>(), signs ? signs->data_ptr<uint8_t>() : nullptr, norms->data_ptr(), (tq_dtype)dn,
                                           rn ? rn->data_ptr() : nullptr, (tq_dtype)dr, n, signs ? 1 : 0, out.data_ptr<float>(), stream_of(*codes));
    if (declined(rc)) Py_RETURN_NONE;
    if (rc != TQ_OK) return PyLong_FromLong(rc);
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// key_scores(consts, workspace, query (..., n_q, D), codes, sign bits, norms (..., n), residual norms) -> logits, status, or None
PyObject* key_scores(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    ARGS(7);
    const tq_consts* c = address<const tq_consts>(args[0]);
    const at::Tensor *q = tensor_or_null(args[2]), *codes = tensor_or_null(args[3]), *signs = tensor_or_null(args[4]), *norms = tensor_or_null(args[5]),
                     *rn = tensor_or_null(args[6]);
    if (PyErr_Occurred()) return nullptr;
    const int64_t d = c->cfg.head_dim;
    if (!rows_tensor(q) || !rows_tensor(codes) || !rows_tensor(signs) || !rows_tensor(norms) || !rows_tensor(rn) || q->dim() < 2 || q->size(-1) != d)
        Py_RETURN_NONE;
    const int64_t n = norms->size(-1), heads = norms->numel() / n, n_q = q->size(-2);
    const int dq = dtype_code(q->scalar_type()), dn = dtype_code(norms->scalar_type()), dr = dtype_code(rn->scalar_type());
    if (dq < 0 || dn < 0 || dr < 0 || q->numel() != heads * n_q * d || rn->numel() != norms->numel() || codes->scalar_type() != at::kByte ||
        signs->scalar_type() != at::kByte || codes->numel() != heads * n * (c->cfg.key_bits == 3 ? d / 4 : d / 2) || signs->numel() != heads * n * (d / 8))
        Py_RETURN_NONE;
    size_t need = 0, bytes = 0;
    void* ws = nullptr;
    int rc = tq_scores_workspace_bytes(&c->cfg, heads * n_q, &need);
    if (rc != TQ_OK) return PyLong_FromLong(rc);
    if (!workspace(args[1], need, &ws, &bytes)) return nullptr;
    std::vector<int64_t> shape(norms->sizes().begin(), norms->sizes().end() - 1);
    shape.push_back(n_q);
    shape.push_back(n);
    at::Tensor logits = at::empty(shape, norms->options().dtype(at::kFloat));
    rc = tq_rows_scores(c, codes->data_ptr<uint8_t>(), signs->data_ptr<uint8_t>(), norms->data_ptr(), (tq_dtype)dn, rn->data_ptr(), (tq_dtype)dr,
                        (int32_t)heads, n, q->data_ptr(), (tq_dtype)dq, (int32_t)n_q, logits.data_ptr<float>(), ws, bytes, stream_of(*q));
    if (declined(rc)) Py_RETURN_NONE;
    if (rc != TQ_OK) return PyLong_FromLong(rc);
    return THPVariable_Wrap(std::move(logits));
    END_HANDLE_TH_ERRORS
}

// quantize_values(v (..., D), bits) -> (codes, scales, zero points), status, or None
PyObject* quantize_values(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    ARGS(2);
    const at::Tensor* v = tensor_or_null(args[0]);
    const int64_t bits = PyLong_AsLongLong(args[1]);
    if (PyErr_Occurred()) return nullptr;
    if (!rows_tensor(v)) Py_RETURN_NONE;
    const int64_t d = v->size(-1);
    const int dt = dtype_code(v->scalar_type());
    if (dt < 0 || (d != 128 && d != 256) || (bits != 2 && bits != 4)) Py_RETURN_NONE;
    at::Tensor data = at::empty(lead_shape(*v, {d * bits / 8}), v->options().dtype(at::kByte)), scales = at::empty(lead_shape(*v, {d / 32}), v->options()),
               zeros = at::empty(lead_shape(*v, {d / 32}), v->options());
    const int rc = tq_rows_quantize_values(v->data_ptr(), (tq_dtype)dt, v->numel() / d, (int32_t)d, d, (int32_t)bits, data.data_ptr<uint8_t>(),
                                           scales.data_ptr(), zeros.data_ptr(), stream_of(*v));
    if (declined(rc)) Py_RETURN_NONE;
    if (rc != TQ_OK) return PyLong_FromLong(rc);
    return tuple_of({data, scales, zeros});
    END_HANDLE_TH_ERRORS
}

// dequantize_values(codes, scales, zero points, bits) -> rows fp32, status, or None
PyObject* dequantize_values(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    ARGS(4);
    const at::Tensor *data = tensor_or_null(args[0]), *sc = tensor_or_null(args[1]), *zr = tensor_or_null(args[2]);
    const int64_t bits = PyLong_AsLongLong(args[3]);
    if (PyErr_Occurred()) return nullptr;
    if (!rows_tensor(data) || !rows_tensor(sc) || !rows_tensor(zr) || (bits != 2 && bits != 4) || data->scalar_type() != at::kByte) Py_RETURN_NONE;
    const int64_t d = data->size(-1) * 8 / bits, n = data->numel() / data->size(-1);
    const int dt = dtype_code(sc->scalar_type());
    if (dt < 0 || (d != 128 && d != 256) || zr->scalar_type() != sc->scalar_type() || sc->numel() != n * (d / 32) || zr->numel() != sc->numel()) Py_RETURN_NONE;
    at::Tensor out = at::empty(lead_shape(*data, {d}), data->options().dtype(at::kFloat));
    const int rc = tq_rows_dequantize_values(data->data_ptr<uint8_t>(), sc->data_ptr(), zr->data_ptr(), (tq_dtype)dt, n, (int32_t)d, (int32_t)bits,
                                             out.data_ptr<float>(), stream_of(*data));
    if (declined(rc)) Py_RETURN_NONE;
    if (rc != TQ_OK) return PyLong_FromLong(rc);
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// ------------------------------------------------------------------ the single-object cache

// cache_scores(consts, pool, workspace, block_table, n, query (b, h, n_q, D), exact keys (b, h, m, D) | None, scale)
//   -> scaled logits (b, h, n_q, n + m)
// cache_attend(consts, pool, workspace, block_table, n, weights (b, h, n_q, n + m), exact values | None) -> (b, h, n_q, D)
// Both: the tensor, a status, None where strides or types are not the kernel's, NotImplemented where the call is too large for it
// (nothing has been allocated then).
PyObject* cache_call(PyObject* const* args, bool scores) {
    const tq_consts* c = address<const tq_consts>(args[0]);
    const tq_pool* pool = address<const tq_pool>(args[1]);
    const at::Tensor *bt = tensor_or_null(args[3]), *x = tensor_or_null(args[5]), *buf = tensor_or_null(args[6]);
    const int64_t n = PyLong_AsLongLong(args[4]), d = c->cfg.head_dim;
    const double scale = scores ? PyFloat_AsDouble(args[7]) : 0.0;
    if (PyErr_Occurred()) return nullptr;
    if (!bt || !x || !x->is_cuda() || x->dim() != 4 || x->numel() == 0 || x->get_device() != bt->get_device() || n < 1) Py_RETURN_NONE;
    const int64_t b = x->size(0), h = x->size(1), n_q = x->size(2), m = buf ? buf->size(2) : 0;
    const int dt = dtype_code(x->scalar_type()), db = m ? dtype_code(buf->scalar_type()) : TQ_F32;
    if (dt < 0 || db < 0 || b * h != pool->num_kv_heads || x->size(3) != (scores ? d : n + m)) Py_RETURN_NONE;
    size_t need = 0, bytes = 0;
    void* ws = nullptr;
    int rc = scores ? tq_cache_scores_workspace_bytes(&c->cfg, (int32_t)(b * h), (int32_t)n_q, &need)
                    : tq_cache_attend_workspace_bytes(&c->cfg, (int32_t)(b * h), n, m, (int32_t)n_q, &need);
    if (rc == TQ_ERR_UNSUPPORTED) Py_RETURN_NOTIMPLEMENTED;
    if (rc != TQ_OK) return PyLong_FromLong(rc);
    if (!x->is_contiguous()) Py_RETURN_NONE;
    if (m) {
        const int64_t es = (int64_t)buf->element_size();
        if (buf->dim() != 4 || buf->size(0) != b || buf->size(1) != h || buf->size(3) != d || !buf->is_cuda() || buf->get_device() != x->get_device() ||
            buf->stride(3) != 1 || (b > 1 && buf->stride(0) != h * buf->stride(1)) || !aligned16(buf->data_ptr()) || (buf->stride(1) * es) % 16 ||
            (buf->stride(2) * es) % 16)
            Py_RETURN_NONE;
    }
    if (!workspace(args[2], need, &ws, &bytes)) return nullptr;
    at::Tensor out = at::empty({b, h, n_q, scores ? n + m : d}, x->options().dtype(at::kFloat));
    const void* rows = m ? buf->data_ptr() : nullptr;
    const int64_t sh = m ? buf->stride(1) : 0, st = m ? buf->stride(2) : 0;
    if (scores)
        rc = tq_cache_scores(c, pool, bt->data_ptr<int32_t>(), n, x->data_ptr(), (tq_dtype)dt, (int32_t)n_q, rows, (tq_dtype)db, m, sh, st,
                             (float)scale, out.data_ptr<float>(), ws, bytes, stream_of(*x));
    else
        rc = tq_cache_attend(c, pool, bt->data_ptr<int32_t>(), n, x->data_ptr(), (tq_dtype)dt, (int32_t)n_q, rows, (tq_dtype)db, m, sh, st,
                             out.data_ptr<float>(), ws, bytes, stream_of(*x));
    if (rc == TQ_ERR_UNSUPPORTED || rc == TQ_ERR_ALIGN) Py_RETURN_NONE;
    if (rc != TQ_OK) return PyLong_FromLong(rc);
    return THPVariable_Wrap(std::move(out));
}
PyObject* cache_scores(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    ARGS(8);
    return cache_call(args, true);
    END_HANDLE_TH_ERRORS
}
PyObject* cache_attend(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    ARGS(7);
    return cache_call(args, false);
    END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"cache_scores", (PyCFunction)(void (*)(void))cache_scores, METH_FASTCALL, nullptr},
    {"cache_attend", (PyCFunction)(void (*)(void))cache_attend, METH_FASTCALL, nullptr},
    {"quantize_keys", (PyCFunction)(void (*)(void))quantize_keys, METH_FASTCALL, nullptr},
    {"dequantize_keys", (PyCFunction)(void (*)(void))dequantize_keys, METH_FASTCALL, nullptr},
    {"key_scores", (PyCFunction)(void (*)(void))key_scores, METH_FASTCALL, nullptr},
    {"quantize_values", (PyCFunction)(void (*)(void))quantize_values, METH_FASTCALL, nullptr},
    {"dequantize_values", (PyCFunction)(void (*)(void))dequantize_values, METH_FASTCALL, nullptr},
    {"ring_write", (PyCFunction)(void (*)(void))ring_write, METH_FASTCALL, nullptr},
    {"store", (PyCFunction)(void (*)(void))store, METH_FASTCALL, nullptr},
    {"hybrid", (PyCFunction)(void (*)(void))hybrid, METH_FASTCALL, nullptr},
    {"step", (PyCFunction)(void (*)(void))step, METH_FASTCALL, nullptr},
    {"batch", (PyCFunction)(void (*)(void))batch, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Host side of the decode-step calls", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&module); }
