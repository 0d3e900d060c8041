// Native host path of the calls that are mostly host work: a prompt into a fresh cache, a dense result, the row codec.  Each of them made ten
// to forty small steps in Python (allocations, views, argument blocks field by field, a library call at a time): 160 us of host for 45 us of
// kernels where 4000 tokens of 8 heads go into a cache that hands dense tensors back, 25 us for the codec's two calls.
//
// Every function takes tensors as they are and checks what the launch relies on: CUDA, current device, types, strides.  Anything but the plain
// case is None, and the caller in Python takes its own path, with its conversions and its errors.  A library error is its negative code.
// The GIL is released around library calls, as ctypes does.
#include <torch/csrc/python_headers.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>

#include <cstring>

#include "../../include/tq_abi.h"

namespace {

struct Release {                                        // the GIL, around library calls
    PyThreadState* s = PyEval_SaveThread();
    ~Release() { PyEval_RestoreThread(s); }
};

PyObject* none() { Py_RETURN_NONE; }
PyObject* status(int rc) { return PyLong_FromLong(rc); }
bool is_tensor(PyObject* o) { return THPVariable_Check(o); }
const at::Tensor& tensor(PyObject* o) { return THPVariable_Unpack(o); }
int64_t integer(PyObject* o) { return PyLong_AsLongLong(o); }

int type_code(at::ScalarType t) { return t == at::kHalf ? TQ_F16 : t == at::kBFloat16 ? TQ_BF16 : t == at::kFloat ? TQ_F32 : -1; }
bool here(const at::Tensor& t, int device) { return t.is_cuda() && t.get_device() == device && t.layout() == at::kStrided; }
at::Tensor empty(at::IntArrayRef size, at::ScalarType type, int device) { return at::empty(size, at::TensorOptions().dtype(type).device(at::kCUDA, device)); }
void* stream_of(int device) { return c10::cuda::getCurrentCUDAStream(device).stream(); }

// Rows (B, H, T, D) with one stride per lane and one per row
struct Rows { int64_t b, h, t, d, lane, row; };
bool rows_of(const at::Tensor& x, Rows& r) {
    if (x.dim() != 4 || x.stride(3) != 1) return false;
    r = Rows{x.size(0), x.size(1), x.size(2), x.size(3), 0, 0};
    if (r.b > 1 && r.h > 1 && x.stride(0) != r.h * x.stride(1)) return false;
    r.lane = r.h > 1 ? x.stride(1) : r.b > 1 ? x.stride(0) : 0;
    r.row = r.t > 1 ? x.stride(2) : r.d;
    return true;
}
// ... rows next to one another, lanes a whole number of rows apart that do not overlap: what the row copies take.  src_ls: rows between lanes.
bool copyable(const at::Tensor& x, int64_t first, int64_t n, Rows& r, int64_t& src_ls) {
    if (!rows_of(x, r) || r.row != r.d || first + n > r.t || (r.d * int64_t(x.element_size())) % 16) return false;
    src_ls = r.b * r.h > 1 ? r.lane / r.d : first + n;
    return r.b * r.h == 1 || (r.lane % r.d == 0 && src_ls >= first + n);
}
const char* at_row(const at::Tensor& x, int64_t row) { return static_cast<const char*>(x.data_ptr()) + row * x.size(-1) * int64_t(x.element_size()); }

// ---- row codec -------------------------------------------------------------------------------------------------
// codec_quantize(block, width, x, table): contiguous rows (..., d) -> packed, norms
PyObject* codec_quantize(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 4 || !PyBytes_Check(a[0]) || PyBytes_GET_SIZE(a[0]) != sizeof(tq_quantize_args) || !is_tensor(a[2]) || !is_tensor(a[3])) return none();
    const at::Tensor &x = tensor(a[2]), &table = tensor(a[3]);
    tq_quantize_args q;
    std::memcpy(&q, PyBytes_AS_STRING(a[0]), sizeof q);
    const int device = c10::cuda::current_device(), code = type_code(x.scalar_type());
    if (code < 0 || !here(x, device) || !here(table, device) || x.dim() < 1 || x.size(-1) != q.d || !x.is_contiguous()) return none();
    auto size = x.sizes().vec();
    size.back() = integer(a[1]);
    at::Tensor packed = empty(size, at::kByte, device);
    size.pop_back();
    at::Tensor norms = empty(size, at::kFloat, device);
    q.x = x.data_ptr(); q.x_dtype = code;
    q.packed_hi = packed.data_ptr<uint8_t>(); q.norms = norms.data_ptr<float>();
    q.n_rows = q.out_lane_stride = norms.numel();
    int rc;
    {
        Release gil;
        rc = tq_quantize_pack(&q, stream_of(device));
    }
    if (rc) return status(rc);
    return PyTuple_Pack(2, THPObjectPtr(THPVariable_Wrap(packed)).get(), THPObjectPtr(THPVariable_Wrap(norms)).get());
    END_HANDLE_TH_ERRORS
}
// codec_dequantize(block, width, packed, norms, table): -> float32 rows
PyObject* codec_dequantize(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 5 || !PyBytes_Check(a[0]) || PyBytes_GET_SIZE(a[0]) != sizeof(tq_dequantize_args) || !is_tensor(a[2]) || !is_tensor(a[3]) || !is_tensor(a[4])) return none();
    const at::Tensor &packed = tensor(a[2]), &norms = tensor(a[3]), &table = tensor(a[4]);
    tq_dequantize_args r;
    std::memcpy(&r, PyBytes_AS_STRING(a[0]), sizeof r);
    const int device = c10::cuda::current_device();
    if (!here(packed, device) || !here(norms, device) || !here(table, device) || packed.scalar_type() != at::kByte || norms.scalar_type() != at::kFloat ||
        !packed.is_contiguous() || !norms.is_contiguous() || packed.numel() != norms.numel() * integer(a[1]))
        return none();
    auto size = norms.sizes().vec();
    size.push_back(r.d);
    at::Tensor out = empty(size, at::kFloat, device);
    r.packed_hi = packed.data_ptr<uint8_t>(); r.norms = norms.data_ptr<float>(); r.out = out.data_ptr();
    r.n_rows = r.in_lane_stride = norms.numel();
    r.out_lane_stride = r.n_rows * r.d;
    int rc;
    {
        Release gil;
        rc = tq_dequantize(&r, stream_of(device));
    }
    return rc ? status(rc) : THPVariable_Wrap(out);
    END_HANDLE_TH_ERRORS
}

// ---- token buffers ---------------------------------------------------------------------------------------------
// Whether keys and values (and the buffers they go with) agree in type, shape and strides
bool pair_of(const at::Tensor& k, const at::Tensor& v, int device) {
    return here(k, device) && here(v, device) && k.dim() == 4 && k.scalar_type() == v.scalar_type() && k.sizes() == v.sizes() && k.strides() == v.strides();
}
bool buffers_of(const at::Tensor& k, const at::Tensor& v, const at::Tensor& like, int device) {
    return pair_of(k, v, device) && k.scalar_type() == like.scalar_type() && k.size(0) == like.size(0) && k.size(1) == like.size(1) && k.size(3) == like.size(3) &&
           k.is_contiguous();
}
// append(k_buf, v_buf, k_new, v_new, first, n, row): rows [first, first + n) of the new tokens to rows row, ... of the buffers -> status
PyObject* append(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    if (n_args != 7) return none();
    for (int i = 0; i < 4; ++i)
        if (!is_tensor(a[i])) return none();
    const at::Tensor &kb = tensor(a[0]), &vb = tensor(a[1]), &k = tensor(a[2]), &v = tensor(a[3]);
    const int64_t first = integer(a[4]), n = integer(a[5]), row = integer(a[6]);
    const int device = c10::cuda::current_device();
    Rows r;
    int64_t src_ls;
    if (!pair_of(k, v, device) || !buffers_of(kb, vb, k, device) || !copyable(k, first, n, r, src_ls) || row + n > kb.size(2)) return none();
    int rc;
    {
        Release gil;
        rc = tq_append_tokens(at_row(k, first), at_row(v, first), kb.data_ptr(), vb.data_ptr(), r.b * r.h, n, r.d * int64_t(k.element_size()), src_ls, kb.size(2), row, stream_of(device));
    }
    return rc == TQ_ERR_UNSUPPORTED ? none() : status(rc);
    END_HANDLE_TH_ERRORS
}
// buffers(k_new, v_new, first, n, capacity, k_old, v_old, old_first, kept): fresh buffers (B, H, capacity, D) x 2: kept rows of the old ones, then
// rows [first, first + n) of the new tokens, then zeros
PyObject* buffers(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    if (n_args != 9 || !is_tensor(a[0]) || !is_tensor(a[1])) return none();
    const at::Tensor &k = tensor(a[0]), &v = tensor(a[1]);
    const int64_t first = integer(a[2]), n = integer(a[3]), cap = integer(a[4]), old_first = integer(a[7]), kept = integer(a[8]);
    const int device = c10::cuda::current_device();
    Rows r;
    int64_t src_ls;
    if (!pair_of(k, v, device) || type_code(k.scalar_type()) < 0 || !copyable(k, first, n, r, src_ls)) return none();
    const char *k_old = nullptr, *v_old = nullptr;
    int64_t old_ls = 0;
    if (kept > 0) {
        if (!is_tensor(a[5]) || !is_tensor(a[6])) return none();
        const at::Tensor &ko = tensor(a[5]), &vo = tensor(a[6]);
        if (!buffers_of(ko, vo, k, device) || old_first + kept > ko.size(2)) return none();
        k_old = at_row(ko, old_first); v_old = at_row(vo, old_first); old_ls = ko.size(2);
    }
    const int64_t size[4] = {r.b, r.h, cap, r.d};
    at::Tensor kb = empty(size, k.scalar_type(), device), vb = empty(size, k.scalar_type(), device);
    int rc;
    {
        Release gil;
        rc = tq_fill_tokens(k_old, v_old, kept, old_ls, n > 0 ? at_row(k, first) : nullptr, n > 0 ? at_row(v, first) : nullptr, n, src_ls, kb.data_ptr(), vb.data_ptr(), r.b * r.h,
                            r.d * int64_t(k.element_size()), cap, stream_of(device));
    }
    if (rc) return rc == TQ_ERR_UNSUPPORTED ? none() : status(rc);
    return PyTuple_Pack(2, THPObjectPtr(THPVariable_Wrap(kb)).get(), THPObjectPtr(THPVariable_Wrap(vb)).get());
    END_HANDLE_TH_ERRORS
}

// ---- packed storage --------------------------------------------------------------------------------------------
// storage(b, h, capacity, width_hi, width_lo, sketches, device): codes, second codes or None, norms, sign words or None, residual norms or None
PyObject* storage(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 7) return none();
    const int64_t b = integer(a[0]), h = integer(a[1]), cap = integer(a[2]), w_hi = integer(a[3]), w_lo = integer(a[4]);
    const bool sketches = PyObject_IsTrue(a[5]) == 1;
    const int device = int(integer(a[6]));
    const int64_t hi[4] = {b, h, cap, w_hi}, lo[4] = {b, h, cap, w_lo}, one[3] = {b, h, cap};
    auto wrap = [](at::Tensor t) { return THPVariable_Wrap(std::move(t)); };
    auto absent = [] { Py_INCREF(Py_None); return Py_None; };
    THPObjectPtr t0(wrap(empty(hi, at::kByte, device))), t1(w_lo > 0 ? wrap(empty(lo, at::kByte, device)) : absent()), t2(wrap(empty(one, at::kFloat, device))),
        t3(sketches ? wrap(empty(one, at::kInt, device)) : absent()), t4(sketches ? wrap(empty(one, at::kFloat, device)) : absent());
    return PyTuple_Pack(5, t0.get(), t1.get(), t2.get(), t3.get(), t4.get());
    END_HANDLE_TH_ERRORS
}
// quantize(at, sides...): per side (block, buffer or None, old, new, n_new, hi, lo or None, norms, sign words or None, residual norms or None): the
// first `old` rows of the buffer and the first n_new of the new tokens to packed rows at, at + old, ... -> status
PyObject* quantize(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n < 2 || n > 3) return none();
    const int64_t at0 = integer(a[0]);
    const int device = c10::cuda::current_device();
    tq_quantize_args jobs[4];
    int count = 0;
    for (Py_ssize_t i = 1; i < n; ++i) {
        if (!PyTuple_Check(a[i]) || PyTuple_GET_SIZE(a[i]) != 10) return none();
        PyObject* const* f = &PyTuple_GET_ITEM(a[i], 0);
        if (!PyBytes_Check(f[0]) || PyBytes_GET_SIZE(f[0]) != sizeof(tq_quantize_args) || !is_tensor(f[5]) || !is_tensor(f[7])) return none();
        const at::Tensor &hi = tensor(f[5]), &norms = tensor(f[7]);
        if (!here(hi, device) || !here(norms, device) || !hi.is_contiguous() || !norms.is_contiguous()) return none();
        const int64_t rows[2] = {integer(f[2]), integer(f[4])};
        int64_t row = at0;
        for (int part = 0; part < 2; ++part) {
            if (rows[part] == 0) continue;
            PyObject* src = f[part ? 3 : 1];
            if (!is_tensor(src)) return none();
            const at::Tensor& x = tensor(src);
            const int code = type_code(x.scalar_type());
            Rows r;
            // (one stride per lane and per row; an expanded axis, stride 0, is not for the tensor-core kernel)
            if (code < 0 || !here(x, device) || !rows_of(x, r) || rows[part] > r.t || (r.h > 1 && x.stride(1) == 0) || (r.b > 1 && x.stride(0) == 0) || (r.t > 1 && x.stride(2) == 0) ||
                r.b != hi.size(0) || r.h != hi.size(1) || row + rows[part] > hi.size(2))
                return none();
            tq_quantize_args& q = jobs[count++];
            std::memcpy(&q, PyBytes_AS_STRING(f[0]), sizeof q);
            if (r.d != q.d) return none();
            q.x = x.data_ptr(); q.x_dtype = code; q.n_lanes = r.b * r.h; q.n_rows = rows[part];
            q.x_lane_stride = r.lane; q.x_row_stride = r.row;
            q.packed_hi = hi.data_ptr<uint8_t>() + row * hi.size(3); q.norms = norms.data_ptr<float>() + row; q.out_lane_stride = hi.size(2);
            if (is_tensor(f[6])) {
                const at::Tensor& lo = tensor(f[6]);
                q.packed_lo = lo.data_ptr<uint8_t>() + row * lo.size(3);
            }
            if (q.qjl_proj_rot && is_tensor(f[8]) && is_tensor(f[9])) {
                q.qjl_bits = reinterpret_cast<uint32_t*>(tensor(f[8]).data_ptr<int32_t>()) + row;
                q.qjl_gamma = tensor(f[9]).data_ptr<float>() + row;
            }
            row += rows[part];
        }
    }
    int rc;
    {
        Release gil;
        rc = tq_quantize_pack_many(jobs, count, stream_of(device));
    }
    return status(rc);
    END_HANDLE_TH_ERRORS
}

// ---- dense result ----------------------------------------------------------------------------------------------
// fetch(sink_k, sink_v, sink_len, keys, values, recent_len, packed_len, k_side, v_side, dense_k, dense_v): dense keys and values
// [sink | packed | recent]; a side is (block, hi, lo or None, norms); with dense tensors the middle is copied from them
PyObject* fetch(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 11) return none();
    const int device = c10::cuda::current_device();
    const int64_t len[3] = {integer(a[2]), integer(a[5]), integer(a[6])};
    tq_fetch_args f;
    std::memset(&f, 0, sizeof f);
    const int64_t rows = len[0] + len[1] + len[2];
    int64_t b = 0, h = 0, d = 0;
    at::ScalarType type = at::kFloat;
    auto part = [&](int i, PyObject* ko, PyObject* vo, int64_t count, int64_t dst) -> bool {
        if (count == 0) return true;
        if (!is_tensor(ko) || !is_tensor(vo)) return false;
        const at::Tensor &k = tensor(ko), &v = tensor(vo);
        if (!pair_of(k, v, device) || type_code(k.scalar_type()) < 0 || !k.is_contiguous() || count > k.size(2)) return false;
        if (d == 0) { b = k.size(0); h = k.size(1); d = k.size(3); if (len[2] == 0) type = k.scalar_type(); }
        if (k.size(0) != b || k.size(1) != h || k.size(3) != d || (type != at::kFloat && k.scalar_type() != type)) return false;
        tq_fetch_part& p = f.part[i];
        p.k = k.data_ptr(); p.v = v.data_ptr(); p.dtype = type_code(k.scalar_type()); p.rows = count; p.lane_stride = k.size(2); p.dst_row = dst;
        return true;
    };
    // (the recent tokens' type is the result's where nothing is packed)
    if (!part(1, a[3], a[4], len[1], len[0] + len[2]) || !part(0, a[0], a[1], len[0], 0) || d == 0 || d % 8) return none();
    const bool expanded = is_tensor(a[9]);
    if (len[2] > 0 && expanded && !part(2, a[9], a[10], len[2], len[0])) return none();
    tq_dequantize_args jobs[2];
    const bool unpack = len[2] > 0 && !expanded;
    for (int i = 0; unpack && i < 2; ++i) {
        PyObject* side = a[7 + i];
        if (!PyTuple_Check(side) || PyTuple_GET_SIZE(side) != 4) return none();
        PyObject* const* s = &PyTuple_GET_ITEM(side, 0);
        if (!PyBytes_Check(s[0]) || PyBytes_GET_SIZE(s[0]) != sizeof(tq_dequantize_args) || !is_tensor(s[1]) || !is_tensor(s[3])) return none();
        const at::Tensor &hi = tensor(s[1]), &norms = tensor(s[3]);
        if (!here(hi, device) || !here(norms, device) || !hi.is_contiguous() || !norms.is_contiguous() || hi.size(0) != b || hi.size(1) != h || len[2] > hi.size(2)) return none();
        std::memcpy(&jobs[i], PyBytes_AS_STRING(s[0]), sizeof jobs[i]);
        if (jobs[i].d != d) return none();
        jobs[i].packed_hi = hi.data_ptr<uint8_t>(); jobs[i].norms = norms.data_ptr<float>();
        if (is_tensor(s[2])) jobs[i].packed_lo = tensor(s[2]).data_ptr<uint8_t>();
        jobs[i].n_lanes = b * h; jobs[i].n_rows = len[2]; jobs[i].in_lane_stride = hi.size(2);
    }
    const int64_t size[4] = {b, h, rows, d};
    at::Tensor k = empty(size, type, device), v = empty(size, type, device);
    for (int i = 0; unpack && i < 2; ++i) {
        jobs[i].out = (i ? v : k).data_ptr<float>() + len[0] * d;
        jobs[i].out_dtype = TQ_F32; jobs[i].out_lane_stride = rows * d;
    }
    f.lanes = b * h; f.out_rows = rows; f.d = int(d); f.out_dtype = type_code(type); f.k_out = k.data_ptr(); f.v_out = v.data_ptr();
    int rc;
    {
        Release gil;
        rc = tq_fetch_dense(&f, unpack ? &jobs[0] : nullptr, unpack ? &jobs[1] : nullptr, stream_of(device));
    }
    if (rc) return rc == TQ_ERR_UNSUPPORTED ? none() : status(rc);
    return PyTuple_Pack(2, THPObjectPtr(THPVariable_Wrap(k)).get(), THPObjectPtr(THPVariable_Wrap(v)).get());
    END_HANDLE_TH_ERRORS
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FAST(codec_quantize), FAST(codec_dequantize), FAST(append), FAST(buffers), FAST(storage), FAST(quantize), FAST(fetch), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Native host path; see csrc/host.cpp.", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__host() {
    PyObject* m = PyModule_Create(&module);
    if (m && PyModule_AddStringConstant(m, "built_for", TQ_BUILT_FOR)) Py_CLEAR(m);       // (the loader compares it with what is running)
    return m;
}
