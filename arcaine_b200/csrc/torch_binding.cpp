// CPython / torch binding of the attention calls: tensors in, C-ABI parameter structs out, one library call.
//
// What bounds a small call is the host, not the GPU: reading tensors, filling the parameter struct, finding the
// stream and the scratch through Python objects and ctypes took 17-38 us per call (a single-token decode step: 27 us
// for 12 us of GPU time).  The same checks and the same struct filled here from at::Tensor take 5-7 us, most of it
// the kernel launches themselves.  Python keeps the signatures and their documentation (ops.py) and passes every
// argument by position.  Errors: ValueError for arguments the binding refuses, ArcError for statuses of the
// library; the texts are those of the Python checks this replaces.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <string>

#include "../../include/arc_sdpa.h"

namespace {

using at::Tensor;

// An exception is already set in the interpreter: unwind to the entry point's handler.
[[noreturn]] void python_failed() { throw python_error(); }

[[noreturn]] void bad(const std::string& text) {
    PyErr_SetString(PyExc_ValueError, text.c_str());
    python_failed();
}

// --------------------------------------------------------------------------- arguments
bool is_none(PyObject* o) { return o == nullptr || o == Py_None; }

const Tensor* tensor_or_null(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

const Tensor& need_tensor(PyObject* o, c10::ScalarType type, const char* name) {
    const Tensor* t = tensor_or_null(o);
    if (!t || !t->is_cuda()) bad(std::string(name) + " must be a CUDA tensor (there is no CPU path)");
    if (t->scalar_type() != type) {
        const char* want = type == at::kBFloat16 ? "torch.bfloat16" : type == at::kFloat ? "torch.float32"
                           : type == at::kInt    ? "torch.int32"    : "torch.int64";
        bad(std::string(name) + " must be " + want + ", got " + c10::toString(t->scalar_type()));
    }
    return *t;
}

int64_t to_int(PyObject* o) {  // int(o)
    if (PyLong_Check(o)) {
        const long long v = PyLong_AsLongLong(o);
        if (v == -1 && PyErr_Occurred()) python_failed();
        return v;
    }
    PyObject* n = PyNumber_Long(o);
    if (!n) python_failed();
    const long long v = PyLong_AsLongLong(n);
    Py_DECREF(n);
    if (v == -1 && PyErr_Occurred()) python_failed();
    return v;
}

float to_float(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) python_failed();
    return static_cast<float>(v);
}

// A reference of this function's own.
struct Held {
    PyObject* o;
    explicit Held(PyObject* owned) : o(owned) {}
    Held(const Held&) = delete;
    ~Held() { Py_XDECREF(o); }
};

PyObject* item(PyObject* o, Py_ssize_t i) {  // o[i], of a tuple, a list, an array, a tensor
    if (PyTuple_Check(o) && i < PyTuple_GET_SIZE(o)) {
        Py_INCREF(PyTuple_GET_ITEM(o, i));
        return PyTuple_GET_ITEM(o, i);
    }
    const Held index(PyLong_FromSsize_t(i));
    PyObject* r = index.o ? PyObject_GetItem(o, index.o) : nullptr;
    if (!r) python_failed();
    return r;
}

bool to_bool(PyObject* o) {
    const int v = PyObject_IsTrue(o);
    if (v < 0) python_failed();
    return v != 0;
}

// --------------------------------------------------------------------------- shapes
// Address, sizes and strides (elements) of a tensor of 16-bit values, without a tensor object per view.
struct View {
    char* ptr = nullptr;
    int dim = 0;
    int64_t n[4] = {0, 0, 0, 0}, st[4] = {0, 0, 0, 0};
    bool given() const { return dim > 0; }
};

View view_of(const Tensor& t, const char* name) {
    View v;
    v.dim = static_cast<int>(t.dim());
    if (v.dim > 4) bad(std::string(name) + " must have 3 or 4 dims");
    v.ptr = static_cast<char*>(t.data_ptr());
    for (int i = 0; i < v.dim; ++i) {
        v.n[i] = t.size(i);
        v.st[i] = t.stride(i);
    }
    return v;
}

View unsqueeze0(const View& a) {
    View v = a;
    v.dim = a.dim + 1;
    v.n[0] = 1;
    v.st[0] = a.dim ? a.n[0] * a.st[0] : 1;
    for (int i = 0; i < a.dim; ++i) {
        v.n[i + 1] = a.n[i];
        v.st[i + 1] = a.st[i];
    }
    return v;
}

// t.view(a, b, c); a may be -1.
View view3(const Tensor& t, int64_t a, int64_t b, int64_t c, const char* name) {
    const int64_t bc = b * c, numel = t.numel();
    if (a == -1 && bc > 0 && numel % bc == 0) a = numel / bc;
    if (!t.is_contiguous() || a < 0 || a * bc != numel) return view_of(t.view({a, b, c}), name);  // or its error
    View v;
    v.dim = 3;
    v.ptr = static_cast<char*>(t.data_ptr());
    v.n[0] = a, v.n[1] = b, v.n[2] = c;
    v.st[0] = bc, v.st[1] = c, v.st[2] = 1;
    return v;
}

// v[begin : end] along the first dimension, with Python's rules for ends out of range.
View rows(View v, int64_t begin, int64_t end) {
    const int64_t n = v.n[0];
    auto clamp = [n](int64_t i) { return i < 0 ? (i + n < 0 ? 0 : i + n) : (i > n ? n : i); };
    begin = clamp(begin), end = clamp(end);
    v.n[0] = end > begin ? end - begin : 0;
    v.ptr += begin * v.st[0] * 2;
    return v;
}

void token_strides(const View& v, const char* name, int64_t* sb, int64_t* st) {
    if (v.st[3] != 1 || v.st[2] != v.n[3])
        bad(std::string(name) + ": the (heads, head_dim) block of every token must be contiguous");
    *sb = v.st[0];
    *st = v.st[1];
}

// A buffer the library writes (or reads) as (n0, n1, row) must hold that many: it is given addresses and strides only.
void need_room(const View& v, int64_t n0, int64_t n1, int64_t row, const char* name) {
    if (v.n[0] < n0 || v.n[1] < n1 || v.n[2] * v.n[3] < row) bad(std::string(name) + " is smaller than the call needs");
}

bool same_layout(const View& a, const View& b) {
    if (a.dim != b.dim) return false;
    for (int i = 0; i < a.dim; ++i)
        if (a.n[i] != b.n[i] || a.st[i] != b.st[i]) return false;
    return true;
}

Tensor new_cuda(at::IntArrayRef sizes, c10::ScalarType type, c10::Device device) {
    return at::detail::empty_cuda(sizes, type, device, std::nullopt);
}

// --------------------------------------------------------------------------- library calls
PyObject* g_check = nullptr;          // _lib.check(status, where): raises ArcError
PyObject* g_reserve = nullptr;        // "reserve"

void check_status(int status, const char* where) {
    if (status == ARC_OK) return;
    PyObject* r = PyObject_CallFunction(g_check, "is", status, where);
    Py_XDECREF(r);
    python_failed();
}

// Scratch of a call: from the caller's Workspace, or an allocation of the call's own on its stream, which the caching
// allocator hands out again behind it, so that two streams, threads or captured graphs never share one (0.2 us more than
// a buffer per device took).  Held until the launches are enqueued: that happens without the GIL, and a Workspace may let
// go of its buffer meanwhile.
struct Scratch {
    c10::DataPtr own;
    Tensor borrowed;

    // At least `need` bytes, on the current device and stream.
    void take(PyObject* workspace, size_t need, void** ptr, size_t* bytes) {
        if (is_none(workspace)) {
            own = c10::cuda::CUDACachingAllocator::get()->allocate(need);
            *ptr = own.get();
            *bytes = need;
            return;
        }
        PyObject* n = PyLong_FromSize_t(need);
        PyObject* buf = n ? PyObject_CallMethodOneArg(workspace, g_reserve, n) : nullptr;
        Py_XDECREF(n);
        if (!buf) python_failed();
        if (const Tensor* t = tensor_or_null(buf)) borrowed = *t;
        Py_DECREF(buf);
        if (!borrowed.defined()) bad("workspace.reserve() must return a tensor");
        *ptr = borrowed.data_ptr();
        *bytes = static_cast<size_t>(borrowed.numel()) * borrowed.element_size();
    }
};

template <typename F>
int without_gil(F&& f) {
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = f();
    Py_END_ALLOW_THREADS
    return rc;
}

struct PrefillExtra {
    View gate;
    PyObject* mask = nullptr;
    PyObject* block_ids = nullptr;
    int64_t block_ids_offset = 0;
    PyObject* out_copies = nullptr;
    PyObject* workspace = nullptr;
    float* lse = nullptr;
    int num_splits = 0;
};

// The one prefill call.  q, k, v, out (and gate) are four-dimensional views on `device`.
void run_prefill(c10::Device device, const View& q, const View& k, const View& v, const View& out, float scale,
                 int mask_type, int64_t window, const PrefillExtra& x) {
    const int64_t B = q.n[0], S = q.n[1], L = k.n[1];
    for (int i = 0; i < 4; ++i)
        if (v.n[i] != k.n[i]) bad("k/v shape mismatch");
    if (k.n[0] != B || k.n[3] != q.n[3]) bad("k/v shape mismatch");
    arc_sdpa_prefill_params p{};
    p.q = q.ptr, p.k = k.ptr, p.v = v.ptr, p.out = out.ptr;
    if (x.gate.given()) {
        if (!same_layout(x.gate, out)) bad("gate must be laid out like out");
        p.gate = x.gate.ptr;
    }
    if (!is_none(x.mask)) {
        const Tensor& m = need_tensor(x.mask, at::kFloat, "mask");
        if (m.dim() != 2 || m.size(0) != S || m.size(1) != L || !m.is_contiguous())
            bad("mask must be a contiguous (seq, kv_len) f32 tensor");
        p.mask = static_cast<const float*>(m.data_ptr());
    }
    p.out_lse = x.lse;
    p.batch = (int32_t)B, p.seq = (int32_t)S, p.kv_len = (int32_t)L;
    p.nq = (int32_t)q.n[2], p.nkv = (int32_t)k.n[2], p.hd = (int32_t)q.n[3];
    token_strides(q, "q", &p.q_stride_b, &p.q_stride_t);
    token_strides(k, "k", &p.k_stride_b, &p.k_stride_t);
    token_strides(v, "v", &p.v_stride_b, &p.v_stride_t);
    token_strides(out, "out", &p.o_stride_b, &p.o_stride_t);
    need_room(out, B, S, q.n[2] * q.n[3], "out");
    p.scale = scale, p.mask_type = mask_type, p.window = (int32_t)window, p.num_splits = x.num_splits;
    if (!is_none(x.block_ids)) {
        const Tensor& ids = need_tensor(x.block_ids, at::kInt, "block_ids");
        if (!ids.is_contiguous() || ids.numel() < x.block_ids_offset + L || x.block_ids_offset < 0)
            bad("block_ids must be contiguous and hold block_ids_offset + kv_len entries");
        p.block_ids = static_cast<const int32_t*>(ids.data_ptr());
        p.block_ids_offset = (int32_t)x.block_ids_offset;
    }
    if (!is_none(x.out_copies)) {
        const Tensor& c = need_tensor(x.out_copies, at::kLong, "out_copies");
        if (!c.is_contiguous() || c.numel() > 15) bad("out_copies must be a contiguous int64 tensor of at most 15 addresses");
        p.out_copies = static_cast<const uint64_t*>(c.data_ptr());
        p.out_copy_count = (int32_t)c.numel();
    }
    const c10::cuda::CUDAGuard guard(device);
    const size_t need = arc_sdpa_prefill_workspace_bytes(&p);
    Scratch scratch;
    if (need) scratch.take(x.workspace, need, &p.workspace, &p.workspace_bytes);
    void* stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
    check_status(without_gil([&] { return arc_sdpa_prefill(&p, stream); }), "arc_sdpa_prefill");
}

void need_args(Py_ssize_t got, Py_ssize_t want, const char* name) {
    if (got != want) bad(std::string(name) + ": wrong number of arguments");
}

PyObject* wrap(const Tensor& t) { return THPVariable_Wrap(t); }

PyObject* again(PyObject* o) {
    Py_INCREF(o);
    return o;
}

// sdpa_prefill(q, k, v, scale, mask_type, window, mask, gate, out, num_splits, return_lse, workspace, block_ids,
//              block_ids_offset, out_copies)
PyObject* py_prefill(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    need_args(n, 15, "sdpa_prefill");
    const Tensor& tq = need_tensor(a[0], at::kBFloat16, "q");
    const Tensor& tk = need_tensor(a[1], at::kBFloat16, "k");
    const Tensor& tv = need_tensor(a[2], at::kBFloat16, "v");
    View q = view_of(tq, "q"), k = view_of(tk, "k"), v = view_of(tv, "v");
    const bool three = q.dim == 3;
    auto four = [three](View& t, const char* name) {
        if (t.dim != (three ? 3 : 4)) bad(std::string(name) + " must have 3 or 4 dims");
        if (three) t = unsqueeze0(t);
    };
    four(q, "q");
    four(k, "k");
    four(v, "v");
    PrefillExtra x;
    Tensor made;
    View out;
    if (is_none(a[8])) {
        made = three ? new_cuda({q.n[1], q.n[2], q.n[3]}, at::kBFloat16, tq.device())
                     : new_cuda({q.n[0], q.n[1], q.n[2], q.n[3]}, at::kBFloat16, tq.device());
        out = view_of(made, "out");
    } else {
        out = view_of(need_tensor(a[8], at::kBFloat16, "out"), "out");
    }
    four(out, "out");
    if (!is_none(a[7])) {
        x.gate = view_of(need_tensor(a[7], at::kBFloat16, "gate"), "gate");
        four(x.gate, "gate");
    }
    Tensor lse;
    const bool want_lse = to_bool(a[10]);
    if (want_lse) {
        lse = three ? new_cuda({q.n[1], q.n[2]}, at::kFloat, tq.device())
                    : new_cuda({q.n[0], q.n[1], q.n[2]}, at::kFloat, tq.device());
        x.lse = static_cast<float*>(lse.data_ptr());
    }
    x.mask = a[6], x.workspace = a[11], x.block_ids = a[12], x.out_copies = a[14];
    x.num_splits = (int)to_int(a[9]);
    x.block_ids_offset = to_int(a[13]);
    run_prefill(tq.device(), q, k, v, out, to_float(a[3]), (int)to_int(a[4]), to_int(a[5]), x);
    PyObject* res = made.defined() ? wrap(made) : again(a[8]);
    if (!want_lse) return res;
    return Py_BuildValue("(NN)", res, wrap(lse));
    END_HANDLE_TH_ERRORS
}

// One sequence, token-major: attention(Q, seq, nq, hd, K, V, kv_len, nkv, scale, mask_type, window, mask, out,
//                                      block_ids, block_ids_offset, flat).  flat: K and V may be one-dimensional.
PyObject* py_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    need_args(n, 16, "attention");
    const bool flat = to_bool(a[15]);
    const Tensor& tq = need_tensor(a[0], at::kBFloat16, "q");
    const Tensor& tk = need_tensor(a[4], at::kBFloat16, "k");
    const Tensor& tv = need_tensor(a[5], at::kBFloat16, "v");
    const int64_t seq = to_int(a[1]), nq = to_int(a[2]), hd = to_int(a[3]), kv_len = to_int(a[6]), nkv = to_int(a[7]);
    View q = unsqueeze0(view3(tq, seq, nq, hd, "q"));
    auto cache = [&](const Tensor& t, const char* name) {
        if (flat && t.dim() == 1) return unsqueeze0(view3(t.slice(0, 0, kv_len * nkv * hd), kv_len, nkv, hd, name));
        View v = view_of(t, name);
        if (v.dim != 3) bad(std::string(name) + " must have 3 or 4 dims");
        return unsqueeze0(rows(v, 0, kv_len));
    };
    const View k = cache(tk, "k"), v = cache(tv, "v");
    PrefillExtra x;
    Tensor made;
    View out;
    if (is_none(a[12])) {
        made = new_cuda({seq, nq, hd}, at::kBFloat16, tq.device());
        out = view_of(made, "out");
    } else {
        out = view_of(need_tensor(a[12], at::kBFloat16, "out"), "out");
        if (out.dim != 3) bad("out must have 3 dims");
    }
    x.mask = a[11], x.block_ids = a[13];
    x.block_ids_offset = to_int(a[14]);
    run_prefill(tq.device(), q, k, v, unsqueeze0(out), to_float(a[8]), (int)to_int(a[9]), to_int(a[10]), x);
    return made.defined() ? wrap(made) : again(a[12]);
    END_HANDLE_TH_ERRORS
}

// --------------------------------------------------------------------------- decode
struct DecodeExtra {
    View gate;
    PyObject* kv_len = nullptr;   // None: the whole cache; an int; or an int32 tensor (B,)
    bool kv_len_known = false;    // kv_len_int is used instead of the object
    int64_t kv_len_int = 0;
    PyObject* row_offset = nullptr;
    PyObject* workspace = nullptr;
    PyObject* exchange = nullptr;
    int64_t exchange_wait = 0;
    float* out_f32 = nullptr;
    float* out_lse = nullptr;
    int num_ctas = 0;
};

void run_decode(c10::Device device, const View& q, const View& k, const View& v, const View& out, float scale,
                const DecodeExtra& x) {
    if (q.dim != 3) bad("q must be (B, nq, hd)");
    const int64_t B = q.n[0], nq = q.n[1], hd = q.n[2];
    if (q.st[2] != 1 || q.st[1] != hd) bad("q: (nq, hd) must be contiguous");
    arc_sdpa_decode_params p{};
    int64_t max_len, nkv, hdk;
    if (k.dim == 4) {
        if (!is_none(x.row_offset)) bad("kv_row_offset needs packed (rows, nkv, hd) caches");
        bool same = v.dim == 4;
        for (int i = 0; same && i < 4; ++i) same = v.n[i] == k.n[i];
        if (k.n[0] != B || !same) bad("k/v shape mismatch");
        max_len = k.n[1], nkv = k.n[2], hdk = k.n[3];
        if (k.st[3] != 1 || k.st[2] != hdk || !same_layout(k, v) || k.st[1] == 0 || k.st[0] % k.st[1])
            bad("k/v: unsupported strides");
        p.kv_stride_t = k.st[1];
        p.kv_stride_b = max_len == 0 ? 0 : k.st[0] / k.st[1];  // (an empty slice has no rows at all)
        p.kv_rows_total = (B - 1) * p.kv_stride_b + max_len;
    } else if (k.dim == 3) {
        max_len = k.n[0], nkv = k.n[1], hdk = k.n[2];
        if (k.st[2] != 1 || k.st[1] != hdk || !same_layout(k, v)) bad("k/v: unsupported strides");
        p.kv_stride_t = k.st[0];
        p.kv_stride_b = 0;
        p.kv_rows_total = max_len;
        if (is_none(x.row_offset) && B > 1) bad("packed caches need kv_row_offset");
    } else {
        bad("k must have 3 or 4 dims");
    }
    if (hdk != hd) bad("head_dim mismatch");
    if (!x.kv_len_known && !is_none(x.kv_len) && tensor_or_null(x.kv_len)) {
        const Tensor& t = need_tensor(x.kv_len, at::kInt, "kv_len");
        if (t.dim() != 1 || t.size(0) != B || !t.is_contiguous()) bad("kv_len must be a contiguous (B,) int32 tensor");
        p.kv_len = static_cast<const int32_t*>(t.data_ptr());
    } else {
        const int64_t len = x.kv_len_known ? x.kv_len_int : is_none(x.kv_len) ? max_len : to_int(x.kv_len);
        if (len > max_len) bad("kv_len exceeds the cache");
        p.kv_len_uniform = (int32_t)len;
    }
    if (!is_none(x.row_offset)) {
        const Tensor& t = need_tensor(x.row_offset, at::kLong, "kv_row_offset");
        if (t.dim() != 1 || t.size(0) != B || !t.is_contiguous()) bad("kv_row_offset must be a contiguous (B,) int64 tensor");
        p.kv_row_offset = static_cast<const int64_t*>(t.data_ptr());
    }
    p.max_kv_len = (int32_t)max_len;
    if (out.given()) {
        if (out.dim != 3 || out.n[0] != B || out.n[1] != nq || out.n[2] != hd || out.st[2] != 1 || out.st[1] != hd)
            bad("out must be laid out like q");
        p.out = out.ptr;
        p.o_stride_b = out.st[0];
    }
    if (x.gate.given()) {
        if (!out.given() || !same_layout(x.gate, out)) bad("gate must be laid out like out");
        p.gate = x.gate.ptr;
    }
    p.out_f32 = x.out_f32, p.out_lse = x.out_lse;
    p.q = q.ptr, p.k = k.ptr, p.v = v.ptr;
    p.batch = (int32_t)B, p.nq = (int32_t)nq, p.nkv = (int32_t)nkv, p.hd = (int32_t)hd;
    p.q_stride_b = q.st[0];
    p.scale = scale, p.num_ctas = x.num_ctas;
    if (!is_none(x.exchange)) {
        const Held peers(item(x.exchange, 0)), world(item(x.exchange, 1)), rank(item(x.exchange, 2)), step(item(x.exchange, 3));
        if (PyObject_Size(x.exchange) != 4) bad("exchange must be (peers, world, rank, step)");
        p.xchg_peers = static_cast<const uint64_t*>(need_tensor(peers.o, at::kLong, "exchange peers").data_ptr());
        p.xchg_world = (int32_t)to_int(world.o), p.xchg_rank = (int32_t)to_int(rank.o);
        p.xchg_step = (uint32_t)(to_int(step.o) & 0xFFFFFFFFll);
        p.xchg_wait_cycles = x.exchange_wait;
    }
    const c10::cuda::CUDAGuard guard(device);
    const size_t need = arc_sdpa_decode_workspace_bytes(&p);
    Scratch scratch;
    if (need) scratch.take(x.workspace, need, &p.workspace, &p.workspace_bytes);
    void* stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
    check_status(without_gil([&] { return arc_sdpa_decode(&p, stream); }), "arc_sdpa_decode");
}

// sdpa_decode(q, k, v, scale, kv_len, kv_row_offset, gate, out, return_partial, want_out, num_ctas, partial_out,
//             partial_lse, exchange, workspace, exchange_wait_cycles)
PyObject* py_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    need_args(n, 16, "sdpa_decode");
    const Tensor& tq = need_tensor(a[0], at::kBFloat16, "q");
    const Tensor& tk = need_tensor(a[1], at::kBFloat16, "k");
    const Tensor& tv = need_tensor(a[2], at::kBFloat16, "v");
    const View q = view_of(tq, "q");
    if (q.dim != 3) bad("q must be (B, nq, hd)");
    DecodeExtra x;
    x.kv_len = a[4], x.row_offset = a[5], x.exchange = a[13], x.workspace = a[14];
    x.num_ctas = (int)to_int(a[10]);
    x.exchange_wait = to_int(a[15]);
    Tensor made;
    View out;
    if (!is_none(a[7])) out = view_of(need_tensor(a[7], at::kBFloat16, "out"), "out");
    else if (to_bool(a[9])) {
        made = new_cuda({q.n[0], q.n[1], q.n[2]}, at::kBFloat16, tq.device());
        out = view_of(made, "out");
    }
    if (!is_none(a[6])) x.gate = view_of(need_tensor(a[6], at::kBFloat16, "gate"), "gate");
    const bool partial = to_bool(a[8]);
    Tensor o32, lse;
    if (partial) {
        o32 = is_none(a[11]) ? new_cuda({q.n[0], q.n[1], q.n[2]}, at::kFloat, tq.device())
                             : need_tensor(a[11], at::kFloat, "partial_out");
        lse = is_none(a[12]) ? new_cuda({q.n[0], q.n[1]}, at::kFloat, tq.device()) : need_tensor(a[12], at::kFloat, "partial_lse");
        const bool shapes = o32.dim() == 3 && o32.size(0) == q.n[0] && o32.size(1) == q.n[1] && o32.size(2) == q.n[2] &&
                            lse.dim() == 2 && lse.size(0) == q.n[0] && lse.size(1) == q.n[1];
        if (!shapes || !o32.is_contiguous() || !lse.is_contiguous())
            bad("partial_out / partial_lse must be contiguous (B, nq, hd) / (B, nq) f32");
        x.out_f32 = static_cast<float*>(o32.data_ptr());
        x.out_lse = static_cast<float*>(lse.data_ptr());
    }
    run_decode(tq.device(), q, view_of(tk, "k"), view_of(tv, "v"), out, to_float(a[3]), x);
    PyObject* res = made.defined() ? wrap(made) : again(is_none(a[7]) ? Py_None : a[7]);
    if (!partial) return res;
    return Py_BuildValue("(NNN)", res, wrap(o32), wrap(lse));
    END_HANDLE_TH_ERRORS
}

// One token of one sequence over rows [begin, end) of a token-major cache:
// decode_one(Q, K, V, out, begin, end, nq, nkv, hd, scale, gate, reshape).  reshape: K and V are viewed as
// (rows, nkv, hd) first.  Returns out, or a new (nq, hd) tensor.
PyObject* py_decode_one(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    need_args(n, 12, "decode_one");
    const Tensor& tq = need_tensor(a[0], at::kBFloat16, "q");
    const Tensor& tk = need_tensor(a[1], at::kBFloat16, "k");
    const Tensor& tv = need_tensor(a[2], at::kBFloat16, "v");
    const int64_t begin = to_int(a[4]), end = to_int(a[5]), nq = to_int(a[6]), nkv = to_int(a[7]), hd = to_int(a[8]);
    const bool reshape = to_bool(a[11]);
    auto cache = [&](const Tensor& t, const char* name) {
        return rows(reshape ? view3(t, -1, nkv, hd, name) : view_of(t, name), begin, end);  // (or a block of one sequence)
    };
    Tensor made;
    View out;
    if (is_none(a[3])) {
        made = new_cuda({nq, hd}, at::kBFloat16, tq.device());
        out = view3(made, 1, nq, hd, "out");
    } else {
        out = view3(need_tensor(a[3], at::kBFloat16, "out"), 1, nq, hd, "out");
    }
    DecodeExtra x;
    if (!is_none(a[10])) x.gate = view3(need_tensor(a[10], at::kBFloat16, "gate"), 1, nq, hd, "gate");
    x.kv_len_known = true, x.kv_len_int = end - begin;
    run_decode(tq.device(), view3(tq, 1, nq, hd, "q"), cache(tk, "k"), cache(tv, "v"), out, to_float(a[9]), x);
    return made.defined() ? wrap(made) : again(a[3]);
    END_HANDLE_TH_ERRORS
}

// qwen_attention(query, key, value, output, seq, past, nq, hd, scale): causal over past + seq keys, one token as a
// decode.  Returns output.
PyObject* py_qwen_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    need_args(n, 9, "qwen_attention");
    const Tensor& tq = need_tensor(a[0], at::kBFloat16, "q");
    const View k0 = view_of(need_tensor(a[1], at::kBFloat16, "k"), "k"), v0 = view_of(need_tensor(a[2], at::kBFloat16, "v"), "v");
    const int64_t seq = to_int(a[4]), past = to_int(a[5]), nq = to_int(a[6]), hd = to_int(a[7]);
    const View q = rows(view3(tq, -1, nq, hd, "q"), 0, seq);
    const View o = rows(view3(need_tensor(a[3], at::kBFloat16, "out"), -1, nq, hd, "out"), 0, seq);
    const View k = rows(k0, 0, past + seq), v = rows(v0, 0, past + seq);
    if (seq == 1) {  // (also over a block of one sequence)
        DecodeExtra x;
        x.kv_len_known = true, x.kv_len_int = past + 1;
        run_decode(tq.device(), q, k, v, o, to_float(a[8]), x);
    } else {
        if (k.dim != 3 || v.dim != 3) bad("k must have 3 or 4 dims");
        run_prefill(tq.device(), unsqueeze0(q), unsqueeze0(k), unsqueeze0(v), unsqueeze0(o), to_float(a[8]), ARC_MASK_CAUSAL,
                    ARC_NO_WINDOW, PrefillExtra());
    }
    return again(a[3]);
    END_HANDLE_TH_ERRORS
}

// --------------------------------------------------------------------------- pre-processing
// qkv_prepare(q, k, v, k_cache, v_cache, past_len, q_weight, k_weight, eps, theta, partial_rotary_factor, rope_cos,
//             rope_sin, pos_offset, v_from_k, rotary_dim, mrope_positions, mrope_section, v_copy)
PyObject* py_qkv_prepare(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    need_args(n, 19, "qkv_prepare");
    if (is_none(a[0]) && is_none(a[1])) bad("qkv_prepare needs q or k");
    const Tensor& ref = need_tensor(is_none(a[0]) ? a[1] : a[0], at::kBFloat16, is_none(a[0]) ? "k" : "q");
    const bool three = ref.dim() == 3;
    auto get = [&](int i, const char* name) {
        if (is_none(a[i])) return View();
        View v = view_of(need_tensor(a[i], at::kBFloat16, name), name);
        if (v.dim != (three ? 3 : 4)) bad(std::string(name) + " must have 3 or 4 dims, as q and k");
        return three ? unsqueeze0(v) : v;
    };
    const View q = get(0, "q"), k = get(1, "k"), v = get(2, "v"), kc = get(3, "k_cache"), vc = get(4, "v_cache");
    const View& r = q.given() ? q : k;
    const int64_t past = to_int(a[5]), B = r.n[0], S = r.n[1], hd = r.n[3];
    const bool v_from_k = to_bool(a[14]);
    if (past < 0 && (kc.given() || vc.given())) bad("past_len must not be negative");
    arc_qkv_prepare_params p{};
    if (q.given()) {
        p.q = q.ptr, p.nq = (int32_t)q.n[2];
        token_strides(q, "q", &p.q_stride_b, &p.q_stride_t);
    }
    if (k.given()) {
        p.k_src = k.ptr, p.nkv = (int32_t)k.n[2];
        const int64_t row = k.n[2] * hd;
        need_room(k, B, S, row, "k");
        token_strides(k, "k", &p.k_src_stride_b, &p.k_src_stride_t);
        if (kc.given() && past + S > kc.n[1]) bad("KV cache capacity exceeded");
        if (kc.given()) need_room(kc, B, past + S, row, "k_cache");
        const View& kd = kc.given() ? kc : k;
        token_strides(kd, "k_cache", &p.k_dst_stride_b, &p.k_dst_stride_t);
        p.k_dst = kd.ptr + (kc.given() ? past : 0) * p.k_dst_stride_t * 2;
        if (v.given() || v_from_k) {
            const View& vd = vc.given() ? vc : v;
            if (!vd.given()) bad("v_from_k needs v_cache");
            if (v_from_k && !kc.given())  // K would be rewritten in place while V is still being read from it
                bad("v_from_k needs k_cache: K cannot be normalised in place when V is taken from it");
            need_room(vd, B, vc.given() ? past + S : S, row, vc.given() ? "v_cache" : "v");
            if (v.given() && !v_from_k) need_room(v, B, S, row, "v");
            token_strides(vd, "v_cache", &p.v_dst_stride_b, &p.v_dst_stride_t);
            p.v_dst = vd.ptr + (vc.given() ? past : 0) * p.v_dst_stride_t * 2;
            if (v.given() && !v_from_k) {
                p.v_src = v.ptr;
                token_strides(v, "v", &p.v_src_stride_b, &p.v_src_stride_t);
            }
        }
    }
    auto values = [](const Tensor& t, int64_t n, const char* name) {  // the address of n values in a row
        if (t.numel() < n) bad(std::string(name) + " is smaller than the call needs");
        return t.data_ptr();
    };
    if (!is_none(a[6])) p.q_weight = values(need_tensor(a[6], at::kBFloat16, "q_weight"), hd, "q_weight");
    if (!is_none(a[7])) p.k_weight = values(need_tensor(a[7], at::kBFloat16, "k_weight"), hd, "k_weight");
    p.batch = (int32_t)B, p.seq = (int32_t)S, p.hd = (int32_t)hd;
    const double partial = PyFloat_AsDouble(a[10]);
    if (partial == -1.0 && PyErr_Occurred()) python_failed();
    p.n_active_pairs = (int32_t)(partial * (double)hd / 2.0);
    if (!is_none(a[11])) {
        const Tensor& c = need_tensor(a[11], at::kFloat, "rope_cos");
        const Tensor& s = need_tensor(a[12], at::kFloat, "rope_sin");
        if (!c.is_contiguous() || !s.is_contiguous()) bad("rope tables must be contiguous");
        p.rope_stride_b = c.dim() == 3 ? S * p.n_active_pairs : 0;
        const int64_t pairs = is_none(a[15]) ? p.n_active_pairs : to_int(a[15]) / 2;
        const int64_t angles = S * pairs + (B - 1) * p.rope_stride_b;
        p.rope_cos = static_cast<const float*>(values(c, angles, "rope_cos"));
        p.rope_sin = static_cast<const float*>(values(s, angles, "rope_sin"));
    }
    if (!is_none(a[13]) && tensor_or_null(a[13]))
        p.pos_offset = static_cast<const int32_t*>(values(need_tensor(a[13], at::kInt, "pos_offset"), B, "pos_offset"));
    else
        p.pos0 = (int32_t)(is_none(a[13]) ? past : to_int(a[13]));
    p.eps = to_float(a[8]), p.theta = to_float(a[9]);
    if (!is_none(a[15])) {
        const int64_t rd = to_int(a[15]);
        p.rot_half = (int32_t)(rd / 2), p.freq_denom = (int32_t)rd, p.n_active_pairs = (int32_t)(rd / 2);
    }
    if (!is_none(a[16])) {
        const Tensor& pos = need_tensor(a[16], at::kInt, "mrope_positions");
        if (!pos.is_contiguous() || pos.numel() != B * 3 * S) bad("mrope_positions must be a contiguous (B, 3, S) int32 tensor");
        p.mrope_positions = static_cast<const int32_t*>(pos.data_ptr());
        if (is_none(a[17]) || PyObject_Size(a[17]) != 3) bad("Qwen3.5 MRoPE needs three sections");
        for (int i = 0; i < 3; ++i) p.mrope_section[i] = (int32_t)to_int(Held(item(a[17], i)).o);
    }
    p.v_copy = to_bool(a[18]) ? 1 : 0;
    const c10::cuda::CUDAGuard guard(ref.device());
    void* stream = c10::cuda::getCurrentCUDAStream(ref.device().index()).stream();
    check_status(without_gil([&] { return arc_qkv_prepare(&p, stream); }), "arc_qkv_prepare");
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

// --------------------------------------------------------------------------- small calls
// mul_sigmoid_inplace(a, gate) -> a
PyObject* py_mul_sigmoid(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    need_args(n, 2, "mul_sigmoid_inplace");
    const Tensor& t = need_tensor(a[0], at::kBFloat16, "a");
    const Tensor& g = need_tensor(a[1], at::kBFloat16, "gate");
    if (!t.is_contiguous() || !g.is_contiguous() || t.numel() != g.numel()) bad("a and gate must be contiguous and of equal size");
    const c10::cuda::CUDAGuard guard(t.device());
    void* stream = c10::cuda::getCurrentCUDAStream(t.device().index()).stream();
    check_status(without_gil([&] { return arc_mul_sigmoid_inplace(t.data_ptr(), g.data_ptr(), t.numel(), stream); }),
                 "arc_mul_sigmoid_inplace");
    return again(a[0]);
    END_HANDLE_TH_ERRORS
}

// fill_causal_mask(out, q_len, kv_len, past_offset, window) -> out
PyObject* py_fill_causal_mask(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    need_args(n, 5, "fill_causal_mask");
    const Tensor& out = need_tensor(a[0], at::kFloat, "out");
    const int q_len = (int)to_int(a[1]), kv_len = (int)to_int(a[2]), past = (int)to_int(a[3]), window = (int)to_int(a[4]);
    const c10::cuda::CUDAGuard guard(out.device());
    void* stream = c10::cuda::getCurrentCUDAStream(out.device().index()).stream();
    if (!out.is_contiguous() || (q_len > 0 && kv_len > 0 && out.numel() < (int64_t)q_len * kv_len))
        bad("out must be contiguous and hold q_len * kv_len values");
    float* mask = static_cast<float*>(out.data_ptr());
    check_status(without_gil([&] { return arc_fill_causal_mask(mask, q_len, kv_len, past, window, stream); }), "arc_fill_causal_mask");
    return again(a[0]);
    END_HANDLE_TH_ERRORS
}

// setup(check): the Python callable the binding needs.
PyObject* py_setup(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 1) {
        PyErr_SetString(PyExc_TypeError, "setup(check)");
        return nullptr;
    }
    g_check = again(a[0]);
    g_reserve = PyUnicode_InternFromString("reserve");
    Py_RETURN_NONE;
}

#define ARC_METHOD(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {
    ARC_METHOD("setup", py_setup),
    ARC_METHOD("sdpa_prefill", py_prefill),
    ARC_METHOD("attention", py_attention),
    ARC_METHOD("sdpa_decode", py_decode),
    ARC_METHOD("decode_one", py_decode_one),
    ARC_METHOD("qwen_attention", py_qwen_attention),
    ARC_METHOD("qkv_prepare", py_qkv_prepare),
    ARC_METHOD("mul_sigmoid_inplace", py_mul_sigmoid),
    ARC_METHOD("fill_causal_mask", py_fill_causal_mask),
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", "Tensor binding of libarc_sdpa.so", -1, g_methods,
                        nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&g_module); }
