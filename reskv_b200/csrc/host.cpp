// Native host path of the decode-step calls: a CPython module (`_host`) that takes torch tensors, checks them,
// allocates results and scratch from torch's caching allocator and calls the C ABI of libreskv_b200.so.
//
// Why native: a batch-1 decode attention is two kernels of ~8 us each, and the same work in Python (30 tensor
// attribute reads, four allocations, a 30-argument ctypes call) took 65 us per call, so the GPU waited for the host
// up to batch 8.  Nothing is kept between calls here: every pointer and size is read from the tensors of the call.
#include <ATen/ATen.h>
#include <ATen/TensorSubclassLikeUtils.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <Python.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/python_variable.h>

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/reskv_b200.h"

namespace {

struct PyError {};  // a Python exception is set

// An error found while the interpreter lock is not held; `guarded` makes the Python exception of it.
struct Failure {
    PyObject* type;
    std::string text;
};

[[noreturn]] void value_error(std::string msg) { throw Failure{PyExc_ValueError, std::move(msg)}; }

// The exception a failed library call stands for: argument problems are ValueError, the rest RuntimeError.
void check(int rc) {
    if (rc >= 0) return;
    throw Failure{rc == RESKV_ERR_INVALID || rc == RESKV_ERR_LIMIT ? PyExc_ValueError : PyExc_RuntimeError, reskv_last_error()};
}

void check_cuda(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return;
    cudaGetLastError();
    throw Failure{PyExc_RuntimeError, std::string(what) + ": " + cudaGetErrorString(e)};
}

// Everything from the first allocation to the last launch of a call runs without the interpreter lock: an allocation may go
// to cudaMalloc and a launch waits when the stream's queue is full, and the other Python threads are to run meanwhile.  What
// a call needs of its arguments is taken (tensors by reference count) before.  Letting go and taking it again costs 0.2 to
// 0.3 us when no other thread wants it (attention 7.9 -> 8.1 us of host time, window_append 6.9 -> 7.2).
class Unlocked {
public:
    Unlocked() : state_(PyEval_SaveThread()) {}
    ~Unlocked() { PyEval_RestoreThread(state_); }
    Unlocked(const Unlocked&) = delete;
    Unlocked& operator=(const Unlocked&) = delete;

private:
    PyThreadState* state_;
};

std::atomic<long long> g_launches{0};  // kernels launched through this module
bool g_check_status = false;

at::Tensor tensor(PyObject* o, const char* what) {
    if (!THPVariable_Check(o)) {
        PyErr_Format(PyExc_TypeError, "%s must be a tensor", what);
        throw PyError{};
    }
    return THPVariable_Unpack(o);
}
// None -> undefined tensor
at::Tensor optional_tensor(PyObject* o, const char* what) { return o == Py_None ? at::Tensor() : tensor(o, what); }

long long integer(PyObject* o) {  // int(o)
    PyObject* i = PyLong_Check(o) ? Py_NewRef(o) : PyNumber_Long(o);
    const long long v = i ? PyLong_AsLongLong(i) : -1;
    Py_XDECREF(i);
    if (v == -1 && PyErr_Occurred()) throw PyError{};
    return v;
}
double number(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw PyError{};
    return v;
}
PyObject* item(PyObject* tuple, Py_ssize_t i) {
    PyObject* o = PyTuple_Check(tuple) ? PyTuple_GetItem(tuple, i) : nullptr;
    if (!o) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "expected a tuple");
        throw PyError{};
    }
    return o;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

const void* data(const at::Tensor& t) { return t.defined() && t.numel() ? t.const_data_ptr() : nullptr; }

void same_device(c10::DeviceIndex dev, const at::Tensor& t) {
    if (t.defined() && (!t.is_cuda() || t.get_device() != dev))
        value_error("all tensors of this call must live on cuda:" + std::to_string(static_cast<int>(dev)) + ", got one on " + t.device().str());
}

// A tensor whose memory a kernel may read behind the dispatcher's back: nothing that a tensor operation would do with it
// besides is lost (a gradient or a forward-mode tangent, the wrappers of vmap, jvp and functionalisation, a subclass or a
// mode that wants to see the operation, a trace being recorded), and it has memory at all.
bool plain(PyObject* o, const at::Tensor& x) {
    return THPVariable_CheckExact(o) && !at::isTensorSubclassLike(x) && x.unsafeGetTensorImpl()->has_storage() && !x._is_zerotensor() &&
           !x.is_conj() && !x.is_neg() && !(c10::GradMode::is_enabled() && x.requires_grad()) && !x._fw_grad(0).defined() &&
           !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::Tracer);
}

// Tokens between (sequence, head) units of x[B,H,T,128] when it is dense or a token slice of a dense
// [B,H,capacity,128] buffer, else -1 (same rule as `token_stride_of` of the Python module).
int64_t token_stride_of(const at::Tensor& x) {
    const int64_t b = x.size(0), h = x.size(1), t = x.size(2);
    if (x.size(3) != 128 || x.stride(3) != 1 || (t > 1 && x.stride(2) != 128)) return -1;
    int64_t step;
    if (h > 1)
        step = x.stride(1);
    else if (b > 1)
        step = x.stride(0);
    else
        return t;
    if (step % 128 || step / 128 < t || (h > 1 && b > 1 && x.stride(0) != h * step)) return -1;
    return step / 128;
}

// One side of a compressed cache as the kernels take it: (centroids [U,C,128], ids [U,T], payload [U,T,w],
// metadata [U,T,m] or None, scale [U,T] or None).
struct Side {
    at::Tensor centroids, ids, payload, meta, scale;
    explicit Side(PyObject* native)
        : centroids(tensor(item(native, 0), "centroids")), ids(tensor(item(native, 1), "ids")),
          payload(tensor(item(native, 2), "payload")), meta(optional_tensor(item(native, 3), "metadata")),
          scale(optional_tensor(item(native, 4), "scale")) {}
    Side(PyObject* c, PyObject* i, PyObject* p, PyObject* m, PyObject* s)
        : centroids(tensor(c, "centroids")), ids(tensor(i, "ids")), payload(tensor(p, "payload")),
          meta(optional_tensor(m, "metadata")), scale(optional_tensor(s, "scale")) {}
};

int64_t rows_stride(const at::Tensor& rows) {  // tokens between units
    const int64_t width = rows.dim() == 3 ? rows.size(2) : 1;
    return rows.size(0) == 1 ? rows.size(1) : rows.stride(0) / width;
}

struct Decode {
    int layout, bits, nnz;
    const Side *k, *v;
    int64_t kv_heads, q_heads, start, position;
    double theta, scaling;
    int64_t splits;
    at::Tensor inv_freq;  // f32 [64], contiguous, or undefined
    at::Tensor rq, rk, rv;  // dense window: rotated query, rotated keys, values; undefined for none
    bool stats;
};

struct Result {
    at::Tensor out, m, l;
};

// Outputs and scratch, then the library call; without the interpreter lock.  q: contiguous [B*NH,128].
Result run_decode(const Decode& d, const at::Tensor& q) {
    const at::AutoDispatchBelowADInplaceOrView plain;  // nothing here is differentiated
    const c10::DeviceIndex dev = q.get_device();
    for (const Side* s : {d.k, d.v})
        for (const at::Tensor* t : {&s->centroids, &s->ids, &s->payload, &s->meta, &s->scale}) same_device(dev, *t);
    for (const at::Tensor* t : {&d.inv_freq, &d.rq, &d.rk, &d.rv}) same_device(dev, *t);
    const int64_t tokens = d.k->payload.size(1), stride = rows_stride(d.k->payload);
    for (const at::Tensor* t : {&d.k->ids, &d.k->meta, &d.k->scale, &d.v->ids, &d.v->payload, &d.v->meta, &d.v->scale})
        if (t->defined() && t->numel() && rows_stride(*t) != stride) value_error("K and V cache tensors must share one token stride");
    const c10::cuda::CUDAGuard guard(dev);
    const int64_t rows = q.size(0);
    reskv_decode_args a{};
    a.layout = d.layout, a.bits = d.bits, a.nnz = d.nnz;
    a.q = data(q);
    a.k_centroids = data(d.k->centroids), a.k_ids = data(d.k->ids), a.k_payload = data(d.k->payload);
    a.k_meta = data(d.k->meta), a.k_scale = data(d.k->scale);
    a.v_centroids = data(d.v->centroids), a.v_ids = data(d.v->ids), a.v_payload = data(d.v->payload);
    a.v_meta = data(d.v->meta), a.v_scale = data(d.v->scale);
    a.batch = static_cast<int>(rows / d.q_heads), a.kv_heads = static_cast<int>(d.kv_heads), a.q_heads = static_cast<int>(d.q_heads);
    a.tokens = static_cast<int>(tokens), a.tok_stride = stride;
    a.k_clusters = static_cast<int>(d.k->centroids.size(1)), a.v_clusters = static_cast<int>(d.v->centroids.size(1));
    a.start_pos = static_cast<int>(d.start), a.pos_q = static_cast<int>(d.position);
    a.rope_theta = static_cast<float>(d.theta);
    a.inv_freq = static_cast<const float*>(data(d.inv_freq));
    a.scaling = static_cast<float>(d.scaling);
    a.splits = static_cast<int>(d.splits);
    at::Tensor rq, rk, rv;  // keep copies alive until the launch
    if (d.rk.defined() && d.rk.size(2) > 0) {
        rq = d.rq.contiguous(), rk = d.rk, rv = d.rv;
        // window views of one token stride and 16-byte alignment are read in place
        int64_t step = token_stride_of(rk);
        if (step < 0 || step != token_stride_of(rv) || !aligned16(rk.const_data_ptr()) || !aligned16(rv.const_data_ptr())) {
            rk = rk.contiguous(), rv = rv.contiguous();
            step = rk.size(2);
        }
        a.recent_q = data(rq), a.recent_k = data(rk), a.recent_v = data(rv);
        a.recent_tokens = static_cast<int>(rk.size(2)), a.recent_tok_stride = step;
    }
    a.device_memory = 1;
    Result r;
    // straight from the caching allocator (no dispatcher): ~1 us of host time per call
    const auto empty = [&](at::IntArrayRef size, at::ScalarType type) {
        return at::detail::empty_cuda(size, type, q.device(), std::nullopt);
    };
    r.out = empty({rows, 128}, at::kHalf);
    if (d.stats) r.m = empty({rows}, at::kFloat), r.l = empty({rows}, at::kFloat);
    const size_t need = reskv_decode_args_workspace_bytes(&a);
    const at::Tensor ws = empty({static_cast<int64_t>(need < 256 ? 256 : need)}, at::kByte);
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev).stream();
    if (g_check_status) cudaMemsetAsync(ws.data_ptr(), 0, 256, stream);
    a.workspace = ws.data_ptr(), a.workspace_bytes = static_cast<size_t>(ws.numel());
    a.out = r.out.data_ptr();
    a.out_m = d.stats ? static_cast<float*>(r.m.data_ptr()) : nullptr;
    a.out_l = d.stats ? static_cast<float*>(r.l.data_ptr()) : nullptr;
    a.stream = stream;
    check(reskv_decode_run(&a));
    g_launches += 2;
    if (g_check_status) {
        unsigned status = 0;
        cudaMemcpyAsync(&status, ws.data_ptr(), sizeof(status), cudaMemcpyDeviceToHost, stream);
        cudaStreamSynchronize(stream);
        if (status) {
            char text[64];
            std::snprintf(text, sizeof(text), "decode: device status 0x%x (bounded wait ran out)", status);
            throw Failure{PyExc_RuntimeError, text};
        }
    }
    return r;
}

// Runs `f`, turning C++ exceptions into Python ones.
template <class F>
PyObject* guarded(F&& f) {
    try {
        return f();
    } catch (const PyError&) {
    } catch (const Failure& e) {
        PyErr_SetString(e.type, e.text.c_str());
    } catch (const c10::OutOfMemoryError& e) {
        PyObject* torch = PyImport_ImportModule("torch");
        PyObject* type = torch ? PyObject_GetAttrString(torch, "OutOfMemoryError") : nullptr;
        PyErr_SetString(type ? type : PyExc_RuntimeError, e.what_without_backtrace());
        Py_XDECREF(type);
        Py_XDECREF(torch);
    } catch (const c10::Error& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}

// undefined tensor -> None
PyObject* wrap(const at::Tensor& t) { return t.defined() ? THPVariable_Wrap(t) : Py_NewRef(Py_None); }

void expect(Py_ssize_t got, Py_ssize_t want) {
    if (got == want) return;
    PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, got);
    throw PyError{};
}

// The two integers (layout, nnz) of an operator call: the retained count of the layouts that need one follows
// from the payload width.
int retained(int layout, int bits, const at::Tensor& payload) {
    const int width = static_cast<int>(payload.size(2));
    if (layout == RESKV_LAYOUT_COMPACT) return width * 32 / bits;
    return bits == 16 ? width : 0;
}

// decode(layout, bits, q, kc, ki, kp, km, ks, vc, vi, vp, vm, vs, kh, nh, start, position, theta, scaling, splits,
//        inv_freq, stats, recent, device) -> (out, m, l) or (out,).  The operator tables' calls; `device`: theirs.
PyObject* py_decode(PyObject*, PyObject* const* o, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        expect(n, 24);
        const at::Tensor q = tensor(o[2], "q");
        same_device(static_cast<c10::DeviceIndex>(integer(o[23])), q);
        const Side k(o[3], o[4], o[5], o[6], o[7]), v(o[8], o[9], o[10], o[11], o[12]);
        Decode d{};
        d.layout = static_cast<int>(integer(o[0])), d.bits = static_cast<int>(integer(o[1])), d.nnz = retained(d.layout, d.bits, k.payload);
        d.k = &k, d.v = &v;
        d.kv_heads = integer(o[13]), d.q_heads = integer(o[14]), d.start = integer(o[15]), d.position = integer(o[16]);
        d.theta = number(o[17]), d.scaling = number(o[18]), d.splits = integer(o[19]);
        d.inv_freq = optional_tensor(o[20], "inv_freq");
        d.stats = PyObject_IsTrue(o[21]);
        if (o[22] != Py_None) {
            d.rq = tensor(item(o[22], 0), "recent query"), d.rk = tensor(item(o[22], 1), "recent keys");
            d.rv = tensor(item(o[22], 2), "recent values");
        }
        const Result r = [&] {
            const Unlocked free;
            return run_decode(d, q);
        }();
        if (!d.stats) {
            PyObject* t = PyTuple_New(1);
            PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(r.out));
            return t;
        }
        PyObject* t = PyTuple_New(3);
        PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(r.out));
        PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(r.m));
        PyTuple_SET_ITEM(t, 2, THPVariable_Wrap(r.l));
        return t;
    });
}

// attention(query, k_table [B,H,C,128], k_native, v_native, layout, bits, position, start, theta, inv_freq, scaling,
//           recent, splits) -> [B,NH,1,128].  The tensor checks of the public `attention` (reskv/_attention.py:24-57).
PyObject* py_attention(PyObject*, PyObject* const* o, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        expect(n, 13);
        if (!THPVariable_Check(o[0])) value_error("query must be FP16 CUDA [batch, query_heads, 1, 128]");
        const at::Tensor query = THPVariable_Unpack(o[0]);
        if (query.dim() != 4 || query.size(2) != 1 || query.size(3) != 128 || !query.is_cuda() || query.scalar_type() != at::kHalf)
            value_error("query must be FP16 CUDA [batch, query_heads, 1, 128]");
        const int64_t b = query.size(0), nh = query.size(1);
        const at::Tensor table = tensor(o[1], "centroids");
        const Side k(o[2]), v(o[3]);
        const int64_t kh = table.size(1);
        if (query.device() != k.payload.device() || query.device() != v.payload.device())
            value_error("query and cache must be on the same CUDA device");
        if (b != table.size(0) || k.ids.size(1) != v.ids.size(1)) value_error("query/cache batch or K/V sequence lengths differ");
        if (nh % kh || (nh / kh != 1 && nh / kh != 4 && nh / kh != 8)) value_error("supported query/kv head ratios are 1, 4, and 8");
        Decode d{};
        d.layout = static_cast<int>(integer(o[4])), d.bits = static_cast<int>(integer(o[5])), d.nnz = retained(d.layout, d.bits, k.payload);
        d.k = &k, d.v = &v, d.kv_heads = kh, d.q_heads = nh;
        d.position = integer(o[6]), d.start = integer(o[7]);
        if (d.position < d.start + k.ids.size(1) - 1) value_error("query position precedes compressed tokens");
        d.theta = number(o[8]);
        if (o[9] != Py_None) {
            d.inv_freq = tensor(o[9], "inv_freq");
            if (d.inv_freq.dim() != 1 || d.inv_freq.size(0) != 64 || d.inv_freq.device() != query.device())
                value_error("inv_freq must be [64] on the query CUDA device");
        }
        d.scaling = o[10] == Py_None ? 0.08838834764831845 : number(o[10]);  // 128 ** -0.5
        if (o[11] != Py_None) {
            const at::Tensor rk = tensor(item(o[11], 1), "recent keys");
            if (rk.dim() < 3 || rk.size(2) > 0) {
                const at::Tensor rq = tensor(item(o[11], 0), "recent query"), rv = tensor(item(o[11], 2), "recent values");
                if (rq.sizes() != query.sizes() || rk.sizes() != rv.sizes() || rk.dim() != 4 || rk.size(0) != b || rk.size(1) != kh)
                    value_error("recent Q/K/V shapes do not match the compressed cache");
                for (const at::Tensor* t : {&rq, &rk, &rv})
                    if (t->device() != query.device() || t->scalar_type() != at::kHalf)
                        value_error("recent tensors must be FP16 on the query device");
                d.rq = rq, d.rk = rk, d.rv = rv;
            }
        }
        d.splits = integer(o[12]);
        const at::Tensor out = [&] {
            const Unlocked free;
            const at::AutoDispatchBelowADInplaceOrView plain;
            if (d.inv_freq.defined() && (d.inv_freq.scalar_type() != at::kFloat || !d.inv_freq.is_contiguous()))
                d.inv_freq = d.inv_freq.to(at::kFloat).contiguous();
            // only the memory order of q matters to the kernels: [B,NH,1,128] dense is [B*NH,128] dense
            const at::Tensor q = (query.is_contiguous() ? query : query.contiguous()).view({b * nh, 128});
            return run_decode(d, q).out.view({b, nh, 1, 128});
        }();
        return THPVariable_Wrap(out);
    });
}

// window_append(keys, raw_keys, values, key, raw_key, value, live) -> (keys, values) of the live + 1 tokens: the new
// token's three rows go to slot `live` of the window buffers [B,H,capacity,128] (this library's own, dense).
PyObject* py_window_append(PyObject*, PyObject* const* o, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        expect(n, 7);
        const at::Tensor wk = tensor(o[0], "keys"), wr = tensor(o[1], "raw keys"), wv = tensor(o[2], "values");
        const int64_t b = wk.size(0), h = wk.size(1), live = integer(o[6]);
        const c10::DeviceIndex dev = wk.get_device();
        at::Tensor token[3];
        for (int i = 0; i < 3; ++i) {
            token[i] = tensor(o[3 + i], "token");
            same_device(dev, token[i]);
            if (token[i].scalar_type() != at::kHalf || token[i].numel() != b * h * 128) value_error("window_append expects FP16 rows [B,H,1,128]");
        }
        at::Tensor keys, values;
        {
            const Unlocked free;
            const at::AutoDispatchBelowADInplaceOrView plain;
            const c10::cuda::CUDAGuard guard(dev);
            for (at::Tensor& t : token)
                if (!t.is_contiguous()) t = t.contiguous();
            check(reskv_window_put(wk.data_ptr(), wr.data_ptr(), wv.data_ptr(), token[0].const_data_ptr(), token[1].const_data_ptr(),
                                   token[2].const_data_ptr(), static_cast<int>(b), static_cast<int>(h), static_cast<int>(wk.size(2)),
                                   static_cast<int>(live), c10::cuda::getCurrentCUDAStream(dev).stream()));
            ++g_launches;
            keys = wk.narrow(2, 0, live + 1), values = wv.narrow(2, 0, live + 1);
        }
        PyObject* views = PyTuple_New(2);
        PyTuple_SET_ITEM(views, 0, THPVariable_Wrap(keys));
        PyTuple_SET_ITEM(views, 1, THPVariable_Wrap(values));
        return views;
    });
}

// encode(layout, bits, nnz, x, centroids, ids32, ids8) -> (payload, metadata, scale, native): one side packed, and the
// views the decode kernels take: (centroids [U,C,128], ids [U,T], payload [U,T,w], metadata [U,T,m], scale [U,T]).
PyObject* py_encode(PyObject*, PyObject* const* o, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        expect(n, 7);
        const int layout = static_cast<int>(integer(o[0])), bits = static_cast<int>(integer(o[1])), nnz = static_cast<int>(integer(o[2]));
        const at::Tensor x = tensor(o[3], "x"), cen = tensor(o[4], "centroids"), ids = tensor(o[5], "ids"), ids8 = tensor(o[6], "ids");
        if (x.scalar_type() != at::kHalf || cen.scalar_type() != at::kHalf || ids.scalar_type() != at::kInt)
            value_error("compression ops expect FP16 x/centroids and int32 ids");
        if (x.dim() != 4 || cen.dim() != 4 || ids.dim() != 3 || x.size(3) != 128 || cen.size(3) != 128)
            value_error("compression ops expect x[B,H,T,128], centroids[B,H,C,128], ids[B,H,T]");
        const int64_t stride = token_stride_of(x);
        if (stride < 0 || !cen.is_contiguous() || !ids.is_contiguous() || !ids8.is_contiguous())
            value_error("compression ops expect contiguous tensors (x may be a token slice of a dense buffer)");
        const c10::DeviceIndex dev = x.get_device();
        for (const at::Tensor* t : {&cen, &ids, &ids8}) same_device(dev, *t);
        const int64_t b = x.size(0), h = x.size(1), t = x.size(2), c = cen.size(2);
        at::Tensor payload, meta, scale, units[5];
        {
            const Unlocked free;
            const c10::cuda::CUDAGuard guard(dev);
            const at::AutoDispatchBelowADInplaceOrView plain;
            const auto empty = [&](at::IntArrayRef size, at::ScalarType type) {
                return at::detail::empty_cuda(size, type, x.device(), std::nullopt);
            };
            const bool compact = layout == RESKV_LAYOUT_COMPACT, structured = layout == RESKV_LAYOUT_STRUCTURED;
            const int64_t width = bits == 16 ? nnz : compact ? static_cast<int64_t>(nnz) * bits / 32 : structured ? 4 : 4 * bits;
            payload = empty({b, h, t, width}, bits == 16 ? at::kHalf : at::kInt);
            if (compact || (layout == RESKV_LAYOUT_UNSTRUCTURED && bits == 16))
                meta = empty({b, h, t, 2}, at::kLong);
            else if (bits == 16 || structured)
                meta = empty({b, h, t, bits == 4 ? 2 : 4}, at::kInt);
            if (bits != 16) scale = empty({b, h, t}, at::kHalf);
            const int bi = static_cast<int>(b), hi = static_cast<int>(h), ti = static_cast<int>(t), ci = static_cast<int>(c);
            const auto* id = static_cast<const int32_t*>(ids.const_data_ptr());
            const void *xp = x.const_data_ptr(), *cp = cen.const_data_ptr();
            void *pp = payload.data_ptr(), *mp = meta.defined() ? meta.data_ptr() : nullptr, *sp = scale.defined() ? scale.data_ptr() : nullptr;
            const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev).stream();
            check(compact ? reskv_encode_compact(xp, cp, id, bi, hi, ti, stride, ci, nnz, bits, pp, mp, sp, t, stream)
                  : bits == 16 && layout == RESKV_LAYOUT_UNSTRUCTURED ? reskv_encode_bitmap_fp16(xp, cp, id, bi, hi, ti, stride, ci, nnz, pp, mp, t, stream)
                  : bits == 16 ? reskv_encode_tiled_fp16(xp, cp, id, bi, hi, ti, stride, ci, nnz, structured, pp, mp, t, stream)
                  : structured ? reskv_encode_structured_int4(xp, cp, id, bi, hi, ti, stride, ci, pp, mp, sp, t, stream)
                               : reskv_encode_quantized(xp, cp, id, bi, hi, ti, stride, ci, nnz, bits, pp, sp, t, stream));
            ++g_launches;
            const at::Tensor* parts[5] = {&cen, &ids8, &payload, &meta, &scale};
            for (int i = 0; i < 5; ++i)
                if (parts[i]->defined())
                    units[i] = parts[i]->dim() == 4 ? parts[i]->view({b * h, parts[i]->size(2), parts[i]->size(3)}) : parts[i]->view({b * h, t});
        }
        PyObject* native = PyTuple_New(5);
        for (int i = 0; i < 5; ++i) PyTuple_SET_ITEM(native, i, wrap(units[i]));
        PyObject* r = PyTuple_New(4);
        PyTuple_SET_ITEM(r, 0, wrap(payload));
        PyTuple_SET_ITEM(r, 1, wrap(meta));
        PyTuple_SET_ITEM(r, 2, wrap(scale));
        PyTuple_SET_ITEM(r, 3, native);
        return r;
    });
}

// kmeans_pair(key, value, clusters, iterations) -> for K and V (centroids [B,H,C,128], int32 ids [B,H,T], int8 ids)
PyObject* py_kmeans_pair(PyObject*, PyObject* const* o, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        expect(n, 4);
        const at::Tensor k = tensor(o[0], "key"), v = tensor(o[1], "value");
        const int64_t count = integer(o[2]), iterations = integer(o[3]);
        const c10::DeviceIndex dev = k.get_device();
        same_device(dev, v);
        if (k.scalar_type() != at::kHalf || v.scalar_type() != at::kHalf || k.dim() != 4 || k.sizes() != v.sizes() ||
            token_stride_of(k) < 0 || token_stride_of(v) < 0)
            value_error("kmeans_pair expects FP16 K and V [B,H,T,128], dense or token slices of dense buffers");
        const int64_t b = k.size(0), h = k.size(1), t = k.size(2);
        const int bi = static_cast<int>(b), hi = static_cast<int>(h), ci = static_cast<int>(count);
        if (count < 1 || count > 32 || count > t) value_error("kmeans_pair: cluster count must be in [1,32] and at most the token count");
        at::Tensor part[2][3];
        {
            const Unlocked free;
            const c10::cuda::CUDAGuard guard(dev);
            const at::AutoDispatchBelowADInplaceOrView plain;
            const auto empty = [&](at::IntArrayRef size, at::ScalarType type) {
                return at::detail::empty_cuda(size, type, k.device(), std::nullopt);
            };
            const size_t need = reskv_kmeans_workspace_bytes(2 * bi, hi, ci);
            const at::Tensor ws = empty({static_cast<int64_t>(need)}, at::kByte);
            for (auto& side : part) side[0] = empty({b, h, count, 128}, at::kHalf), side[1] = empty({b, h, t}, at::kInt), side[2] = empty({b, h, t}, at::kChar);
            check(reskv_kmeans_pair(k.const_data_ptr(), v.const_data_ptr(), bi, hi, static_cast<int>(t), token_stride_of(k), token_stride_of(v), ci,
                                    static_cast<int>(iterations), ws.data_ptr(), need, part[0][0].data_ptr(), part[1][0].data_ptr(),
                                    static_cast<int32_t*>(part[0][1].data_ptr()), static_cast<int32_t*>(part[1][1].data_ptr()),
                                    part[0][2].data_ptr(), part[1][2].data_ptr(), c10::cuda::getCurrentCUDAStream(dev).stream()));
            ++g_launches;  // all iterations
        }
        PyObject* both = PyTuple_New(2);
        for (int i = 0; i < 2; ++i) {
            PyObject* side = PyTuple_New(3);
            for (int j = 0; j < 3; ++j) PyTuple_SET_ITEM(side, j, THPVariable_Wrap(part[i][j]));
            PyTuple_SET_ITEM(both, i, side);
        }
        return both;
    });
}

// ---- a decode group behind the live tokens of a cache ------------------------------------------------------------------
// The buffers [B,H,capacity,...] of one side: ids, payload, metadata or None, scale or None.
struct Buffers {
    at::Tensor part[4];
    explicit Buffers(PyObject* tuple) {
        for (int i = 0; i < 4; ++i) part[i] = i < 2 ? tensor(item(tuple, i), "buffer") : optional_tensor(item(tuple, i), "buffer");
    }
};

// regrow(k_buffers, v_buffers, tokens, capacity) -> ((buffers, merged views) of K, the same of V): the first `tokens` tokens
// in fresh buffers of `capacity` tokens, all carved from one allocation (every buffer starts on a 256-byte boundary); the
// merged views are the buffers as [B*H, capacity, ...].
PyObject* py_regrow(PyObject*, PyObject* const* o, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        expect(n, 4);
        const Buffers sides[2] = {Buffers(o[0]), Buffers(o[1])};
        const int64_t tokens = integer(o[2]), capacity = integer(o[3]);
        const at::Tensor& first = sides[0].part[0];
        const c10::DeviceIndex dev = first.get_device();
        at::Tensor whole[2][4], merged[2][4];
        {
            const Unlocked free;
            const c10::cuda::CUDAGuard guard(dev);
            const at::AutoDispatchBelowADInplaceOrView plain;
            const int64_t units = first.size(0) * first.size(1);
            int64_t row[2][4] = {}, total = 0;  // bytes of a token
            for (int i = 0; i < 8; ++i) {
                const at::Tensor& t = sides[i / 4].part[i % 4];
                if (!t.defined()) continue;
                same_device(dev, t);
                if (!t.is_contiguous() || t.dim() < 3 || t.size(0) * t.size(1) != units || t.size(2) < tokens || capacity < tokens)
                    value_error("regrow expects dense buffers [B,H,capacity,...] that hold the tokens");
                row[i / 4][i % 4] = t.element_size() * (t.dim() == 4 ? t.size(3) : 1);
                total += (units * capacity * row[i / 4][i % 4] + 255) / 256 * 256;
            }
            const at::Tensor arena = at::detail::empty_cuda({total}, at::kByte, first.device(), std::nullopt);
            const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev).stream();
            int64_t at = 0;
            for (int side = 0; side < 2; ++side)
                for (int i = 0; i < 4; ++i) {
                    const at::Tensor& t = sides[side].part[i];
                    if (!t.defined()) continue;
                    const int64_t bytes = row[side][i], used = units * capacity * bytes;
                    const at::Tensor typed = arena.narrow(0, at, used).view(t.scalar_type());
                    const bool wide = t.dim() == 4;
                    whole[side][i] = wide ? typed.view({t.size(0), t.size(1), capacity, t.size(3)}) : typed.view({t.size(0), t.size(1), capacity});
                    merged[side][i] = wide ? typed.view({units, capacity, t.size(3)}) : typed.view({units, capacity});
                    check_cuda(cudaMemcpy2DAsync(typed.data_ptr(), capacity * bytes, t.const_data_ptr(), t.size(2) * bytes, tokens * bytes,
                                                 units, cudaMemcpyDeviceToDevice, stream),
                               "regrow");
                    at += (used + 255) / 256 * 256;
                }
        }
        PyObject* both = PyTuple_New(2);
        for (int side = 0; side < 2; ++side) {
            PyObject *grown = PyTuple_New(4), *flat = PyTuple_New(4);
            for (int i = 0; i < 4; ++i) {
                PyTuple_SET_ITEM(grown, i, wrap(whole[side][i]));
                PyTuple_SET_ITEM(flat, i, wrap(merged[side][i]));
            }
            PyTuple_SET_ITEM(both, side, PyTuple_Pack(2, grown, flat));
            Py_DECREF(grown), Py_DECREF(flat);
        }
        return both;
    });
}

// append_group(layout, bits, nnz, limit, seq_len, x_k, x_v, then for K and for V: centroids, centroids [B*H,C,128], buffers,
// merged views) -> for K and V (centroids, the views of seq_len + T tokens, the views the decode kernels take): clusters
// the group, packs it and writes it behind token seq_len of the buffers.
PyObject* py_append_group(PyObject*, PyObject* const* o, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        expect(n, 15);
        const int layout = static_cast<int>(integer(o[0])), bits = static_cast<int>(integer(o[1])), nnz = static_cast<int>(integer(o[2]));
        const int64_t limit = integer(o[3]), seq = integer(o[4]);
        at::Tensor x[2] = {tensor(o[5], "key"), tensor(o[6], "value")}, given[2], old[2], merged[2][4];
        const Buffers sides[2] = {Buffers(o[9]), Buffers(o[13])};
        for (int i = 0; i < 2; ++i) {
            given[i] = tensor(o[7 + 4 * i], "centroids"), old[i] = tensor(o[8 + 4 * i], "centroids");
            for (int k = 0; k < 4; ++k) merged[i][k] = optional_tensor(item(o[10 + 4 * i], k), "buffer");
        }
        const c10::DeviceIndex dev = x[0].get_device();
        at::Tensor next[2], views[2][4], native[2][5];
        {
            const Unlocked free;
            const c10::cuda::CUDAGuard guard(dev);
            const at::AutoDispatchBelowADInplaceOrView plain;
            if (token_stride_of(x[0]) < 0 || token_stride_of(x[0]) != token_stride_of(x[1]))
                x[0] = x[0].contiguous(), x[1] = x[1].contiguous();
            const int64_t b = x[0].size(0), h = x[0].size(1), t = x[0].size(2);
            for (int i = 0; i < 2; ++i) {
                const int64_t c = old[i].size(1);
                same_device(dev, old[i]);
                if (x[i].scalar_type() != at::kHalf || old[i].scalar_type() != at::kHalf || !old[i].is_contiguous())
                    value_error("append_group expects FP16 keys, values and dense FP16 centroids");
                if (c < limit)
                    next[i] = at::detail::empty_cuda({b, h, c + 1, 128}, at::kHalf, x[0].device(), std::nullopt);
                else
                    next[i] = given[i].is_contiguous() ? given[i] : old[i].view({b, h, c, 128});
                for (const at::Tensor& part : sides[i].part)
                    if (part.defined()) {
                        same_device(dev, part);
                        if (!part.is_contiguous()) value_error("append_group expects dense capacity buffers");
                    }
                if (sides[i].part[0].scalar_type() != at::kChar) value_error("append_group expects int8 ids");
            }
            const at::Tensor scratch = at::detail::empty_cuda({2, b * h, t}, at::kInt, x[0].device(), std::nullopt);
            const auto at_part = [&](int i, int k) { return sides[i].part[k].defined() ? sides[i].part[k].data_ptr() : nullptr; };
            check(reskv_compress_group(
                layout, bits, nnz, x[0].const_data_ptr(), x[1].const_data_ptr(), static_cast<int>(b), static_cast<int>(h), static_cast<int>(t),
                token_stride_of(x[0]), old[0].const_data_ptr(), static_cast<int>(old[0].size(1)), next[0].data_ptr(),
                static_cast<int>(next[0].size(2)), at_part(0, 0), at_part(0, 1), at_part(0, 2), at_part(0, 3), sides[0].part[0].size(2),
                old[1].const_data_ptr(), static_cast<int>(old[1].size(1)), next[1].data_ptr(), static_cast<int>(next[1].size(2)),
                at_part(1, 0), at_part(1, 1), at_part(1, 2), at_part(1, 3), sides[1].part[0].size(2), static_cast<int>(seq),
                static_cast<int32_t*>(scratch.data_ptr()), c10::cuda::getCurrentCUDAStream(dev).stream()));
            g_launches += 5;
            for (int i = 0; i < 2; ++i) {
                native[i][0] = next[i].view({b * h, next[i].size(2), 128});
                for (int k = 0; k < 4; ++k)
                    if (merged[i][k].defined())
                        views[i][k] = sides[i].part[k].narrow(2, 0, seq + t), native[i][k + 1] = merged[i][k].narrow(1, 0, seq + t);
            }
        }
        PyObject* both = PyTuple_New(2);
        for (int i = 0; i < 2; ++i) {
            PyObject *shown = PyTuple_New(4), *kernels = PyTuple_New(5), *centroids = THPVariable_Wrap(next[i]);
            for (int k = 0; k < 4; ++k) PyTuple_SET_ITEM(shown, k, wrap(views[i][k]));
            for (int k = 0; k < 5; ++k) PyTuple_SET_ITEM(kernels, k, wrap(native[i][k]));
            PyTuple_SET_ITEM(both, i, PyTuple_Pack(3, centroids, shown, kernels));
            Py_DECREF(centroids), Py_DECREF(shown), Py_DECREF(kernels);
        }
        return both;
    });
}

// window_shift(keys, raw_keys, values, dst, src, count): moves `count` tokens of the window buffers [B,H,capacity,128]
PyObject* py_window_shift(PyObject*, PyObject* const* o, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        expect(n, 6);
        const at::Tensor wk = tensor(o[0], "keys"), wr = tensor(o[1], "raw keys"), wv = tensor(o[2], "values");
        const c10::DeviceIndex dev = wk.get_device();
        const int dst = static_cast<int>(integer(o[3])), src = static_cast<int>(integer(o[4])), count = static_cast<int>(integer(o[5]));
        {
            const Unlocked free;
            const c10::cuda::CUDAGuard guard(dev);
            check(reskv_window_shift(wk.data_ptr(), wr.data_ptr(), wv.data_ptr(), static_cast<int>(wk.size(0)), static_cast<int>(wk.size(1)),
                                     static_cast<int>(wk.size(2)), dst, src, count, c10::cuda::getCurrentCUDAStream(dev).stream()));
            ++g_launches;
        }
        return Py_NewRef(Py_None);
    });
}

// window_fill(keys, raw_keys, values, key, raw_key, value, slot, first, count) -> bool: tokens [first, first + count) of a
// prompt's [B,H,T,128] tensors into the window buffers from `slot` on, in one launch; False (nothing done) for tensors that
// the kernel does not take as they are.
PyObject* py_window_fill(PyObject*, PyObject* const* o, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        expect(n, 9);
        const at::Tensor window[3] = {tensor(o[0], "keys"), tensor(o[1], "raw keys"), tensor(o[2], "values")};
        const at::Tensor src[3] = {tensor(o[3], "key"), tensor(o[4], "raw key"), tensor(o[5], "value")};
        const int64_t slot = integer(o[6]), first = integer(o[7]), count = integer(o[8]);
        for (int i = 0; i < 6; ++i)
            if (!plain(o[i], i < 3 ? window[i] : src[i - 3])) return Py_NewRef(Py_False);
        const c10::DeviceIndex dev = window[0].get_device();
        int64_t stride[3];
        for (int i = 0; i < 3; ++i) {
            const at::Tensor& x = src[i];
            if (!x.is_cuda() || x.get_device() != dev || x.scalar_type() != at::kHalf || window[i].scalar_type() != at::kHalf || x.dim() != 4 ||
                x.size(0) != window[i].size(0) || x.size(1) != window[i].size(1) || x.size(2) < first + count || !window[i].is_contiguous())
                return Py_NewRef(Py_False);
            stride[i] = token_stride_of(x);
            if (stride[i] < x.size(2) || !aligned16(x.const_data_ptr()) || !aligned16(window[i].const_data_ptr())) return Py_NewRef(Py_False);
        }
        {
            const Unlocked free;
            const c10::cuda::CUDAGuard guard(dev);
            check(reskv_window_fill(window[0].data_ptr(), window[1].data_ptr(), window[2].data_ptr(), src[0].const_data_ptr(), src[1].const_data_ptr(),
                                    src[2].const_data_ptr(), static_cast<int>(window[0].size(0)), static_cast<int>(window[0].size(1)),
                                    static_cast<int>(window[0].size(2)), static_cast<int>(slot), stride[0], stride[1], stride[2],
                                    static_cast<int>(first), static_cast<int>(count), c10::cuda::getCurrentCUDAStream(dev).stream()));
            ++g_launches;
        }
        return Py_NewRef(Py_True);
    });
}

// ---- verdicts of take_ids -------------------------------------------------------------------------------------------
// A word of mapped pinned host memory and an event per call in flight (the event is made for the call's device).  They are
// kept for later calls of any thread, about kKeptVerdicts of them.  A ticket may be dropped by a finaliser, at any time and
// inside a stream capture too, so dropping one makes no CUDA call: the slot goes back as it is, is taken again only once its
// event is over, and surplus slots are freed by the calls that take one.
struct Verdict {
    volatile uint32_t* word;
    cudaEvent_t event;
    c10::DeviceIndex device;
    std::atomic<bool> seen{false};  // the event of its last call is known to be over
};
constexpr size_t kKeptVerdicts = 16;
std::mutex g_verdict_lock;
std::vector<Verdict*> g_verdicts;

bool is_over(Verdict* v) {
    if (v->seen) return true;
    const cudaError_t e = cudaEventQuery(v->event);
    if (e != cudaSuccess) cudaGetLastError();
    return e == cudaSuccess;
}

Verdict* get_verdict(c10::DeviceIndex device) {
    Verdict* found = nullptr;
    std::vector<Verdict*> surplus;
    {
        const std::lock_guard<std::mutex> lock(g_verdict_lock);
        for (size_t i = 0; i < g_verdicts.size();) {
            Verdict* v = g_verdicts[i];
            const bool take = !found && v->device == device, free = g_verdicts.size() > kKeptVerdicts;
            if ((take || free) && is_over(v)) {
                if (take) found = v; else surplus.push_back(v);
                g_verdicts[i] = g_verdicts.back();
                g_verdicts.pop_back();
            } else {
                ++i;
            }
        }
    }
    for (Verdict* v : surplus) {
        cudaEventDestroy(v->event);
        cudaFreeHost(const_cast<uint32_t*>(v->word));
        delete v;
    }
    if (!found) {
        void* word = nullptr;
        cudaEvent_t event = nullptr;
        check_cuda(cudaHostAlloc(&word, sizeof(uint32_t), cudaHostAllocMapped | cudaHostAllocPortable), "cudaHostAlloc");
        check_cuda(cudaEventCreateWithFlags(&event, cudaEventDisableTiming), "cudaEventCreate");
        found = new Verdict{static_cast<volatile uint32_t*>(word), event, device};
    }
    found->seen = false;
    return found;
}

void put_verdict(Verdict* v) noexcept {
    try {
        const std::lock_guard<std::mutex> lock(g_verdict_lock);
        g_verdicts.push_back(v);
    } catch (...) {  // no memory for the list: the slot is lost
    }
}

void drop_ticket(PyObject* capsule) { put_verdict(static_cast<Verdict*>(PyCapsule_GetPointer(capsule, "reskv verdict"))); }

// take_ids(k_ids, v_ids, k_clusters, v_clusters) -> (int32 ids [2,...], k int8 ids, v int8 ids, ticket)
PyObject* py_take_ids(PyObject*, PyObject* const* o, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        expect(n, 4);
        at::Tensor k = tensor(o[0], "ids"), v = tensor(o[1], "ids"), wide, narrow_k, narrow_v;
        const int clusters_k = static_cast<int>(integer(o[2])), clusters_v = static_cast<int>(integer(o[3]));
        Verdict* verdict = nullptr;
        {
            const Unlocked free;
            k = k.contiguous(), v = v.contiguous();
            const c10::DeviceIndex dev = k.get_device();
            const c10::cuda::CUDAGuard guard(dev);
            const at::AutoDispatchBelowADInplaceOrView plain;
            const auto empty = [&](at::IntArrayRef size, at::ScalarType type) {
                return at::detail::empty_cuda(size, type, k.device(), std::nullopt);
            };
            std::vector<int64_t> both(k.sizes().begin(), k.sizes().end());
            both.insert(both.begin(), 2);
            wide = empty(both, at::kInt), narrow_k = empty(k.sizes(), at::kChar), narrow_v = empty(k.sizes(), at::kChar);
            const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev).stream();
            verdict = get_verdict(dev);
            *verdict->word = 0;
            void* word = nullptr;
            int rc = RESKV_OK;
            const cudaError_t mapped = cudaHostGetDevicePointer(&word, const_cast<uint32_t*>(verdict->word), 0);
            if (mapped == cudaSuccess)
                rc = reskv_take_ids(k.const_data_ptr(), v.const_data_ptr(), static_cast<int>(k.element_size()), static_cast<int>(v.element_size()),
                                    k.numel(), clusters_k, clusters_v, static_cast<int32_t*>(wide.data_ptr()), narrow_k.data_ptr(),
                                    narrow_v.data_ptr(), static_cast<uint32_t*>(word), stream);
            const cudaError_t recorded = cudaEventRecord(verdict->event, stream);
            if (recorded != cudaSuccess) cudaStreamSynchronize(stream);  // nothing else tells when the word is written
            if (mapped != cudaSuccess || rc < 0 || recorded != cudaSuccess) {
                put_verdict(verdict);
                check_cuda(mapped, "cudaHostGetDevicePointer");
                check(rc);
                check_cuda(recorded, "cudaEventRecord");
            }
            ++g_launches;
        }
        PyObject* ticket = PyCapsule_New(verdict, "reskv verdict", drop_ticket);
        if (!ticket) {
            put_verdict(verdict);
            throw PyError{};
        }
        PyObject* t = PyTuple_New(4);
        PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(wide));
        PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(narrow_k));
        PyTuple_SET_ITEM(t, 2, THPVariable_Wrap(narrow_v));
        PyTuple_SET_ITEM(t, 3, ticket);
        return t;
    });
}

// ids_in_range(ticket) -> bool; waits until the ids have been looked at
PyObject* py_ids_in_range(PyObject*, PyObject* ticket) {
    return guarded([&]() -> PyObject* {
        auto* v = static_cast<Verdict*>(PyCapsule_GetPointer(ticket, "reskv verdict"));
        if (!v) throw PyError{};
        cudaError_t e;
        Py_BEGIN_ALLOW_THREADS;
        e = cudaEventSynchronize(v->event);
        Py_END_ALLOW_THREADS;
        check_cuda(e, "cudaEventSynchronize");
        v->seen = true;
        return PyBool_FromLong(*v->word == 0);
    });
}

PyObject* py_launches(PyObject*, PyObject*) { return PyLong_FromLongLong(g_launches); }

#define FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f))
PyMethodDef g_methods[] = {
    {"decode", FAST(py_decode), METH_FASTCALL, "decode attention on given operands"},
    {"attention", FAST(py_attention), METH_FASTCALL, "decode attention on a compressed cache"},
    {"window_append", FAST(py_window_append), METH_FASTCALL, "append one token to the dense window"},
    {"encode", FAST(py_encode), METH_FASTCALL, "pack one side"},
    {"kmeans_pair", FAST(py_kmeans_pair), METH_FASTCALL, "cluster K and V in the same launch"},
    {"regrow", FAST(py_regrow), METH_FASTCALL, "larger buffers for a cache"},
    {"append_group", FAST(py_append_group), METH_FASTCALL, "cluster, pack and append one decode group"},
    {"window_fill", FAST(py_window_fill), METH_FASTCALL, "a prompt's dense tail into the window"},
    {"window_shift", FAST(py_window_shift), METH_FASTCALL, "move tokens of the dense window"},
    {"take_ids", FAST(py_take_ids), METH_FASTCALL, "check and convert given cluster ids"},
    {"ids_in_range", py_ids_in_range, METH_O, "verdict of take_ids"},
    {"launches", py_launches, METH_NOARGS, "kernels launched through this module"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, g_methods};

}  // namespace

PyMODINIT_FUNC PyInit__host() {
    const char* v = std::getenv("RESKV_CHECK_STATUS");
    g_check_status = v && std::string(v) == "1";
    return PyModule_Create(&g_module);
}
