// Host path of the torch operators: argument checks, output and scratch buffers, the current stream and the C call, in
// one native function per operator.
//
// The kernels of a small decode step take a few microseconds; with the checks, the device guard, the stream lookup and
// the foreign-function call in Python a call cost 24 us of host time (15 us for a plain scatter), which bounded every
// batch that moves less than about 150 MB.  Here the same work takes a few hundred nanoseconds on top of the launches.
//
// The module calls the C ABI of libnvllm_b200_attn.so through addresses handed over by `bind` (so that another build of
// the library can be selected at run time) and holds no device code itself.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "../../include/nvllm_b200_attn.h"

namespace {

struct Api {
    decltype(&nvllm_b200_store_kvcache) store_kvcache;
    decltype(&nvllm_b200_paged_decode_workspace_bytes) decode_workspace_bytes;
    decltype(&nvllm_b200_paged_decode) paged_decode;
    decltype(&nvllm_b200_decode_step) decode_step;
    decltype(&nvllm_b200_varlen_prefill_workspace_bytes) prefill_workspace_bytes;
    decltype(&nvllm_b200_varlen_prefill) varlen_prefill;
    decltype(&nvllm_b200_paged_prefill) paged_prefill;
    decltype(&nvllm_b200_prefill_step) prefill_step;
    decltype(&nvllm_b200_qk_norm_rope_store) qk_norm_rope_store;
    decltype(&nvllm_b200_fused_decode_step) fused_decode_step;
} api = {};
PyObject* check_fn = nullptr;  // raises NvllmError for a non-zero status, from the library's thread-local text

struct Raised {};  // a Python error is set: unwind to the entry point

[[noreturn]] void raise(PyObject* type, const std::string& text) {
    PyErr_SetString(type, text.c_str());
    throw Raised();
}

std::string shape_text(const at::Tensor& t) {
    std::string s = "(";
    for (int64_t i = 0; i < t.dim(); ++i) s += (i ? ", " : "") + std::to_string(t.size(i));
    return s + (t.dim() == 1 ? ",)" : ")");
}

const char* dtype_text(at::ScalarType t) {
    switch (t) {
        case at::kBFloat16: return "torch.bfloat16";
        case at::kFloat: return "torch.float32";
        case at::kInt: return "torch.int32";
        default: return c10::toString(t);
    }
}

const at::Tensor& tensor(PyObject* o, const char* name) {
    if (!THPVariable_Check(o)) raise(PyExc_TypeError, std::string(name) + " must be a CUDA tensor");
    return THPVariable_Unpack(o);
}

void need(const at::Tensor& t, const char* name, at::ScalarType dtype, int ndim) {
    if (!t.is_cuda()) raise(PyExc_TypeError, std::string(name) + " must be a CUDA tensor");
    if (t.scalar_type() != dtype)
        raise(PyExc_TypeError, std::string(name) + " must be " + dtype_text(dtype) + ", got " + dtype_text(t.scalar_type()));
    if (!t.is_contiguous()) raise(PyExc_ValueError, std::string(name) + " must be contiguous");
    if (ndim >= 0 && t.dim() != ndim)
        raise(PyExc_ValueError, std::string(name) + " must have " + std::to_string(ndim) + " dims, got shape " + shape_text(t));
}

const at::Tensor& need(PyObject* o, const char* name, at::ScalarType dtype, int ndim) {
    const at::Tensor& t = tensor(o, name);
    need(t, name, dtype, ndim);
    return t;
}

// dtype of a K/V source: bf16 or fp32
int source_dtype(const at::Tensor& key) {
    if (key.scalar_type() == at::kBFloat16) return NVLLM_B200_DTYPE_BF16;
    if (key.scalar_type() == at::kFloat) return NVLLM_B200_DTYPE_F32;
    raise(PyExc_TypeError, std::string("key must be bf16 or fp32, got ") + dtype_text(key.scalar_type()));
}

// A Python int -> 32 bits; a null pointer stands for an error that is set.
int narrow(PyObject* i) {
    if (!i) throw Raised();
    int overflow = 0;
    const long v = PyLong_AsLongAndOverflow(i, &overflow);
    if (v == -1 && PyErr_Occurred()) throw Raised();
    if (overflow || v > INT32_MAX || v < INT32_MIN) raise(PyExc_OverflowError, "value does not fit 32 bits");
    return (int)v;
}
struct Owned {
    PyObject* o;
    ~Owned() { Py_XDECREF(o); }
};
// A size: integers, numpy and tensor scalars, floats without a fraction.
int to_int(PyObject* o) {
    if (PyLong_Check(o)) return narrow(o);
    if (PyIndex_Check(o)) {
        const Owned i{PyNumber_Index(o)};
        if (i.o) return narrow(i.o);
        if (!PyErr_ExceptionMatches(PyExc_TypeError)) throw Raised();
        PyErr_Clear();  // a tensor of a floating type
    }
    const double d = PyFloat_AsDouble(o);
    if (d == -1.0 && PyErr_Occurred()) throw Raised();
    if (d > INT32_MAX || d < INT32_MIN) raise(PyExc_OverflowError, "value does not fit 32 bits");
    if (!(d == std::floor(d))) raise(PyExc_ValueError, "a size must be a whole number, got " + std::to_string(d));
    return (int)d;
}
// An upper bound: whatever int() takes.
int to_bound(PyObject* o) {
    if (PyLong_Check(o)) return narrow(o);
    const Owned i{PyNumber_Long(o)};
    return narrow(i.o);
}
float to_float(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw Raised();
    return (float)v;
}

// One scratch buffer per (device, stream), grown on demand: calls on one stream are ordered, so they may share it.  At
// most kMaxWorkspaces buffers are kept; the one used longest ago goes back to torch's allocator first (it was allocated
// on its own stream, so the allocator hands it out again only behind that stream's work).  A buffer that a stream capture
// has seen is never given back: the graph refers to it for as long as it may be replayed.  Used under the GIL.
struct Workspace {
    int device;
    cudaStream_t stream;
    uint64_t used;
    bool captured;
    at::Tensor buf;
};
constexpr size_t kMaxWorkspaces = 64;
std::vector<at::Tensor>& captured_buffers() {
    static auto* list = new std::vector<at::Tensor>();
    return *list;
}
std::vector<Workspace>& workspaces() {
    static auto* list = new std::vector<Workspace>();  // never destroyed: the allocator may be gone at exit
    return *list;
}
uint64_t workspace_clock = 0;

const at::Tensor& workspace(int device, cudaStream_t stream, size_t nbytes) {
    auto& list = workspaces();
    Workspace* w = nullptr;
    for (auto& e : list)
        if (e.stream == stream && e.device == device) {
            w = &e;
            break;
        }
    if (!w || (size_t)w->buf.numel() < nbytes) {
        const int64_t n = (int64_t)std::max(nbytes, (size_t)1 << 20);
        at::Tensor buf = at::empty({n}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, device));
        if (!w) {
            if (list.size() < kMaxWorkspaces) {
                list.push_back(Workspace{});
                w = &list.back();
            } else {
                w = &list[0];
                for (auto& e : list)
                    if (e.used < w->used) w = &e;
            }
        }
        if (w->captured) captured_buffers().push_back(w->buf);
        w->device = device;
        w->stream = stream;
        w->captured = false;
        w->buf = std::move(buf);
    }
    w->used = ++workspace_clock;
    if (!w->captured) {
        cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) (void)cudaGetLastError();
        w->captured = status != cudaStreamCaptureStatusNone;
    }
    return w->buf;
}

// The device guard and the stream of one call.
struct Site {
    c10::cuda::CUDAGuard guard;
    int device;
    cudaStream_t stream;
    explicit Site(const at::Tensor& t)
        : guard(t.device()), device(t.get_device()), stream(c10::cuda::getCurrentCUDAStream(t.get_device()).stream()) {}
    const at::Tensor& scratch(size_t nbytes) const { return workspace(device, stream, nbytes); }
};

template <class F>
void call(F&& f) {
    int rc;
    Py_BEGIN_ALLOW_THREADS;
    rc = f();
    Py_END_ALLOW_THREADS;
    if (rc != NVLLM_B200_OK) {
        PyObject* r = PyObject_CallFunction(check_fn, "i", rc);
        Py_XDECREF(r);
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "nvllm_b200: unknown error");
        throw Raised();
    }
}

const void* ptr(const at::Tensor& t) { return t.const_data_ptr(); }
void* mptr(const at::Tensor& t) { return t.data_ptr(); }
const int32_t* iptr(const at::Tensor& t) { return static_cast<const int32_t*>(t.const_data_ptr()); }
const float* fptr(const at::Tensor& t) { return static_cast<const float*>(t.const_data_ptr()); }

template <class F>
PyObject* entry(const char* name, Py_ssize_t got, Py_ssize_t want, F&& f) {
    HANDLE_TH_ERRORS
    if (got != want) {
        PyErr_Format(PyExc_TypeError, "%s takes %zd arguments, got %zd", name, want, got);
        return nullptr;
    }
    try {
        return f();
    } catch (const Raised&) {
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}

// out argument or a new tensor like q
at::Tensor output_like(PyObject* out, const at::Tensor& q) {
    if (out == Py_None) return at::empty_like(q);
    const at::Tensor& t = need(out, "out", at::kBFloat16, 3);
    if (t.sizes() != q.sizes()) raise(PyExc_ValueError, "out shape mismatch");
    return t;
}
// the caller's own object where it gave one
PyObject* result(PyObject* out, const at::Tensor& t) {
    if (out == Py_None) return THPVariable_Wrap(t);
    Py_INCREF(out);
    return out;
}

// ---- operators ---------------------------------------------------------------------------------------------------

struct Cache {
    int64_t slots;  // num_slots of the flattened cache
    int nb, block, kvh, d;
};
// [NB, block, KVH, D] caches that fit q [.., D]
Cache paged_cache(const at::Tensor& k_cache, const at::Tensor& v_cache, const at::Tensor& q, int block_size) {
    const int64_t nb = k_cache.size(0), blk = k_cache.size(1), kvh = k_cache.size(2), d = k_cache.size(3);
    if (v_cache.sizes() != k_cache.sizes() || d != q.size(2) || blk != block_size)
        raise(PyExc_ValueError, "cache shape " + shape_text(k_cache) + " inconsistent with q " + shape_text(q) + " / block " +
                                    std::to_string(block_size));
    return {nb * blk, (int)nb, (int)blk, (int)kvh, (int)d};
}
// caches of any leading shape that end in [kvh, d]
int64_t flat_slots(const at::Tensor& k_cache, const at::Tensor& v_cache, int64_t kvh, int64_t d) {
    const int64_t n = k_cache.dim();
    if (k_cache.sizes() != v_cache.sizes() || n < 2 || k_cache.size(n - 2) != kvh || k_cache.size(n - 1) != d)
        raise(PyExc_ValueError, "cache shape " + shape_text(k_cache) + " does not end in (" + std::to_string(kvh) + ", " +
                                    std::to_string(d) + ")");
    return kvh * d ? k_cache.numel() / (kvh * d) : 0;
}

// store_kvcache(key, value, k_cache, v_cache, slot_mapping)
PyObject* store_kvcache(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return entry("store_kvcache", n, 5, [&]() -> PyObject* {
        const at::Tensor& key = tensor(a[0], "key");
        const int src = source_dtype(key);
        need(key, "key", key.scalar_type(), 3);
        const at::Tensor& value = need(a[1], "value", key.scalar_type(), 3);
        const at::Tensor& kc = need(a[2], "k_cache", at::kBFloat16, -1);
        const at::Tensor& vc = need(a[3], "v_cache", at::kBFloat16, -1);
        const at::Tensor& slots = need(a[4], "slot_mapping", at::kInt, 1);
        const int64_t t = key.size(0), kvh = key.size(1), d = key.size(2);
        if (value.sizes() != key.sizes()) raise(PyExc_ValueError, "key and value shapes differ");
        if (slots.size(0) != t)
            raise(PyExc_ValueError, "slot_mapping has " + std::to_string(slots.size(0)) + " entries for " + std::to_string(t) +
                                        " tokens");
        const int64_t num_slots = flat_slots(kc, vc, kvh, d);
        const Site site(key);
        call([&] {
            return api.store_kvcache(ptr(key), ptr(value), mptr(kc), mptr(vc), iptr(slots), t, (int)kvh, (int)d, num_slots, src,
                                     site.stream);
        });
        Py_RETURN_NONE;
    });
}

// paged_decode(q, k_cache, v_cache, block_tables, context_lens, scale, block_size, out, scratch)
PyObject* paged_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return entry("paged_decode", n, 9, [&]() -> PyObject* {
        const at::Tensor& q = need(a[0], "q", at::kBFloat16, 3);
        const at::Tensor& kc = need(a[1], "k_cache", at::kBFloat16, 4);
        const at::Tensor& vc = need(a[2], "v_cache", at::kBFloat16, 4);
        const at::Tensor& bt = need(a[3], "block_tables", at::kInt, 2);
        const at::Tensor& cl = need(a[4], "context_lens", at::kInt, 1);
        const float scale = to_float(a[5]);
        const Cache c = paged_cache(kc, vc, q, to_int(a[6]));
        const int b = (int)q.size(0), h = (int)q.size(1), mb = (int)bt.size(1);
        if (bt.size(0) != b || cl.size(0) != b) raise(PyExc_ValueError, "block_tables / context_lens batch mismatch");
        const Site site(q);
        const at::Tensor out = output_like(a[7], q);
        const at::Tensor ws = a[8] == Py_None
                                  ? site.scratch(api.decode_workspace_bytes(b, h, c.kvh, c.d, mb, c.block))
                                  : tensor(a[8], "scratch");
        call([&] {
            return api.paged_decode(ptr(q), ptr(kc), ptr(vc), iptr(bt), iptr(cl), mptr(out), mptr(ws), ws.nbytes(), b, h, c.kvh,
                                    c.d, c.nb, c.block, mb, scale, site.stream);
        });
        return result(a[7], out);
    });
}

// decode_step(q, key, value, k_cache, v_cache, slot_mapping, block_tables, context_lens, scale, block_size, out, coerce)
// coerce: bring q to the cache's dtype and q, key, value to contiguous memory first (the attention layer's contract)
PyObject* decode_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return entry("decode_step", n, 12, [&]() -> PyObject* {
        at::Tensor q = tensor(a[0], "q"), key = tensor(a[1], "key"), value = tensor(a[2], "value");
        const at::Tensor& kc = need(a[3], "k_cache", at::kBFloat16, 4);
        const at::Tensor& vc = need(a[4], "v_cache", at::kBFloat16, 4);
        if (a[11] == Py_True) {
            if (q.scalar_type() != kc.scalar_type()) q = q.to(kc.scalar_type());
            if (!q.is_contiguous()) q = q.contiguous();
            if (!key.is_contiguous()) key = key.contiguous();
            if (!value.is_contiguous()) value = value.contiguous();
        }
        const int src = source_dtype(key);
        need(q, "q", at::kBFloat16, 3);
        need(key, "key", key.scalar_type(), 3);
        need(value, "value", key.scalar_type(), 3);
        const at::Tensor& slots = need(a[5], "slot_mapping", at::kInt, 1);
        const at::Tensor& bt = need(a[6], "block_tables", at::kInt, 2);
        const at::Tensor& cl = need(a[7], "context_lens", at::kInt, 1);
        const float scale = to_float(a[8]);
        const Cache c = paged_cache(kc, vc, q, to_int(a[9]));
        const int b = (int)q.size(0), h = (int)q.size(1), mb = (int)bt.size(1);
        if (key.size(0) != b || key.size(1) != c.kvh || key.size(2) != c.d || value.sizes() != key.sizes())
            raise(PyExc_ValueError, "key/value must be [" + std::to_string(b) + ", " + std::to_string(c.kvh) + ", " +
                                        std::to_string(c.d) + "], got " + shape_text(key) + " / " + shape_text(value));
        if (bt.size(0) != b || cl.size(0) != b || slots.size(0) != b)
            raise(PyExc_ValueError, "block_tables / context_lens / slot_mapping batch mismatch");
        const Site site(q);
        const at::Tensor out = output_like(a[10], q);
        const at::Tensor ws = site.scratch(api.decode_workspace_bytes(b, h, c.kvh, c.d, mb, c.block));
        call([&] {
            return api.decode_step(ptr(q), ptr(key), ptr(value), mptr(kc), mptr(vc), iptr(slots), iptr(bt), iptr(cl), mptr(out),
                                   mptr(ws), ws.nbytes(), b, h, c.kvh, c.d, c.nb, c.block, mb, scale, src, site.stream);
        });
        return result(a[10], out);
    });
}

// Host copy of cu_seqlens: a contiguous one-dimensional int32 buffer (the Python wrapper hands over nothing else).
struct HostLengths {
    Py_buffer view = {};
    const int32_t* data = nullptr;
    HostLengths(PyObject* o, int64_t want) {
        if (o == Py_None) return;
        int64_t count;
        if (THPVariable_Check(o)) {
            const at::Tensor& t = THPVariable_Unpack(o);
            if (t.is_cuda() || t.scalar_type() != at::kInt || !t.is_contiguous())
                raise(PyExc_TypeError, "cu_seqlens_host must be a contiguous int32 host tensor");
            data = iptr(t);
            count = t.dim() ? t.size(0) : 0;
        } else {
            if (PyObject_GetBuffer(o, &view, PyBUF_FORMAT | PyBUF_C_CONTIGUOUS) != 0) throw Raised();
            if (view.ndim != 1 || view.itemsize != 4 || !view.format || view.format[0] != 'i' || view.format[1]) {
                PyBuffer_Release(&view);
                raise(PyExc_TypeError, "cu_seqlens_host must be a contiguous int32 array");
            }
            data = static_cast<const int32_t*>(view.buf);
            count = view.shape[0];
        }
        if (count != want) {
            if (view.obj) PyBuffer_Release(&view);
            raise(PyExc_ValueError, "cu_seqlens_host length mismatch");
        }
    }
    ~HostLengths() {
        if (view.obj) PyBuffer_Release(&view);
    }
};

// Rows of out behind the last sequence belong to no sequence: they are returned as zeros (where the host knows the lengths).
void zero_uncovered(const HostLengths& host, int b, const at::Tensor& out, int64_t t) {
    if (!host.data) return;
    const int64_t covered = host.data[b];
    if (covered >= 0 && covered < t) out.narrow(0, covered, t - covered).zero_();
}

// varlen_prefill(q, k, v, cu_seqlens, max_seqlen, scale, out, cu_seqlens_host, cu_seqlens_k)
PyObject* varlen_prefill(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return entry("varlen_prefill", n, 9, [&]() -> PyObject* {
        const at::Tensor& q = need(a[0], "q", at::kBFloat16, 3);
        const at::Tensor& k = need(a[1], "k", at::kBFloat16, 3);
        const at::Tensor& v = need(a[2], "v", at::kBFloat16, 3);
        const at::Tensor& cu = need(a[3], "cu_seqlens", at::kInt, 1);
        const int max_seqlen = to_bound(a[4]);
        const float scale = to_float(a[5]);
        const at::Tensor& cu_k = a[8] == Py_None ? cu : need(a[8], "cu_seqlens_k", at::kInt, 1);
        const int64_t t = q.size(0), h = q.size(1), d = q.size(2);
        if (k.sizes() != v.sizes() || k.size(0) != t || k.size(2) != d)
            raise(PyExc_ValueError, "k/v shape " + shape_text(k) + " inconsistent with q " + shape_text(q));
        const int kvh = (int)k.size(1), b = (int)cu.size(0) - 1;
        const HostLengths host(a[7], b + 1);
        const Site site(q);
        const at::Tensor out = a[6] == Py_None ? at::empty_like(q) : tensor(a[6], "out");
        zero_uncovered(host, b, out, t);
        const at::Tensor ws = site.scratch(std::max<size_t>(api.prefill_workspace_bytes(t, b, (int)h, kvh, (int)d), 256));
        call([&] {
            return api.varlen_prefill(ptr(q), ptr(k), ptr(v), iptr(cu), iptr(cu_k), host.data, mptr(out), mptr(ws), ws.nbytes(), t,
                                      b, max_seqlen, (int)h, kvh, (int)d, scale, site.stream);
        });
        return result(a[6], out);
    });
}

// paged_prefill(q, k_cache, v_cache, block_tables, cu_seqlens_q, cu_seqlens_k, max_seqlen_q, scale, block_size, out,
//               cu_seqlens_host)
PyObject* paged_prefill(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return entry("paged_prefill", n, 11, [&]() -> PyObject* {
        const at::Tensor& q = need(a[0], "q", at::kBFloat16, 3);
        const at::Tensor& kc = need(a[1], "k_cache", at::kBFloat16, 4);
        const at::Tensor& vc = need(a[2], "v_cache", at::kBFloat16, 4);
        const at::Tensor& bt = need(a[3], "block_tables", at::kInt, 2);
        const at::Tensor& cu = need(a[4], "cu_seqlens_q", at::kInt, 1);
        const at::Tensor& cu_k = need(a[5], "cu_seqlens_k", at::kInt, 1);
        const int max_seqlen_q = to_bound(a[6]);
        const float scale = to_float(a[7]);
        const Cache c = paged_cache(kc, vc, q, to_int(a[8]));
        const int64_t t = q.size(0);
        const int h = (int)q.size(1), b = (int)cu.size(0) - 1;
        if (cu_k.size(0) != b + 1 || bt.size(0) != b) raise(PyExc_ValueError, "cu_seqlens_k / block_tables batch mismatch");
        const HostLengths host(a[10], b + 1);
        const Site site(q);
        const at::Tensor out = a[9] == Py_None ? at::empty_like(q) : tensor(a[9], "out");
        zero_uncovered(host, b, out, t);
        const at::Tensor ws = site.scratch(std::max<size_t>(api.prefill_workspace_bytes(t, b, h, c.kvh, c.d), 256));
        call([&] {
            return api.paged_prefill(ptr(q), ptr(kc), ptr(vc), iptr(cu), iptr(cu_k), iptr(bt), host.data, mptr(out), mptr(ws),
                                     ws.nbytes(), t, b, max_seqlen_q, h, c.kvh, c.d, c.nb, c.block, (int)bt.size(1), scale,
                                     site.stream);
        });
        return result(a[9], out);
    });
}

// prefill_step(q, key, value, k_cache, v_cache, slot_mapping, block_tables, cu_seqlens_q, cu_seqlens_k, max_seqlen, scale,
//              block_size, num_heads, num_kv_heads, cu_seqlens_host)
// The attention layer's prefill: q comes in the cache's dtype where the keys are read from the pages, and q, key, value are
// made contiguous.  Returns None, and does nothing, for sources or caches of another kind than bf16 [NB, block, KVH, D].
PyObject* prefill_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return entry("prefill_step", n, 15, [&]() -> PyObject* {
        at::Tensor q = tensor(a[0], "q"), key = tensor(a[1], "key"), value = tensor(a[2], "value");
        const at::Tensor &kc = tensor(a[3], "k_cache"), &vc = tensor(a[4], "v_cache");
        const bool paged = a[6] != Py_None;
        const int block_size = to_int(a[11]);
        if (key.scalar_type() != at::kBFloat16 || kc.scalar_type() != at::kBFloat16 || kc.dim() != 4 || key.dim() != 3 ||
            kc.size(1) != block_size || kc.size(2) != key.size(1) || kc.size(3) != key.size(2))
            Py_RETURN_NONE;
        if (paged && q.scalar_type() != at::kBFloat16) q = q.to(at::kBFloat16);
        if (!q.is_contiguous()) q = q.contiguous();
        if (!key.is_contiguous()) key = key.contiguous();
        if (!value.is_contiguous()) value = value.contiguous();
        need(q, "q", at::kBFloat16, 3);
        need(key, "k", at::kBFloat16, 3);
        need(value, "v", at::kBFloat16, 3);
        need(kc, "k_cache", at::kBFloat16, 4);
        need(vc, "v_cache", at::kBFloat16, 4);
        const at::Tensor& slots = need(a[5], "slot_mapping", at::kInt, 1);
        const at::Tensor& cu = need(a[7], "cu_seqlens_q", at::kInt, 1);
        const at::Tensor& cu_k = need(a[8], "cu_seqlens_k", at::kInt, 1);
        const int max_seqlen = to_bound(a[9]);
        const float scale = to_float(a[10]);
        const Cache c = paged_cache(kc, vc, q, block_size);
        const int64_t t = q.size(0);
        const int h = (int)q.size(1), b = (int)cu.size(0) - 1;
        if (value.sizes() != key.sizes() || key.size(0) != t)
            raise(PyExc_ValueError, "k/v shape " + shape_text(key) + " inconsistent with q " + shape_text(q));
        if ((!paged && h != to_int(a[12])) || c.kvh != to_int(a[13])) raise(PyExc_ValueError, "head counts do not match the tensors");
        if (slots.size(0) != t)
            raise(PyExc_ValueError, "slot_mapping has " + std::to_string(slots.size(0)) + " entries for " + std::to_string(t) +
                                        " tokens");
        const int32_t* tables = nullptr;
        int mb = 0;
        if (paged) {
            const at::Tensor& bt = need(a[6], "block_tables", at::kInt, 2);
            if (bt.size(0) != b) raise(PyExc_ValueError, "cu_seqlens_k / block_tables batch mismatch");
            tables = iptr(bt);
            mb = (int)bt.size(1);
        }
        if (cu_k.size(0) != b + 1) raise(PyExc_ValueError, "cu_seqlens_k / cu_seqlens_q batch mismatch");
        const HostLengths host(a[14], b + 1);
        const Site site(q);
        const at::Tensor out = at::empty_like(q);
        zero_uncovered(host, b, out, t);
        const at::Tensor ws = site.scratch(std::max<size_t>(api.prefill_workspace_bytes(t, b, h, c.kvh, c.d), 256));
        call([&] {
            return api.prefill_step(ptr(q), ptr(key), ptr(value), mptr(kc), mptr(vc), iptr(slots), iptr(cu), iptr(cu_k), tables,
                                    host.data, mptr(out), mptr(ws), ws.nbytes(), t, b, max_seqlen, h, c.kvh, c.d, c.nb, c.block,
                                    mb, scale, site.stream);
        });
        return THPVariable_Wrap(out);
    });
}

struct PreAttention {
    const at::Tensor &q, &key, &value, &q_weight, &k_weight, &cos_sin, &positions, &slots;
    int64_t t, h, kvh, d;
};
// q, key, value, q_weight, k_weight, cos_sin_cache, positions at a[0..6]; slot_mapping apart
PreAttention pre_attention(PyObject* const* a, PyObject* slot_mapping) {
    PreAttention p{need(a[0], "q", at::kBFloat16, 3),        need(a[1], "key", at::kBFloat16, 3),
                   need(a[2], "value", at::kBFloat16, 3),    need(a[3], "q_weight", at::kFloat, 1),
                   need(a[4], "k_weight", at::kFloat, 1),    need(a[5], "cos_sin_cache", at::kFloat, 2),
                   need(a[6], "positions", at::kInt, 1),     need(slot_mapping, "slot_mapping", at::kInt, 1),
                   0, 0, 0, 0};
    p.t = p.q.size(0), p.h = p.q.size(1), p.kvh = p.key.size(1), p.d = p.q.size(2);
    if (p.key.sizes() != p.value.sizes() || p.key.size(0) != p.t || p.key.size(2) != p.d)
        raise(PyExc_ValueError, "key/value shape " + shape_text(p.key) + " inconsistent with q " + shape_text(p.q));
    if (p.q_weight.size(0) != p.d || p.k_weight.size(0) != p.d || p.cos_sin.size(1) != p.d)
        raise(PyExc_ValueError, "q_weight / k_weight / cos_sin_cache must have head_dim entries per row");
    if (p.positions.size(0) != p.t || p.slots.size(0) != p.t)
        raise(PyExc_ValueError, "positions / slot_mapping must have one entry per token");
    return p;
}

// qk_norm_rope_store(q, key, value, q_weight, k_weight, cos_sin_cache, positions, k_cache, v_cache, slot_mapping, eps)
PyObject* qk_norm_rope_store(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return entry("qk_norm_rope_store", n, 11, [&]() -> PyObject* {
        const PreAttention p = pre_attention(a, a[9]);
        const at::Tensor& kc = need(a[7], "k_cache", at::kBFloat16, -1);
        const at::Tensor& vc = need(a[8], "v_cache", at::kBFloat16, -1);
        const int64_t num_slots = flat_slots(kc, vc, p.kvh, p.d);
        const float eps = to_float(a[10]);
        const Site site(p.q);
        call([&] {
            return api.qk_norm_rope_store(mptr(p.q), mptr(p.key), ptr(p.value), fptr(p.q_weight), fptr(p.k_weight),
                                          fptr(p.cos_sin), iptr(p.positions), mptr(kc), mptr(vc), iptr(p.slots), p.t, (int)p.h,
                                          (int)p.kvh, (int)p.d, num_slots, p.cos_sin.size(0), eps, site.stream);
        });
        Py_RETURN_NONE;
    });
}

// fused_decode_step(q, key, value, q_weight, k_weight, cos_sin_cache, positions, k_cache, v_cache, slot_mapping,
//                   block_tables, context_lens, scale, block_size, eps, out)
PyObject* fused_decode_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return entry("fused_decode_step", n, 16, [&]() -> PyObject* {
        const PreAttention p = pre_attention(a, a[9]);
        const at::Tensor& kc = need(a[7], "k_cache", at::kBFloat16, 4);
        const at::Tensor& vc = need(a[8], "v_cache", at::kBFloat16, 4);
        const at::Tensor& bt = need(a[10], "block_tables", at::kInt, 2);
        const at::Tensor& cl = need(a[11], "context_lens", at::kInt, 1);
        const float scale = to_float(a[12]);
        const int block_size = to_int(a[13]);
        const float eps = to_float(a[14]);
        if (vc.sizes() != kc.sizes() || kc.size(2) != p.kvh || kc.size(3) != p.d || kc.size(1) != block_size)
            raise(PyExc_ValueError, "cache shape " + shape_text(kc) + " inconsistent with key " + shape_text(p.key) +
                                        " / block " + std::to_string(block_size));
        const int b = (int)p.t, h = (int)p.h, kvh = (int)p.kvh, d = (int)p.d, mb = (int)bt.size(1);
        if (bt.size(0) != b || cl.size(0) != b) raise(PyExc_ValueError, "block_tables / context_lens batch mismatch");
        const Site site(p.q);
        const at::Tensor out = a[15] == Py_None ? at::empty_like(p.q) : tensor(a[15], "out");
        const at::Tensor ws = site.scratch(api.decode_workspace_bytes(b, h, kvh, d, mb, block_size));
        call([&] {
            return api.fused_decode_step(mptr(p.q), mptr(p.key), ptr(p.value), fptr(p.q_weight), fptr(p.k_weight),
                                         fptr(p.cos_sin), iptr(p.positions), p.cos_sin.size(0), eps, mptr(kc), mptr(vc),
                                         iptr(p.slots), iptr(bt), iptr(cl), mptr(out), mptr(ws), ws.nbytes(), b, h, kvh, d,
                                         (int)kc.size(0), block_size, mb, scale, site.stream);
        });
        return result(a[15], out);
    });
}

// workspace(device_index, nbytes): the scratch buffer of the device's current stream
PyObject* py_workspace(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return entry("workspace", n, 2, [&]() -> PyObject* {
        const int device = to_int(a[0]);
        const long long nbytes = PyLong_AsLongLong(a[1]);
        if (nbytes < 0) {
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "negative size");
            throw Raised();
        }
        return THPVariable_Wrap(
            workspace(device, c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream(), (size_t)nbytes));
    });
}

// ---- fixed-shape decode metadata -------------------------------------------------------------------------------------

int32_t as_i32(PyObject* o) {
    int overflow = 0;
    long v = PyLong_CheckExact(o) ? PyLong_AsLongAndOverflow(o, &overflow) : -1;
    if (!PyLong_CheckExact(o)) {
        PyObject* i = PyNumber_Long(o);  // numpy and tensor scalars
        if (!i) throw Raised();
        v = PyLong_AsLongAndOverflow(i, &overflow);
        Py_DECREF(i);
    }
    if (overflow || v > INT32_MAX || v < INT32_MIN) raise(PyExc_OverflowError, "value does not fit 32 bits");
    return (int32_t)v;
}

// A list or tuple of integers -> n int32 values at dst.
void fill_list(PyObject* seq, int64_t n, int32_t* dst) {
    PyObject** items = PySequence_Fast_ITEMS(seq);
    for (int64_t i = 0; i < n; ++i) dst[i] = as_i32(items[i]);
}

// fill_decode_metadata(...) with
//   a[0..3]  lists / tuples of n integers, a[4] a list / tuple of n lists / tuples (the caller has checked the lengths)
//   a[5..9]  addresses of the host arrays ids, positions, slots, lens (int32 [rows]) and tables (int32 [rows, width])
//   a[10]    width of the tables, a[11] rows to pad up to
// Rows n .. rows-1 become padding: id 0, position 0, slot -1, length 0, every page -1.
PyObject* fill_decode_metadata(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
    return entry("fill_decode_metadata", n_args, 12, [&]() -> PyObject* {
        const int64_t n = PySequence_Fast_GET_SIZE(a[0]), width = PyLong_AsLongLong(a[10]), rows = PyLong_AsLongLong(a[11]);
        int32_t* dst[5];
        for (int i = 0; i < 5; ++i) dst[i] = static_cast<int32_t*>(PyLong_AsVoidPtr(a[5 + i]));
        if (PyErr_Occurred()) throw Raised();
        const int32_t pad[4] = {0, 0, -1, 0};
        for (int i = 0; i < 4; ++i) {
            fill_list(a[i], n, dst[i]);
            std::fill(dst[i] + n, dst[i] + rows, pad[i]);
        }
        PyObject** tables = PySequence_Fast_ITEMS(a[4]);
        for (int64_t i = 0; i < n; ++i) {
            int32_t* row = dst[4] + i * width;
            const int64_t len = PySequence_Fast_GET_SIZE(tables[i]);
            fill_list(tables[i], len, row);
            std::fill(row + len, row + width, -1);
        }
        std::fill(dst[4] + n * width, dst[4] + rows * width, -1);
        Py_RETURN_NONE;
    });
}

// bind({name: address}, check): the entry points of the shared library and the function that raises its errors
PyObject* bind(PyObject*, PyObject* args) {
    PyObject *table, *check;
    if (!PyArg_ParseTuple(args, "O!O", &PyDict_Type, &table, &check)) return nullptr;
    const struct {
        const char* name;
        void** slot;
    } entries[] = {
        {"nvllm_b200_store_kvcache", (void**)&api.store_kvcache},
        {"nvllm_b200_paged_decode_workspace_bytes", (void**)&api.decode_workspace_bytes},
        {"nvllm_b200_paged_decode", (void**)&api.paged_decode},
        {"nvllm_b200_decode_step", (void**)&api.decode_step},
        {"nvllm_b200_varlen_prefill_workspace_bytes", (void**)&api.prefill_workspace_bytes},
        {"nvllm_b200_varlen_prefill", (void**)&api.varlen_prefill},
        {"nvllm_b200_paged_prefill", (void**)&api.paged_prefill},
        {"nvllm_b200_prefill_step", (void**)&api.prefill_step},
        {"nvllm_b200_qk_norm_rope_store", (void**)&api.qk_norm_rope_store},
        {"nvllm_b200_fused_decode_step", (void**)&api.fused_decode_step},
    };
    for (const auto& e : entries) {
        PyObject* addr = PyDict_GetItemString(table, e.name);
        if (!addr) return PyErr_Format(PyExc_KeyError, "%s", e.name);
        void* p = PyLong_AsVoidPtr(addr);
        if (PyErr_Occurred()) return nullptr;
        *e.slot = p;
    }
    Py_INCREF(check);
    Py_XSETREF(check_fn, check);
    Py_RETURN_NONE;
}

#define FAST(name, fn) {name, (PyCFunction)(void (*)(void))fn, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    FAST("store_kvcache", store_kvcache),
    FAST("paged_decode", paged_decode),
    FAST("decode_step", decode_step),
    FAST("varlen_prefill", varlen_prefill),
    FAST("paged_prefill", paged_prefill),
    FAST("prefill_step", prefill_step),
    FAST("qk_norm_rope_store", qk_norm_rope_store),
    FAST("fused_decode_step", fused_decode_step),
    FAST("workspace", py_workspace),
    FAST("fill_decode_metadata", fill_decode_metadata),
    {"bind", bind, METH_VARARGS, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_torch_binding", "Host path of the torch operators.", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__torch_binding() { return PyModule_Create(&module); }
