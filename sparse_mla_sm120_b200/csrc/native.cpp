// The host side of the ops as a CPython extension (module _smla_native): argument checks, output allocation, choice of the
// split and the calls into libsmla_b200.so.
//
// Why: a decode step of one request takes the GPU about 24 us, and the same host work in Python took 27 (argument
// handling, the split policy's loop, dictionary look-ups, a 21-argument foreign call); here it is a few.
// Kept between calls: the answers of the split policy (integers per call shape), the address of the device status words and
// the library's entry points; what is kept is read and written under the interpreter lock, which a launch gives up (a launch
// waits when the queue of its stream is full, and other threads drive other streams meanwhile).
#include <Python.h>
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdarg>
#include <map>
#include <tuple>
#include <vector>

#include "../../include/smla.h"

namespace {

struct Api {
    decltype(&smla_last_error) last_error;
    decltype(&smla_sched_meta) sched_meta;
    decltype(&smla_decode_splitkv) decode_splitkv;
    decltype(&smla_decode_splitkv_ext) decode_splitkv_ext;
    decltype(&smla_decode_uniform) decode_uniform;
    decltype(&smla_prefill) prefill;
    decltype(&smla_prefill_ext) prefill_ext;
    decltype(&smla_combine) combine;
    decltype(&smla_pack_kv) pack_kv;
    decltype(&smla_mqa_logits) mqa_logits;
    decltype(&smla_topk) topk;
    decltype(&smla_topk_paged) topk_paged;
    decltype(&smla_copy_batch) copy_batch;
} api;
PyObject* g_runtime = nullptr;      // module _runtime: split policy, status buffer, default numerics of MODEL1
PyObject* g_error = nullptr;        // SmlaError

struct Failure {};                  // a Python exception has been set

[[noreturn]] void fail(PyObject* type, const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    PyErr_FormatV(type, fmt, ap);
    va_end(ap);
    throw Failure();
}

// 0 -> ok; negative -> ValueError (argument error); positive -> SmlaError (CUDA error)
void check(int rc) {
    if (rc == 0) return;
    if (rc < 0) fail(PyExc_ValueError, "smla error %d: %s", rc, api.last_error());
    fail(g_error, "CUDA error %d: %s", rc, api.last_error());
}

// The result of a call into the library, made without the interpreter lock.  (Its message is the calling thread's.)
template <typename F>
void launch(F&& f) {
    int rc;
    {
        struct Unlocked {
            PyThreadState* s = PyEval_SaveThread();
            ~Unlocked() { PyEval_RestoreThread(s); }
        } unlocked;
        rc = f();
    }
    check(rc);
}

void require(bool ok) { if (!ok) fail(PyExc_AssertionError, "unsupported tensor: expected a contiguous one of the documented type"); }

// Argument i of a call; None is an undefined tensor.
struct Args {
    PyObject* const* a;
    at::Tensor tensor(int i) const {
        if (a[i] == Py_None) return at::Tensor();
        if (!THPVariable_Check(a[i])) fail(PyExc_TypeError, "argument %d must be a tensor or None", i);
        return THPVariable_Unpack(a[i]);
    }
    at::Tensor needed(int i) const {
        at::Tensor t = tensor(i);
        if (!t.defined()) fail(PyExc_TypeError, "argument %d must be a tensor", i);
        return t;
    }
    int64_t integer(int i) const {
        const long long v = PyLong_AsLongLong(a[i]);
        if (v == -1 && PyErr_Occurred()) throw Failure();
        return v;
    }
    double real(int i) const {
        const double v = PyFloat_AsDouble(a[i]);
        if (v == -1.0 && PyErr_Occurred()) throw Failure();
        return v;
    }
    bool none(int i) const { return a[i] == Py_None; }
};

void require_cuda(std::initializer_list<const at::Tensor*> ts) {
    for (const at::Tensor* t : ts)
        if (t->defined() && !t->is_cuda()) fail(PyExc_ValueError, "sparse_mla_sm120_b200 runs on CUDA tensors only (there is no CPU path)");
}

// All CUDA tensors of a call lie on one device.  (Every launch is made with that device current, by a CUDAGuard: the library
// asks for the current device's attributes, and a default stream's handle means the current device's.)
void require_one_device(const at::Tensor& first, std::initializer_list<const at::Tensor*> ts) {
    for (const at::Tensor* t : ts)
        if (t->defined() && t->is_cuda() && t->device() != first.device())
            fail(PyExc_ValueError, "tensors on different devices: %s and %s", first.device().str().c_str(), t->device().str().c_str());
}

void* ptr(const at::Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
template <typename T> T* ptr_as(const at::Tensor& t) { return static_cast<T*>(ptr(t)); }
void* stream_of(const at::Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

// Device address of the status words of a device (made once by _runtime.status_buffer, which keeps the tensor).
int32_t* status_of(const at::Tensor& t) {
    static int32_t* cache[64] = {};
    const int d = (int)t.get_device();
    if (d < 0 || d >= 64) fail(PyExc_ValueError, "device ordinal %d not supported", d);
    if (cache[d] == nullptr) {
        PyObject* r = PyObject_CallMethod(g_runtime, "status_pointer", "i", d);
        if (r == nullptr) throw Failure();
        cache[d] = reinterpret_cast<int32_t*>(PyLong_AsLongLong(r));
        Py_DECREF(r);
        if (PyErr_Occurred()) throw Failure();
    }
    return cache[d];
}

struct Cache {           // layout and page geometry of a cache tensor
    int layout;
    int64_t block, stride;
};

int layout_of(const at::Tensor& kv) {
    const auto t = kv.scalar_type();
    if (t != at::kByte && t != at::kChar && t != at::kFloat8_e4m3fn) fail(PyExc_ValueError, "kv_cache must be a byte tensor, got %s", c10::toString(t));
    const int64_t row = kv.dim() > 0 ? kv.size(-1) : 0;
    if (row == SMLA_ROW_BYTES) return SMLA_LAYOUT_V32;
    if (row == SMLA_M1_ROW_BYTES) return SMLA_LAYOUT_MODEL1;
    fail(PyExc_ValueError, "kv_cache rows must be 656 bytes (V32) or 584 bytes (MODEL1), got %lld", (long long)row);
}

// The rules of _runtime.kv_geometry.
Cache geometry(const at::Tensor& kv) {
    Cache c;
    c.layout = layout_of(kv);
    const int64_t row = kv.size(-1);
    if (kv.stride(-1) != 1) fail(PyExc_ValueError, "kv_cache rows must be contiguous");
    if (kv.dim() == 4) {
        if (kv.size(2) != 1 || kv.stride(1) != row)
            fail(PyExc_ValueError, "kv_cache must be [num_blocks, block, 1, %lld] with %lld-byte rows", (long long)row, (long long)row);
        c.block = kv.size(1); c.stride = kv.stride(0);
        return c;
    }
    if (c.layout != SMLA_LAYOUT_V32) fail(PyExc_ValueError, "a MODEL1 cache must be [num_blocks, block, 1, 584]");
    if (kv.dim() == 3) {
        if (kv.size(1) != 1 || kv.stride(0) != row) fail(PyExc_ValueError, "kv_cache must be [pool, 1, 656] with 656-byte rows");
    } else if (kv.dim() == 2) {
        if (kv.stride(0) != row) fail(PyExc_ValueError, "kv_cache must be [pool, 656] with 656-byte rows");
    } else {
        fail(PyExc_ValueError, "unsupported kv_cache rank %lld", (long long)kv.dim());
    }
    c.block = std::max<int64_t>(kv.size(0), 1);
    c.stride = c.block * row;
    return c;
}

void check_q(const at::Tensor& q) {
    if (q.dim() != 3) fail(PyExc_ValueError, "q must be [num_tokens, num_heads, d_qk], got %lld dimensions", (long long)q.dim());
    if (q.scalar_type() != at::kBFloat16) fail(PyExc_ValueError, "q must be bf16, got %s", c10::toString(q.scalar_type()));
    if (q.size(2) != SMLA_D_QK && q.size(2) != SMLA_M1_D_QK)
        fail(PyExc_ValueError, "Unsupported d_qk=%lld; expected 576 (V32) or 512 (MODEL1)", (long long)q.size(2));
    require(q.is_contiguous());
}

// The attention arguments that decode and prefill share.
struct Attn {
    at::Tensor q, kv, indices, sink, topk_length, extra_kv, extra_indices, extra_length, out;
    Cache c{}, ec{};
    int tokens = 0, heads = 0, topk = 0, extra_topk = 0, impl = 0;
    float sm_scale = 0.f;
    bool ext = false, aligned = true;

    // q, the caches and the index lists; `d_v` as the caller gave it.
    void init(int64_t d_v) {
        check_q(q);
        c.layout = layout_of(kv);
        const int want = q.size(2) == SMLA_M1_D_QK ? SMLA_LAYOUT_MODEL1 : SMLA_LAYOUT_V32;
        if (c.layout != want)
            fail(PyExc_ValueError, "q with %lld dims does not go with cache rows of %lld bytes", (long long)q.size(2), (long long)kv.size(-1));
        if (impl == SMLA_IMPL_AUTO && c.layout == SMLA_LAYOUT_MODEL1) {
            PyObject* r = PyObject_GetAttrString(g_runtime, "MODEL1_DEFAULT_IMPL");
            if (r == nullptr) throw Failure();
            impl = (int)PyLong_AsLong(r);
            Py_DECREF(r);
        }
        c = geometry(kv);
        if (d_v != SMLA_D_V) fail(PyExc_ValueError, "d_v must be 512, got %lld", (long long)d_v);
        tokens = (int)q.size(0); heads = (int)q.size(1);
        if (indices.scalar_type() != at::kInt || indices.dim() < 1) fail(PyExc_AssertionError, "indices must be int32");
        require(indices.is_contiguous());
        topk = (int)indices.size(-1);
        if (extra_topk <= 0) {
            extra_topk = 0;
            extra_kv = extra_indices = extra_length = at::Tensor();
        } else {
            if (!extra_kv.defined() || !extra_indices.defined())
                fail(PyExc_ValueError, "extra_topk=%d needs extra_k_cache and extra_indices", extra_topk);
            if (layout_of(extra_kv) != c.layout) fail(PyExc_ValueError, "the extra cache must have the layout of the main cache");
            require_cuda({&extra_kv, &extra_indices, &extra_length});
            if (extra_indices.scalar_type() != at::kInt || !extra_indices.is_contiguous() || extra_indices.numel() != (int64_t)tokens * extra_topk)
                fail(PyExc_ValueError, "extra_indices must be contiguous int32 [%d, %d]", tokens, extra_topk);
            ec = geometry(extra_kv);
        }
        require_cuda({&q, &kv, &indices});
        require_one_device(q, {&kv, &indices, &sink, &topk_length, &extra_kv, &extra_indices, &extra_length, &out});
        ext = c.layout != SMLA_LAYOUT_V32 || extra_topk > 0;
        if (ext) {
            auto al = [](const at::Tensor& t, const Cache& g) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0 && g.stride % 16 == 0; };
            aligned = al(kv, c) && (!extra_kv.defined() || al(extra_kv, ec));
        } else {
            aligned = c.stride == c.block * SMLA_ROW_BYTES && (reinterpret_cast<uintptr_t>(kv.data_ptr()) & 15u) == 0;
        }
    }
    at::Tensor output() const {
        return out.defined() ? out.view({tokens, heads, SMLA_D_V}) : at::empty({tokens, heads, SMLA_D_V}, q.options());
    }
    at::Tensor row_stats() const { return at::empty({tokens, heads}, q.options().dtype(at::kFloat)); }

    // Attention alone, every request whole.
    void run_whole(const at::Tensor& o, const at::Tensor& lse, const at::Tensor& mx) const {
        int32_t* status = status_of(q);
        launch([&] {
            if (ext)
                return api.prefill_ext(ptr(q), ptr(kv), ptr_as<int32_t>(indices), ptr(extra_kv), ptr_as<int32_t>(extra_indices), ptr(o),
                                       ptr_as<float>(lse), ptr_as<float>(mx), tokens, heads, topk, extra_topk, sm_scale, c.layout, (int)c.block,
                                       c.stride, (int)ec.block, ec.stride, ptr_as<float>(sink), ptr_as<int32_t>(topk_length),
                                       ptr_as<int32_t>(extra_length), impl, status, stream_of(q));
            return api.prefill(ptr(q), ptr(kv), ptr_as<int32_t>(indices), ptr(o), ptr_as<float>(lse), ptr_as<float>(mx), tokens, heads, topk,
                               sm_scale, (int)c.block, c.stride, ptr_as<float>(sink), ptr_as<int32_t>(topk_length), impl, status, stream_of(q));
        });
    }
};

// _runtime.split_plan's answer for a call shape: partitions, the scheduler's fixed overhead, and equal partitions per
// request (> 1: the attention kernel derives the schedule itself).  Integers only; forgotten as a whole when there are many.
struct Plan { int parts, overhead, uniform; };
Plan plan_for(const Attn& a, int blocks, bool uniform) {
    using Key = std::tuple<int, int, int, int, int, int, int, int>;
    static std::map<Key, Plan> cache;
    const Key key{(int)a.q.get_device(), a.tokens, a.heads, blocks, (int)uniform, a.c.layout, a.ext * 2 + a.aligned, a.impl};
    const auto it = cache.find(key);
    if (it != cache.end()) return it->second;
    PyObject* r = PyObject_CallMethod(g_runtime, "split_plan", "iiiiiiiii", (int)a.q.get_device(), a.tokens, a.heads, blocks, (int)uniform,
                                      a.c.layout, (int)a.ext, (int)a.aligned, a.impl);
    if (r == nullptr) throw Failure();
    Plan p{};
    const bool ok = PyArg_ParseTuple(r, "iii", &p.parts, &p.overhead, &p.uniform);
    Py_DECREF(r);
    if (!ok) throw Failure();
    if (cache.size() >= 4096) cache.clear();
    cache.emplace(key, p);
    return p;
}

PyObject* wrap2(const at::Tensor& a, const at::Tensor& b) {
    PyObject* r = PyTuple_New(2);
    PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(a));
    PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(b));
    return r;
}

// (q, kv_cache, indices, sm_scale, d_v, attn_sink, extra_k_cache, extra_indices, topk_length, extra_topk_length, extra_topk, out,
//  impl, num_sm_parts) -> (out, lse)
PyObject* decode(const Args& x) {
    Attn a;
    a.q = x.needed(0); a.kv = x.needed(1); a.indices = x.needed(2); a.sm_scale = (float)x.real(3);
    a.sink = x.tensor(5); a.extra_kv = x.tensor(6); a.extra_indices = x.tensor(7); a.topk_length = x.tensor(8);
    a.extra_length = x.tensor(9); a.extra_topk = (int)x.integer(10); a.out = x.tensor(11); a.impl = (int)x.integer(12);
    a.init(x.integer(4));
    const int blocks = std::max((a.topk + SMLA_BLOCK_N - 1) / SMLA_BLOCK_N, 1) + (a.extra_topk + SMLA_BLOCK_N - 1) / SMLA_BLOCK_N;
    Plan p{0, 5, 0};
    if (x.none(13)) p = plan_for(a, blocks, !a.topk_length.defined() && a.extra_topk == 0);
    else p.parts = (int)x.integer(13);
    const c10::cuda::CUDAGuard on(a.q.device());
    const at::Tensor o = a.output(), lse = a.row_stats();
    if (p.parts == a.tokens) {      // one partition per request: nothing to schedule or to combine
        a.run_whole(o, lse, at::Tensor());
        return wrap2(o, lse);
    }
    void* stream = stream_of(a.q);
    // equal partitions write fp16 records, one each; the scheduler's write fp32 ones at the positions it gives
    const int64_t row = (int64_t)a.heads * (p.uniform > 1 ? p.parts : (int64_t)a.tokens + p.parts);
    const int64_t o_bytes = row * SMLA_D_V * (p.uniform > 1 ? 2 : 4), l_bytes = (row * 4 + 255) & ~255ll, m_bytes = ((int64_t)p.parts * SMLA_SCHED_META_INTS * 4 + 255) & ~255ll;
    // Scratch of this call alone, from the allocator: of the current stream's memory, of the graph's own while a capture runs.
    // (Kept between calls it would be shared by a graph, which may replay on any stream, and whoever else used the stream that
    // it was captured on.)
    const at::Tensor ws = at::empty({o_bytes + l_bytes + m_bytes + ((int64_t)a.tokens + 1) * 4}, a.q.options().dtype(at::kByte));
    char* w = static_cast<char*>(ws.data_ptr());
    float* o_accum = reinterpret_cast<float*>(w);
    float* lse_accum = reinterpret_cast<float*>(w + o_bytes);
    int32_t* meta = reinterpret_cast<int32_t*>(w + o_bytes + l_bytes);
    int32_t* splits = reinterpret_cast<int32_t*>(w + o_bytes + l_bytes + m_bytes);
    int32_t* status = status_of(a.q);
    if (p.uniform > 1) {
        launch([&] {
            return api.decode_uniform(ptr(a.q), ptr(a.kv), ptr_as<int32_t>(a.indices), o_accum, lse_accum, ptr(o), ptr_as<float>(lse), a.tokens,
                                      a.heads, a.topk, a.sm_scale, (int)a.c.block, a.c.stride, p.uniform, ptr_as<float>(a.sink), a.impl,
                                      status, stream);
        });
        return wrap2(o, lse);
    }
    launch([&] {
        int rc = api.sched_meta(a.tokens, a.topk, a.extra_topk, p.parts, p.overhead, ptr_as<int32_t>(a.topk_length),
                                ptr_as<int32_t>(a.extra_length), meta, splits, stream);
        if (rc != 0) return rc;
        if (a.ext)
            rc = api.decode_splitkv_ext(ptr(a.q), ptr(a.kv), ptr_as<int32_t>(a.indices), ptr(a.extra_kv), ptr_as<int32_t>(a.extra_indices), o_accum,
                                        lse_accum, ptr(o), ptr_as<float>(lse), meta, splits, a.tokens, a.heads, a.topk, a.extra_topk, a.sm_scale,
                                        a.c.layout, (int)a.c.block, a.c.stride, (int)a.ec.block, a.ec.stride, p.parts, ptr_as<float>(a.sink),
                                        ptr_as<int32_t>(a.topk_length), ptr_as<int32_t>(a.extra_length), a.impl, status, stream);
        else
            rc = api.decode_splitkv(ptr(a.q), ptr(a.kv), ptr_as<int32_t>(a.indices), o_accum, lse_accum, ptr(o), ptr_as<float>(lse), meta, splits,
                                    a.tokens, a.heads, a.topk, a.sm_scale, (int)a.c.block, a.c.stride, p.parts, ptr_as<float>(a.sink),
                                    ptr_as<int32_t>(a.topk_length), a.impl, status, stream);
        if (rc != 0) return rc;
        return api.combine(o_accum, lse_accum, ptr(o), ptr_as<float>(lse), splits, a.tokens, a.heads, std::min(blocks, p.parts),
                           ptr_as<float>(a.sink), stream);
    });
    return wrap2(o, lse);
}

// (q, kv_cache, indices, sm_scale, d_v, attn_sink, topk_length, out, extra_k_cache, extra_indices, extra_topk, impl) -> (out, max_logits, lse)
PyObject* prefill(const Args& x) {
    Attn a;
    a.q = x.needed(0); a.kv = x.needed(1); a.indices = x.needed(2); a.sm_scale = (float)x.real(3);
    a.sink = x.tensor(5); a.topk_length = x.tensor(6); a.out = x.tensor(7); a.extra_kv = x.tensor(8); a.extra_indices = x.tensor(9);
    a.extra_topk = (int)x.integer(10); a.impl = (int)x.integer(11);
    a.init(x.integer(4));
    const c10::cuda::CUDAGuard on(a.q.device());
    const at::Tensor o = a.output(), lse = a.row_stats(), mx = a.row_stats();
    a.run_whole(o, lse, mx);
    PyObject* r = PyTuple_New(3);
    PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(o));
    PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(mx));
    PyTuple_SET_ITEM(r, 2, THPVariable_Wrap(lse));
    return r;
}

// (q, k, k_scale, weights, ks, ke, out, impl) -> logits
PyObject* mqa_logits(const Args& x) {
    const at::Tensor q = x.needed(0), k = x.needed(1), k_scale = x.needed(2), w = x.needed(3), ks = x.needed(4), ke = x.needed(5);
    at::Tensor out = x.tensor(6);
    require_cuda({&q, &k, &k_scale, &w, &ks, &ke, &out});
    if (q.scalar_type() != at::kFloat8_e4m3fn || k.scalar_type() != at::kFloat8_e4m3fn) fail(PyExc_ValueError, "q and k must be float8_e4m3fn");
    if (q.dim() != 3 || k.dim() != 2 || q.size(2) != 128 || k.size(1) != 128) fail(PyExc_ValueError, "q must be [s_q, H, 128] and k [s_k, 128]");
    require(q.is_contiguous() && k.is_contiguous() && w.is_contiguous() && k_scale.is_contiguous());
    require(ks.scalar_type() == at::kInt && ke.scalar_type() == at::kInt);
    require_one_device(q, {&k, &k_scale, &w, &ks, &ke, &out});
    const c10::cuda::CUDAGuard on(q.device());
    if (!out.defined()) out = at::empty({q.size(0), k.size(0)}, q.options().dtype(at::kFloat));
    const int impl = (int)x.integer(7);
    int32_t* status = status_of(q);
    launch([&] {
        return api.mqa_logits(ptr(q), ptr(k), ptr_as<float>(k_scale), ptr_as<float>(w), ptr_as<int32_t>(ks), ptr_as<int32_t>(ke), ptr_as<float>(out),
                              (int)q.size(0), (int)q.size(1), (int)k.size(0), out.stride(0), impl, status, stream_of(q));
    });
    return THPVariable_Wrap(out);
}

// (logits, ks, ke, k, block_table, page_size) -> indices, or physical rows where there is a block table
PyObject* topk(const Args& x) {
    const at::Tensor logits = x.needed(0), ks = x.tensor(1), ke = x.tensor(2), table = x.tensor(4);
    const int64_t k = x.integer(3);
    require_cuda({&logits, &ks, &ke, &table});
    require(logits.dim() == 2 && logits.scalar_type() == at::kFloat && logits.stride(1) == 1);
    require_one_device(logits, {&ks, &ke, &table});
    const c10::cuda::CUDAGuard on(logits.device());
    const at::Tensor out = at::empty({logits.size(0), k}, logits.options().dtype(at::kInt));
    if (table.defined()) {
        require(table.dim() == 2 && table.scalar_type() == at::kInt && (table.stride(1) == 1 || table.size(1) == 1) && table.size(0) >= logits.size(0));
        const int page = (int)x.integer(5);
        launch([&] {
            return api.topk_paged(ptr_as<float>(logits), ptr_as<int32_t>(ks), ptr_as<int32_t>(ke), ptr_as<int32_t>(out), (int)logits.size(0),
                                  (int)logits.size(1), logits.stride(0), (int)k, ptr_as<int32_t>(table),
                                  table.size(0) > 1 ? table.stride(0) : table.size(1), (int)table.size(1), page, stream_of(logits));
        });
        return THPVariable_Wrap(out);
    }
    launch([&] {
        return api.topk(ptr_as<float>(logits), ptr_as<int32_t>(ks), ptr_as<int32_t>(ke), ptr_as<int32_t>(out), (int)logits.size(0),
                        (int)logits.size(1), logits.stride(0), (int)k, stream_of(logits));
    });
    return THPVariable_Wrap(out);
}

// (kv_bf16) -> packed
PyObject* pack_kv(const Args& x) {
    const at::Tensor kv = x.needed(0);
    require_cuda({&kv});
    require(kv.scalar_type() == at::kBFloat16 && kv.dim() >= 1 && kv.size(-1) == SMLA_D_QK && kv.is_contiguous());
    const c10::cuda::CUDAGuard on(kv.device());
    auto shape = kv.sizes().vec();
    shape.back() = SMLA_ROW_BYTES;
    const at::Tensor out = at::empty(shape, kv.options().dtype(at::kByte));
    launch([&] { return api.pack_kv(ptr(kv), ptr(out), kv.numel() / SMLA_D_QK, stream_of(kv)); });
    return THPVariable_Wrap(out);
}

// (destinations, sources): sequences of tensors, each source copied into its destination as Tensor.copy_ does.  Those
// that are plain device copies (same type, shape and device, contiguous) go as one launch, unless a destination overlaps some
// source or another destination: then the order counts, and a copy onto part of itself is for Tensor.copy_ to refuse.
PyObject* copy_into(const Args& x) {
    PyObject* d = PySequence_Fast(x.a[0], "destinations must be a sequence");
    if (d == nullptr) throw Failure();
    PyObject* s = PySequence_Fast(x.a[1], "sources must be a sequence");
    if (s == nullptr) { Py_DECREF(d); throw Failure(); }
    std::vector<at::Tensor> dt, st;
    bool ok = PySequence_Fast_GET_SIZE(d) == PySequence_Fast_GET_SIZE(s);
    for (Py_ssize_t i = 0; ok && i < PySequence_Fast_GET_SIZE(d); ++i) {
        PyObject *a = PySequence_Fast_GET_ITEM(d, i), *b = PySequence_Fast_GET_ITEM(s, i);
        ok = THPVariable_Check(a) && THPVariable_Check(b);
        if (ok) { dt.push_back(THPVariable_Unpack(a)); st.push_back(THPVariable_Unpack(b)); }
    }
    Py_DECREF(d);
    Py_DECREF(s);
    if (!ok) fail(PyExc_TypeError, "expected as many source tensors as destination tensors");
    void* dst[SMLA_COPY_BATCH_MAX];
    const void* src[SMLA_COPY_BATCH_MAX];
    int64_t bytes[SMLA_COPY_BATCH_MAX];
    int n = 0;
    struct Range { uintptr_t lo, hi; };
    auto range = [](const at::Tensor& t) {      // every byte between a tensor's first and last element
        int64_t last = 0;
        for (int64_t d = 0; d < t.dim(); ++d) last += (t.size(d) - 1) * t.stride(d);
        const uintptr_t lo = t.is_cuda() && t.numel() > 0 ? reinterpret_cast<uintptr_t>(t.data_ptr()) : 0;
        return Range{lo, lo == 0 ? 0 : lo + (uintptr_t)((last + 1) * (int64_t)t.element_size())};
    };
    std::vector<Range> rd, rs;
    for (size_t i = 0; i < dt.size(); ++i) { rd.push_back(range(dt[i])); rs.push_back(range(st[i])); }
    auto meet = [](const Range& u, const Range& v) { return u.lo < v.hi && v.lo < u.hi; };
    bool apart = true;
    for (size_t i = 0; i < rd.size(); ++i)
        for (size_t j = 0; j < rd.size(); ++j) apart &= !meet(rd[i], rs[j]) && (i == j || !meet(rd[i], rd[j]));
    for (size_t i = 0; i < dt.size(); ++i) {
        const at::Tensor &a = dt[i], &b = st[i];
        if (apart && n < SMLA_COPY_BATCH_MAX && a.is_cuda() && b.is_cuda() && a.device() == b.device() && a.device() == dt[0].device() &&
            a.scalar_type() == b.scalar_type() && a.sizes() == b.sizes() && a.is_contiguous() && b.is_contiguous()) {
            dst[n] = a.data_ptr(); src[n] = b.data_ptr(); bytes[n] = (int64_t)a.nbytes();
            ++n;
        } else {
            a.copy_(b);
        }
    }
    if (n > 0) {
        const c10::cuda::CUDAGuard on(dt[0].device());
        launch([&] { return api.copy_batch(n, dst, src, bytes, stream_of(dt[0])); });
    }
    Py_RETURN_NONE;
}

// (handle of the loaded library, module _runtime, SmlaError)
PyObject* init(const Args& x) {
    void* lib = reinterpret_cast<void*>((uintptr_t)x.integer(0));
    auto get = [&](auto& fn, const char* name) {
        fn = reinterpret_cast<std::decay_t<decltype(fn)>>(dlsym(lib, name));
        if (fn == nullptr) fail(PyExc_ImportError, "%s is missing from the kernel library", name);
    };
    get(api.last_error, "smla_last_error"); get(api.sched_meta, "smla_sched_meta"); get(api.decode_splitkv, "smla_decode_splitkv");
    get(api.decode_splitkv_ext, "smla_decode_splitkv_ext"); get(api.decode_uniform, "smla_decode_uniform"); get(api.prefill, "smla_prefill");
    get(api.prefill_ext, "smla_prefill_ext"); get(api.combine, "smla_combine"); get(api.pack_kv, "smla_pack_kv");
    get(api.mqa_logits, "smla_mqa_logits"); get(api.topk, "smla_topk");
    get(api.topk_paged, "smla_topk_paged"); get(api.copy_batch, "smla_copy_batch");
    g_runtime = x.a[1]; Py_INCREF(g_runtime);
    g_error = x.a[2]; Py_INCREF(g_error);
    Py_RETURN_NONE;
}

template <PyObject* (*F)(const Args&), int N, bool NEEDS_INIT = true>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    try {
        if (n != N) fail(PyExc_TypeError, "expected %d arguments, got %zd", N, n);
        if (NEEDS_INIT && g_runtime == nullptr) fail(PyExc_ImportError, "the kernel library has not been loaded");
        return F(Args{args});
    } catch (const Failure&) {
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}

#define SMLA_FN(name, f, n, ...) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&entry<f, n, ##__VA_ARGS__>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    SMLA_FN("init", init, 3, false), SMLA_FN("decode", decode, 14), SMLA_FN("prefill", prefill, 12),
    SMLA_FN("mqa_logits", mqa_logits, 8), SMLA_FN("topk", topk, 6), SMLA_FN("pack_kv", pack_kv, 1),
    SMLA_FN("copy_into", copy_into, 2),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_smla_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__smla_native() { return PyModule_Create(&module); }
