// Native host path of the per-step entry points: reads the tensors of a call, checks everything the kernels index
// from, fills the C ABI's argument blocks and calls the library.  packkv_b200.ops keeps the public names; this module
// (packkv_b200/_host.so) is what they run.  Not looked at: the other ranks' addresses in an exchange block.
//
// Why native: a decode step on a short context is a 10-20 us launch, and the same checks written in Python
// (about 120 tensor attribute calls and 40 ctypes field stores) took 33 us per call, 15 us per encoder call.
//
// The library's functions are bound by address (bind()), so that a build chosen with PACKKV_SM100_LIB is the one used.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/empty_like.h>
#include <ATen/ops/zeros.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <exception>
#include <memory>

#include "../../include/packkv_sm100.h"

namespace {

struct Library {
    decltype(&pkv_decode_attention) attention;
    decltype(&pkv_decode_attention_append) attention_append;
    decltype(&pkv_decode_attention_exchange) attention_exchange;
    decltype(&pkv_decode_attention_split) attention_split;
    decltype(&pkv_attention_plan) attention_plan;
    decltype(&pkv_encode_tensor) encode;
    decltype(&pkv_encode_tensor_ordered) encode_ordered;
    decltype(&pkv_encode_tensor_static) encode_static;
    decltype(&pkv_value_median_order) value_order;
    decltype(&pkv_append_residual) append;
    decltype(&pkv_rope) rope;
    decltype(&pkv_widen_rows) widen;
    decltype(&pkv_decode_attention_narrow) attention_narrow;
} lib{};

// thrown once a Python exception is set
struct Raised {};

[[noreturn]] void fail(PyObject* type, const char* fmt, ...) {
    char text[400];
    va_list ap;
    va_start(ap, fmt);
    std::vsnprintf(text, sizeof text, fmt, ap);
    va_end(ap);
    PyErr_SetString(type, text);
    throw Raised{};
}

void check(bool ok, const char* what) {
    if (!ok) fail(PyExc_ValueError, "%s", what);
}

// the exceptions the reference's callers see (packkv_b200._lib.check)
void check_status(int32_t st, const char* what) {
    switch (st) {
        case PKV_OK: return;
        case PKV_ERR_UNSUPPORTED: fail(PyExc_RuntimeError, "not supported");
        case PKV_ERR_BAD_ARGUMENT: fail(PyExc_ValueError, "%s: bad argument", what);
        case PKV_ERR_TOO_LARGE:
            fail(PyExc_ValueError, "%s: the call needs more than the %u MiB built-in scratch; pass your own scratch to encode_tensor instead", what,
                 PKV_STATIC_SCRATCH_BYTES >> 20);
        default: fail(PyExc_RuntimeError, "%s: CUDA error", what);
    }
}

const at::Tensor& tensor(PyObject* o, const char* name) {
    if (!THPVariable_Check(o)) fail(PyExc_TypeError, "%s must be a tensor, not %.80s", name, Py_TYPE(o)->tp_name);
    return THPVariable_Unpack(o);
}
const at::Tensor& cuda(PyObject* o, const char* name) {
    const at::Tensor& t = tensor(o, name);
    if (!t.is_cuda()) fail(PyExc_ValueError, "expected CUDA tensors; this library has no CPU path");
    return t;
}
const at::Tensor* maybe_cuda(PyObject* o, const char* name) { return o == Py_None ? nullptr : &cuda(o, name); }

int64_t integer(PyObject* o) {
    const int64_t v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw Raised{};
    return v;
}
double number(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw Raised{};
    return v;
}
bool truth(PyObject* o) {
    const int v = PyObject_IsTrue(o);
    if (v < 0) throw Raised{};
    return v != 0;
}
int extent(int64_t v) {
    if (v < INT32_MIN || v > INT32_MAX) fail(PyExc_OverflowError, "extent %lld does not fit 32 bits", (long long)v);
    return (int)v;
}
// the device status word
uint32_t* status_word(const at::Tensor& flags) {
    check(flags.nbytes() >= 4 && reinterpret_cast<uintptr_t>(flags.data_ptr()) % 4 == 0, "flags must hold a 32-bit word (new_flags)");
    return static_cast<uint32_t*>(flags.data_ptr());
}
bool half_type(const at::Tensor& t) { return t.scalar_type() == at::kHalf || t.scalar_type() == at::kBFloat16; }
int is_bf16(const at::Tensor& t) { return t.scalar_type() == at::kBFloat16; }

// the library's launches run without the interpreter lock: one may wait for room in the stream's queue
template <typename F> int32_t unlocked(F call) {
    PyThreadState* state = PyEval_SaveThread();
    const int32_t st = call();
    PyEval_RestoreThread(state);
    return st;
}

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

at::Tensor new_flags(const at::Tensor& like) { return at::zeros({1}, like.options().dtype(at::kInt)); }

// an attribute of a Python object, held until the end of the call
struct Held {
    PyObject* o;
    Held(PyObject* from, PyObject* name) : o(PyObject_GetAttr(from, name)) {
        if (!o) throw Raised{};
    }
    explicit Held(PyObject* item) : o(item) {
        if (!o) throw Raised{};
    }
    ~Held() { Py_DECREF(o); }
    Held(const Held&) = delete;
};

// interned attribute names of packkv_b200.ops.CompressedLayer
#define LAYER_NAMES(X) \
    X(k_stream) X(k_info) X(k_scale) X(k_zero) X(v_stream) X(v_info) X(v_scale) X(v_zero) X(n_comp) X(kv_heads) X(cbk) X(cbv) X(bits_k) X(bits_v) \
        X(k_mode) X(high_precision_zero)
struct Names {
#define X(n) PyObject* n;
    LAYER_NAMES(X)
#undef X
} names{};

// ---- decode attention ---------------------------------------------------------------------------------------------------
// Host-side bounds of everything the attention kernel indexes from n_comp, kv_heads and the block sizes: a layer whose
// metadata disagrees with its arrays (a caller mistake, a truncated or corrupt blob) must raise here instead of
// reading outside the arrays on the device.
void fill_layer(PyObject* layer, const at::Tensor& q, int64_t batch, int64_t n_comp, int64_t kv_heads, pkv_attn_args& a) {
    const Held h_ks(layer, names.k_stream), h_ki(layer, names.k_info), h_ksc(layer, names.k_scale), h_kz(layer, names.k_zero);
    const Held h_vs(layer, names.v_stream), h_vi(layer, names.v_info), h_vsc(layer, names.v_scale), h_vz(layer, names.v_zero);
    const Held h_cbk(layer, names.cbk), h_cbv(layer, names.cbv), h_bk(layer, names.bits_k), h_bv(layer, names.bits_v);
    const Held h_mode(layer, names.k_mode), h_hp(layer, names.high_precision_zero);
    const at::Tensor &ks = cuda(h_ks.o, "k_stream"), &ki = cuda(h_ki.o, "k_info"), &ksc = cuda(h_ksc.o, "k_scale"), &kz = cuda(h_kz.o, "k_zero");
    const at::Tensor &vs = cuda(h_vs.o, "v_stream"), &vi = cuda(h_vi.o, "v_info"), &vsc = cuda(h_vsc.o, "v_scale"), &vz = cuda(h_vz.o, "v_zero");
    const int64_t cbk = integer(h_cbk.o), cbv = integer(h_cbv.o), mode = integer(h_mode.o);
    for (const at::Tensor* t : {&ksc, &kz, &vsc, &vz})
        check(t->scalar_type() == q.scalar_type() && t->is_contiguous(), "scale / zero tensors must be contiguous and of q's dtype");
    if ((cbk != 64 && cbk != 128) || (cbv != 64 && cbv != 128) || n_comp <= 0 || kv_heads <= 0) {
        if (cbk == 32 || cbv == 32) fail(PyExc_RuntimeError, "not supported");
        fail(PyExc_ValueError, "bad layer metadata");
    }
    const int64_t nkb = n_comp / cbk * kv_heads, nvb = n_comp / cbv * 2 * kv_heads;
    const char* const label[] = {"k_stream", "v_stream", "k_info", "v_info", "k_scale", "k_zero", "v_scale", "v_zero"};
    const at::Tensor* const all[] = {&ks, &vs, &ki, &vi, &ksc, &kz, &vsc, &vz};
    for (int i = 0; i < 8; i++)
        if (all[i]->dim() < 1 || all[i]->size(0) != batch)
            fail(PyExc_ValueError, "%s holds %lld sequences, q holds %lld", label[i], (long long)(all[i]->dim() < 1 ? 0 : all[i]->size(0)), (long long)batch);
    if (ki.dim() != 3 || ki.size(2) != 2 || ki.size(1) < nkb || !ki.is_contiguous())
        fail(PyExc_ValueError, "k_info must be a contiguous (B, >= %lld, 2) table", (long long)nkb);
    if (vi.dim() != 3 || vi.size(2) != 2 || vi.size(1) < nvb || !vi.is_contiguous())
        fail(PyExc_ValueError, "v_info must be a contiguous (B, >= %lld, 2) table", (long long)nvb);
    check(vsc.dim() == 2 && vsc.size(1) >= n_comp && vz.sizes() == vsc.sizes(), "v_scale / v_zero must be (B, >= n_comp)");
    if (mode == PKV_K_CHANNEL) {
        check(ksc.dim() == 4 && ksc.size(1) == kv_heads && ksc.size(2) >= n_comp / cbk && ksc.size(3) == 128 && kz.sizes() == ksc.sizes(),
              "channel-mode k_scale / k_zero must be (B, kv_heads, >= n_comp / cbk, 128)");
    } else {
        check(ksc.dim() == 2 && ksc.size(1) >= n_comp && kz.sizes() == ksc.sizes(), "token-mode k_scale / k_zero must be (B, >= n_comp)");
    }
    check(ks.dim() == 2 && vs.dim() == 2 && ks.stride(1) == 1 && vs.stride(1) == 1, "streams must be (B, capacity) with contiguous bytes");
    a.k_stream = static_cast<const uint8_t*>(ks.data_ptr()); a.k_seq_stride = ks.stride(0); a.k_capacity = ks.size(1) & ~int64_t(15);
    a.k_info = static_cast<const uint32_t*>(ki.data_ptr()); a.k_info_seq_stride = ki.size(1);
    a.k_scale = ksc.data_ptr(); a.k_zero = kz.data_ptr();
    a.v_stream = static_cast<const uint8_t*>(vs.data_ptr()); a.v_seq_stride = vs.stride(0); a.v_capacity = vs.size(1) & ~int64_t(15);
    a.v_info = static_cast<const uint32_t*>(vi.data_ptr()); a.v_info_seq_stride = vi.size(1);
    a.v_scale = vsc.data_ptr(); a.v_zero = vz.data_ptr();
    a.param_tokens = extent(vsc.size(1));
    a.param_blocks = mode == PKV_K_CHANNEL ? extent(ksc.size(2)) : 0;
    check(mode != PKV_K_TOKEN || ksc.size(1) == vsc.size(1), "token-mode K and V parameter arrays must have the same row length");
    a.cbk = (int)cbk; a.cbv = (int)cbv; a.bits_k = extent(integer(h_bk.o)); a.bits_v = extent(integer(h_bv.o));
    a.k_mode = extent(mode); a.high_precision_zero = truth(h_hp.o);
}

const char* const kAppendRows = "append needs k_new / v_new of shape (B, Hkv, 1, %lld) in q's dtype with contiguous channels";

void fill_append(PyObject* append, const at::Tensor& q, const at::Tensor& k_res, int64_t batch, int64_t kv_heads, int64_t n_res, int64_t dim, pkv_attn_append& ap) {
    check(PySequence_Fast_GET_SIZE(append) == 4, "append is (k_new, v_new, cos, sin)");
    PyObject** it = PySequence_Fast_ITEMS(append);
    const at::Tensor &k = cuda(it[0], "k_new"), &v = cuda(it[1], "v_new");
    const at::Tensor *cos = maybe_cuda(it[2], "cos"), *sin = maybe_cuda(it[3], "sin");
    if (!(n_res >= 1 && k.dim() == 4 && k.size(0) == batch && k.size(1) == kv_heads && k.size(2) == 1 && k.size(3) == dim && v.sizes() == k.sizes() &&
          k.stride(3) == 1 && v.stride(3) == 1 && k.scalar_type() == q.scalar_type() && v.scalar_type() == q.scalar_type()))
        fail(PyExc_ValueError, kAppendRows, (long long)dim);
    ap.new_k = k.data_ptr(); ap.new_v = v.data_ptr();
    ap.k_stride_b = k.stride(0); ap.k_stride_h = k.stride(1); ap.v_stride_b = v.stride(0); ap.v_stride_h = v.stride(1);
    if (cos) {
        if (!(sin && cos->scalar_type() == q.scalar_type() && sin->scalar_type() == q.scalar_type() && cos->dim() >= 2 && cos->size(-2) == 1 &&
              cos->size(-1) == dim && sin->sizes() == cos->sizes() && cos->is_contiguous() && sin->is_contiguous() &&
              (cos->size(0) == 1 || cos->numel() >= batch * dim)))
            fail(PyExc_ValueError, "cos / sin must be contiguous (B or 1, 1, %lld) tensors of q's dtype", (long long)dim);
        ap.cos = cos->data_ptr(); ap.sin = sin->data_ptr(); ap.cs_stride_b = cos->size(0) == 1 ? 0 : dim;
    }
    ap.res_capacity = extent(k_res.size(2));
}

// q, layer, k_res, v_res, n_res, scaling, out, flags, kv_heads, exchange (address of its block), append, scratch, plan, plan_only
// NARROW: q and the appended rows have 64 .. 120 channels; no exchange, plan or out
template <bool NARROW> PyObject* decode_attention_of(PyObject* const* p) {
    const at::Tensor& q = cuda(p[0], "q");
    const at::Tensor *k_res = maybe_cuda(p[2], "k_res"), *v_res = maybe_cuda(p[3], "v_res");
    const at::Tensor *out = maybe_cuda(p[6], "out"), *flags = maybe_cuda(p[7], "flags"), *scratch = maybe_cuda(p[11], "scratch");
    const int64_t n_res = integer(p[4]);
    if (NARROW)
        check(q.dim() == 3 && q.size(2) >= 64 && q.size(2) < 128 && q.size(2) % 8 == 0 && q.is_contiguous(), "q must be a contiguous (B, Hq, 64 .. 120) tensor");
    else
        check(q.dim() == 3 && q.size(2) == 128 && q.is_contiguous(), "q must be a contiguous (B, Hq, 128) tensor");
    check(half_type(q), "q must be fp16 or bf16");
    const int64_t batch = q.size(0), q_heads = q.size(1);
    int64_t n_comp = 0, kv_heads;
    if (p[1] != Py_None) {
        const Held h_heads(p[1], names.kv_heads), h_comp(p[1], names.n_comp);
        kv_heads = integer(h_heads.o);
        n_comp = integer(h_comp.o);
    } else if (p[8] != Py_None) {
        kv_heads = integer(p[8]);
    } else {
        check(k_res && k_res->dim() == 4, "kv_heads is needed where neither a layer nor a residual is given");
        kv_heads = k_res->size(1);
    }
    check(kv_heads > 0 && q_heads % kv_heads == 0, "q heads must be a multiple of kv heads");
    at::Tensor own_out, own_flags;
    if (!out) { own_out = NARROW ? at::empty({batch, q_heads, 128}, q.options()) : at::empty_like(q); out = &own_out; }
    if (!flags) { own_flags = new_flags(q); flags = &own_flags; }
    check(out->scalar_type() == q.scalar_type() && out->is_contiguous() && out->numel() >= q.numel(), "out must be contiguous, of q's dtype and size");
    pkv_attn_args a{};
    a.q = q.data_ptr(); a.out = out->data_ptr();
    if (n_comp > 0) fill_layer(p[1], q, batch, n_comp, kv_heads, a);
    if (n_res > 0) {
        check(k_res && v_res && k_res->dim() == 4 && v_res->dim() == 4 && k_res->scalar_type() == q.scalar_type() && v_res->scalar_type() == q.scalar_type() &&
                  k_res->stride(3) == 1 && k_res->stride(2) == 128,
              "residual tensors must be (B, Hkv, R, 128) with contiguous rows, in q's dtype");
        check(k_res->strides() == v_res->strides(), "k_res and v_res must share strides");
        for (const at::Tensor* t : {k_res, v_res})
            check(t->size(0) >= batch && t->size(1) >= kv_heads && t->size(2) >= n_res && t->size(3) == 128,
                  "residual tensors must hold n_res rows of 128 channels for every sequence and KV head");
        a.k_res = k_res->data_ptr(); a.v_res = v_res->data_ptr();
        a.res_seq_stride = k_res->stride(0); a.res_head_stride = k_res->stride(1);
    }
    a.n_res = extent(n_res); a.batch = extent(batch); a.kv_heads = extent(kv_heads); a.group = extent(q_heads / kv_heads); a.n_comp = extent(n_comp);
    a.is_bf16 = is_bf16(q);
    a.scaling = p[5] == Py_None ? (float)std::pow(NARROW ? (double)q.size(2) : 128.0, -0.5) : (float)number(p[5]);   // (a constant for 128)
    a.flags = status_word(*flags);
    pkv_attn_append ap{};
    const bool has_append = p[10] != Py_None;
    const Held append(has_append ? PySequence_Fast(p[10], "append is (k_new, v_new, cos, sin)") : Py_NewRef(Py_None));   // any iterable
    if (has_append) {
        if (n_res < 1 || !k_res) fail(PyExc_ValueError, kAppendRows, (long long)q.size(2));
        fill_append(append.o, q, *k_res, batch, kv_heads, n_res, q.size(2), ap);
    }
    const pkv_attn_exchange* xch = p[9] == Py_None ? nullptr : reinterpret_cast<const pkv_attn_exchange*>(integer(p[9]));
    const bool plan_only = truth(p[13]);
    int32_t st;
    if (NARROW) {
        if (scratch)
            check(scratch->scalar_type() == at::kByte && scratch->is_contiguous() && reinterpret_cast<uintptr_t>(scratch->data_ptr()) % 256 == 0,
                  "scratch must be a contiguous uint8 tensor aligned to 256 bytes (new_attention_scratch)");
        st = unlocked([&, on = stream()] {
            return lib.attention_narrow(&a, has_append ? &ap : nullptr, (int32_t)q.size(2), scratch ? scratch->data_ptr() : nullptr,
                                        scratch ? scratch->numel() : 0, on);
        });
    } else if (scratch || p[12] != Py_None || plan_only) {
        pkv_attn_plan plan{};
        if (p[12] != Py_None) {
            const Held seq(PySequence_Fast(p[12], "plan is (cluster, nsplit, launches[, extra])"));
            const Py_ssize_t n = PySequence_Fast_GET_SIZE(seq.o);
            check(n >= 3, "plan is (cluster, nsplit, launches[, extra])");
            PyObject** it = PySequence_Fast_ITEMS(seq.o);
            plan.cluster = extent(integer(it[0])); plan.nsplit = extent(integer(it[1])); plan.launches = extent(integer(it[2]));
            plan.extra = n > 3 ? extent(integer(it[3])) : 0;
        }
        if (scratch)
            check(scratch->scalar_type() == at::kByte && scratch->is_contiguous() && reinterpret_cast<uintptr_t>(scratch->data_ptr()) % 256 == 0,
                  "scratch must be a contiguous uint8 tensor aligned to 256 bytes (new_attention_scratch)");
        const int64_t bytes = scratch ? scratch->numel() : 0;
        if (plan_only) {
            check_status(lib.attention_plan(&a, &plan, bytes, xch != nullptr), "attention_plan");
            return Py_BuildValue("(iiii)", plan.cluster, plan.nsplit, plan.launches, plan.extra);
        }
        void *room = scratch ? scratch->data_ptr() : nullptr, *on = stream();
        st = unlocked([&] { return lib.attention_split(&a, has_append ? &ap : nullptr, xch, &plan, room, bytes, on); });
    } else if (has_append) {
        st = unlocked([&, on = stream()] { return lib.attention_append(&a, &ap, xch, on); });
    } else {
        st = unlocked([&, on = stream()] { return xch ? lib.attention_exchange(&a, xch, on) : lib.attention(&a, on); });
    }
    check_status(st, "decode_attention");
    if (p[6] != Py_None) return Py_NewRef(p[6]);
    return THPVariable_Wrap(own_out);
}

PyObject* decode_attention(PyObject* const* p) { return decode_attention_of<false>(p); }

// q, layer, k_res, v_res, n_res, scaling, flags, kv_heads, append, scratch
PyObject* decode_attention_narrow(PyObject* const* p) {
    PyObject* const all[14] = {p[0], p[1], p[2], p[3], p[4], p[5], Py_None, p[6], p[7], Py_None, p[8], p[9], Py_None, Py_False};
    return decode_attention_of<true>(all);
}

// ---- encoder ------------------------------------------------------------------------------------------------------------
void check_source(const at::Tensor& x) {
    check(x.dim() == 4 && x.size(3) == 128 && x.stride(3) == 1 && half_type(x), "x must be (B, H, S, 128) fp16/bf16 with contiguous channels");
}

// What the encoder writes behind the `first` tokens that are there: parameters, block table, streams and their lengths.
// (Blocks that do not fit a stream's capacity are skipped and flagged on the device.)
void check_tables(int64_t batch, int64_t heads, int64_t tokens, int64_t first, int64_t block, int64_t cb, int64_t mode, bool is_k, const at::Tensor& x,
                  const at::Tensor& scale, const at::Tensor& zero, const at::Tensor& strm, const at::Tensor& info, const at::Tensor& bytes) {
    if (mode != PKV_K_CHANNEL && mode != PKV_K_TOKEN) fail(PyExc_RuntimeError, "not supported");
    check(first >= 0, "first_token must not be negative");
    const char* const what = "scale / zero must be contiguous tensors of x's dtype with room for all tokens: (B, H, blocks, 128) per channel, (B, tokens) per token";
    check(scale.dim() >= (mode == PKV_K_CHANNEL ? 3 : 2), what);
    const int64_t room = scale.size(mode == PKV_K_CHANNEL ? 2 : 1), need = mode == PKV_K_CHANNEL ? first / block + tokens / block : first + tokens;
    const int64_t rows = mode == PKV_K_CHANNEL ? batch * heads : batch, width = mode == PKV_K_CHANNEL ? 128 : 1;
    for (const at::Tensor* t : {&scale, &zero})
        check(t->scalar_type() == x.scalar_type() && t->is_contiguous() && room >= need && t->numel() >= ((rows - 1) * room + need) * width, what);
    check(strm.dim() == 2 && strm.itemsize() == 1 && strm.stride(1) == 1 && strm.size(0) >= batch, "stream must be (B, capacity) with contiguous bytes");
    const int64_t entries = (first / cb + tokens / cb) * heads * (is_k ? 1 : 2);
    check(info.dim() >= 2 && info.itemsize() == 4 && info.is_contiguous() && info.numel() >= 2 * ((batch - 1) * info.size(1) + entries) &&
              (batch <= 1 || info.size(1) >= entries),
          "info must be a contiguous (B, blocks, 2) table with room for all blocks");
    check((bytes.itemsize() == 4 || (batch <= 1 && bytes.itemsize() > 4)) && bytes.is_contiguous() && bytes.numel() >= batch, "stream_bytes must hold a 32-bit count for every sequence");
}

// which ('k' or 'v'), x, block, rel, mode, bits, cb, scale, zero, stream, info, stream_bytes, flags, first_token,
// high_precision_zero, scratch (tensor or None: allocated here; False: the library's own), order, order_block
PyObject* encode_tensor(PyObject* const* p) {
    const char* which = PyUnicode_AsUTF8(p[0]);
    if (!which) throw Raised{};
    const at::Tensor& x = cuda(p[1], "x");
    const at::Tensor &scale = cuda(p[7], "scale"), &zero = cuda(p[8], "zero"), &strm = cuda(p[9], "stream"), &info = cuda(p[10], "info");
    const at::Tensor &bytes = cuda(p[11], "stream_bytes"), &flags = cuda(p[12], "flags");
    check_source(x);
    const int64_t block = integer(p[2]), mode = integer(p[4]), cb = integer(p[6]), batch = x.size(0), heads = x.size(1), tokens = x.size(2);
    check(block > 0 && cb > 0 && tokens % block == 0 && tokens % cb == 0, "Tensor shape is not divisible by block size");
    const bool is_k = which[0] == 'k';
    check_tables(batch, heads, tokens, integer(p[13]), block, cb, mode, is_k, x, scale, zero, strm, info, bytes);
    pkv_encode_args a{};
    a.x = x.data_ptr(); a.stride_b = x.stride(0); a.stride_h = x.stride(1); a.stride_s = x.stride(2);
    a.scale = scale.data_ptr(); a.zero = zero.data_ptr();
    a.param_blocks = mode == PKV_K_CHANNEL ? extent(scale.size(2)) : 0;
    a.param_tokens = mode == PKV_K_CHANNEL ? 0 : extent(scale.size(1));
    a.stream = static_cast<uint8_t*>(strm.data_ptr()); a.stream_seq_stride = strm.stride(0); a.capacity = strm.size(1);
    a.block_info = static_cast<uint32_t*>(info.data_ptr()); a.info_seq_stride = info.size(1);
    a.stream_bytes = static_cast<uint32_t*>(bytes.data_ptr());
    a.flags = status_word(flags);
    a.batch = extent(batch); a.heads = extent(heads); a.tokens = extent(tokens); a.first_token = extent(integer(p[13]));
    a.qblock = extent(block); a.cb = extent(cb); a.which = is_k ? 0 : 1;
    a.bits = extent(integer(p[5])); a.mode = extent(mode); a.high_precision_zero = truth(p[14]); a.is_bf16 = is_bf16(x); a.rel = (float)number(p[3]);
    const char* what = a.which == 0 ? "encode_tensor(k)" : "encode_tensor(v)";
    if (p[15] == Py_False) {
        check_status(unlocked([&, on = stream()] { return lib.encode_static(&a, on); }), a.which == 0 ? "encode_tensor_static(k)" : "encode_tensor_static(v)");
        Py_RETURN_NONE;
    }
    at::Tensor own;
    const at::Tensor* scratch = maybe_cuda(p[15], "scratch");
    if (!scratch) {
        own = at::empty({std::max<int64_t>(batch * tokens * heads * 128, 16)}, x.options().dtype(at::kByte));
        scratch = &own;
    }
    uint8_t* room = static_cast<uint8_t*>(scratch->data_ptr());
    if (p[16] != Py_None) {
        const at::Tensor& order = cuda(p[16], "order");
        check(order.scalar_type() == at::kByte && order.is_contiguous() && order.numel() == batch * tokens,
              "order must be a contiguous uint8 tensor with one entry per token");
        const uint8_t* rows = static_cast<const uint8_t*>(order.data_ptr());
        const int order_block = extent(integer(p[17]));
        check_status(unlocked([&, on = stream()] { return lib.encode_ordered(&a, rows, order_block, room, scratch->numel(), on); }), what);
    } else {
        check_status(unlocked([&, on = stream()] { return lib.encode(&a, room, scratch->numel(), on); }), what);
    }
    Py_RETURN_NONE;
}

// v, block, rel, flags -> order
PyObject* value_median_order(PyObject* const* p) {
    const at::Tensor& v = cuda(p[0], "v");
    const at::Tensor* flags = maybe_cuda(p[3], "flags");
    check(v.dim() == 4 && v.size(3) == 128 && v.stride(3) == 1 && half_type(v), "v must be (B, H, S, 128) fp16/bf16 with contiguous channels");
    const int64_t block = integer(p[1]);
    check(block > 0 && v.size(2) % block == 0, "Tensor shape is not divisible by block size");
    at::Tensor own;
    if (!flags) { own = new_flags(v); flags = &own; }
    at::Tensor order = at::empty({v.size(0), v.size(2) / block, block}, v.options().dtype(at::kByte));
    pkv_encode_args a{};
    a.x = v.data_ptr(); a.stride_b = v.stride(0); a.stride_h = v.stride(1); a.stride_s = v.stride(2);
    a.batch = extent(v.size(0)); a.heads = extent(v.size(1)); a.tokens = extent(v.size(2)); a.which = 1; a.mode = PKV_K_TOKEN;
    a.is_bf16 = is_bf16(v); a.rel = (float)number(p[2]);
    a.flags = status_word(*flags);
    const int rows = extent(block);
    check_status(unlocked([&, on = stream()] { return lib.value_order(&a, static_cast<uint8_t*>(order.data_ptr()), rows, on); }), "value_median_order");
    return THPVariable_Wrap(order);
}

// ---- append and rope ----------------------------------------------------------------------------------------------------
// cos / sin in x's dtype and contiguous: the tensors themselves where they already are
struct Tables {
    at::Tensor cos, sin;
    int64_t stride_b = 0;
    Tables(const at::Tensor& c, const at::Tensor& s, at::ScalarType dtype, int64_t batch, int64_t tokens, int64_t dim, const char* what)
        : cos(c.to(dtype).contiguous()), sin(s.to(dtype).contiguous()) {
        check(cos.dim() >= 2 && cos.size(-2) == tokens && cos.size(-1) == dim && sin.sizes() == cos.sizes(), what);
        stride_b = cos.size(0) == 1 ? 0 : tokens * dim;
        check(stride_b == 0 || cos.numel() >= batch * stride_b, what);
    }
};

// k_new, v_new, k_res, v_res, position, cos, sin
PyObject* append_residual(PyObject* const* p) {
    const at::Tensor &k = cuda(p[0], "k_new"), &v = cuda(p[1], "v_new"), &kr = cuda(p[2], "k_res"), &vr = cuda(p[3], "v_res");
    const at::Tensor *cos = maybe_cuda(p[5], "cos"), *sin = maybe_cuda(p[6], "sin");
    check(k.dim() == 4 && k.size(3) == 128 && v.sizes() == k.sizes() && k.stride(3) == 1 && v.stride(3) == 1,
          "k_new and v_new must be (B, H, T, 128) with contiguous channels");
    check(kr.dim() == 4 && kr.sizes() == vr.sizes() && kr.strides() == vr.strides() && kr.stride(3) == 1 && kr.stride(2) == 128 &&
              kr.size(0) >= k.size(0) && kr.size(1) >= k.size(1) && kr.size(3) == 128,
          "k_res and v_res must be (B, H, capacity, 128) with contiguous rows and equal strides");
    check(kr.scalar_type() == k.scalar_type() && v.scalar_type() == k.scalar_type() && half_type(k), "dtype mismatch");
    const int64_t T = k.size(2);
    std::unique_ptr<Tables> cs;
    if (cos) {
        check(sin != nullptr, "cos/sin must be (B or 1, T, 128)");
        cs = std::make_unique<Tables>(*cos, *sin, k.scalar_type(), k.size(0), T, 128, "cos/sin must be (B or 1, T, 128)");
    }
    const int capacity = extent(kr.size(2)), position = extent(integer(p[4])), batch = extent(k.size(0)), heads = extent(k.size(1)), tokens = extent(T);
    check_status(unlocked([&, on = stream()] {
                     return lib.append(k.data_ptr(), k.stride(0), k.stride(1), k.stride(2), v.data_ptr(), v.stride(0), v.stride(1), v.stride(2),
                                       cs ? cs->cos.data_ptr() : nullptr, cs ? cs->sin.data_ptr() : nullptr, cs ? cs->stride_b : 0, kr.data_ptr(),
                                       vr.data_ptr(), kr.stride(0), kr.stride(1), capacity, position, batch, heads, tokens, is_bf16(k), on);
                 }),
                 "append_residual");
    Py_RETURN_NONE;
}

// k (B, H, T, 64 <= D <= 128), v or None, k_out, v_out or None (B, H, capacity, 128), position, cos, sin, zero_tail
PyObject* widen_rows(PyObject* const* p) {
    const at::Tensor &k = cuda(p[0], "k"), &ko = cuda(p[2], "k_out");
    const at::Tensor *v = maybe_cuda(p[1], "v"), *vo = maybe_cuda(p[3], "v_out"), *cos = maybe_cuda(p[5], "cos"), *sin = maybe_cuda(p[6], "sin");
    check(k.dim() == 4 && k.size(3) >= 64 && k.size(3) <= 128 && k.size(3) % 8 == 0 && k.stride(3) == 1 && half_type(k),
          "k must be (B, H, T, 64..128) fp16/bf16 with contiguous channels");
    check((v == nullptr) == (vo == nullptr) && (cos == nullptr) == (sin == nullptr), "v with v_out and cos with sin");
    check(!v || (v->sizes() == k.sizes() && v->stride(3) == 1 && v->scalar_type() == k.scalar_type()), "v must have k's shape and type and contiguous channels");
    check(ko.dim() == 4 && ko.size(0) == k.size(0) && ko.size(1) == k.size(1) && ko.size(3) == 128 && ko.stride(3) == 1 && ko.stride(2) == 128 &&
              ko.scalar_type() == k.scalar_type() && (!vo || (vo->sizes() == ko.sizes() && vo->strides() == ko.strides() && vo->scalar_type() == k.scalar_type())),
          "k_out and v_out must be (B, H, capacity, 128) with contiguous rows and equal strides");
    const int64_t T = k.size(2), D = k.size(3);
    std::unique_ptr<Tables> cs;
    if (cos) cs = std::make_unique<Tables>(*cos, *sin, k.scalar_type(), k.size(0), T, D, "cos/sin must be (B or 1, T, D)");
    const int capacity = extent(ko.size(2)), position = extent(integer(p[4])), batch = extent(k.size(0)), heads = extent(k.size(1)), tokens = extent(T);
    const bool zero_tail = truth(p[7]);
    check_status(unlocked([&, on = stream()] {
                     return lib.widen(k.data_ptr(), k.stride(0), k.stride(1), k.stride(2), v ? v->data_ptr() : nullptr, v ? v->stride(0) : 0,
                                      v ? v->stride(1) : 0, v ? v->stride(2) : 0, cs ? cs->cos.data_ptr() : nullptr, cs ? cs->sin.data_ptr() : nullptr,
                                      cs ? cs->stride_b : 0, ko.data_ptr(), vo ? vo->data_ptr() : nullptr, ko.stride(0), ko.stride(1), capacity, position,
                                      batch, heads, tokens, (int)D, zero_tail, is_bf16(k), on);
                 }),
                 "widen_rows");
    Py_RETURN_NONE;
}

// k_res, k_new, v_new, cos, sin -> the current stream of k_new's device if the attention launch can take the step's rows where they are (what
// fill_append and the launch ask of them), None if they have to be converted or refused first
PyObject* waiting_step(PyObject* const* p) {
    for (int i = 0; i < 3; i++)
        if (!THPVariable_Check(p[i])) Py_RETURN_NONE;
    const at::Tensor &res = THPVariable_Unpack(p[0]), &k = THPVariable_Unpack(p[1]), &v = THPVariable_Unpack(p[2]);
    const auto aligned = [](const at::Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; };
    const auto row = [&](const at::Tensor& t) {
        return t.is_cuda() && t.device() == res.device() && t.scalar_type() == res.scalar_type() && t.dim() == 4 && t.size(0) == res.size(0) &&
               t.size(1) == res.size(1) && t.size(2) == 1 && t.size(3) == 128 && t.stride(3) == 1 && t.stride(0) % 8 == 0 && t.stride(1) % 8 == 0 && aligned(t);
    };
    if (res.dim() != 4 || !half_type(res) || !row(k) || !row(v)) Py_RETURN_NONE;
    if (p[3] != Py_None) {
        if (!THPVariable_Check(p[3]) || !THPVariable_Check(p[4])) Py_RETURN_NONE;
        const at::Tensor &cos = THPVariable_Unpack(p[3]), &sin = THPVariable_Unpack(p[4]);
        const auto table = [&](const at::Tensor& t) {
            return t.is_cuda() && t.device() == res.device() && t.scalar_type() == res.scalar_type() && t.dim() >= 2 && t.size(-2) == 1 && t.size(-1) == 128 &&
                   t.is_contiguous() && (t.size(0) == 1 || t.numel() >= res.size(0) * 128) && aligned(t);
        };
        if (!table(cos) || !table(sin) || cos.sizes() != sin.sizes()) Py_RETURN_NONE;
    }
    return PyLong_FromVoidPtr(c10::cuda::getCurrentCUDAStream(res.get_device()).stream());
}

// tensor -> the handle of its device's current stream
PyObject* stream_of(PyObject* const* p) { return PyLong_FromVoidPtr(c10::cuda::getCurrentCUDAStream(cuda(p[0], "tensor").get_device()).stream()); }

// x, cos, sin, out -> out
PyObject* rope(PyObject* const* p) {
    const at::Tensor &x = cuda(p[0], "x"), &cos = cuda(p[1], "cos"), &sin = cuda(p[2], "sin");
    const at::Tensor* out = maybe_cuda(p[3], "out");
    check(x.dim() == 4 && x.stride(3) == 1 && half_type(x), "x must be (B, H, T, D) fp16/bf16 with contiguous channels");
    const Tables cs(cos, sin, x.scalar_type(), x.size(0), x.size(2), x.size(3), "cos/sin must be (B or 1, T, D)");
    at::Tensor own;
    if (!out) { own = at::empty(x.sizes(), x.options()); out = &own; }
    bool holds = out->dim() == 4 && out->scalar_type() == x.scalar_type() && out->stride(3) == 1;
    for (int i = 0; i < 4; i++) holds = holds && out->size(i) >= x.size(i);
    check(holds, "out must be of x's size and dtype with contiguous channels");
    const int batch = extent(x.size(0)), heads = extent(x.size(1)), tokens = extent(x.size(2)), dim = extent(x.size(3));
    check_status(unlocked([&, on = stream()] {
                     return lib.rope(x.data_ptr(), x.stride(0), x.stride(1), x.stride(2), cs.cos.data_ptr(), cs.sin.data_ptr(), cs.stride_b,
                                     out->data_ptr(), out->stride(0), out->stride(1), out->stride(2), batch, heads, tokens, dim, is_bf16(x), on);
                 }),
                 "rope");
    if (p[3] != Py_None) return Py_NewRef(p[3]);
    return THPVariable_Wrap(own);
}

// ---- module -------------------------------------------------------------------------------------------------------------
template <PyObject* (*F)(PyObject* const*), Py_ssize_t N>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != N) {
        PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", N, n);
        return nullptr;
    }
    if (!lib.attention) {
        PyErr_SetString(PyExc_RuntimeError, "the library is not bound");
        return nullptr;
    }
    try {
        return F(args);
    } catch (const Raised&) {
        return nullptr;
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

// addresses of the library's functions, in the order of struct Library
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
    void* at[sizeof(Library) / sizeof(void*)];
    if (n != (Py_ssize_t)(sizeof at / sizeof at[0])) {
        PyErr_SetString(PyExc_TypeError, "bind takes one address for each library function");
        return nullptr;
    }
    for (Py_ssize_t i = 0; i < n; i++) {
        at[i] = PyLong_AsVoidPtr(args[i]);
        if (PyErr_Occurred()) return nullptr;
    }
    static_assert(sizeof at == sizeof lib);
    std::memcpy(&lib, at, sizeof lib);
    Py_RETURN_NONE;
}

#define FAST(fn, n, doc) {#fn, (PyCFunction)(void (*)(void))entry<fn, n>, METH_FASTCALL, doc}
PyMethodDef methods[] = {
    {"bind", (PyCFunction)(void (*)(void))bind, METH_FASTCALL, "addresses of the library's functions"},
    FAST(decode_attention, 14, "ops.decode_attention"),
    FAST(decode_attention_narrow, 10, "ops.decode_attention for heads of 64 .. 120 channels"),
    FAST(encode_tensor, 18, "ops.encode_tensor / ops.encode_tensor_static"),
    FAST(value_median_order, 4, "ops.value_median_order"),
    FAST(append_residual, 7, "ops.append_residual"),
    FAST(waiting_step, 5, "whether a decode step's rows can wait for the attention launch"),
    FAST(stream_of, 1, "handle of the current stream of a tensor's device"),
    FAST(rope, 4, "ops.rope"),
    FAST(widen_rows, 8, "ops.widen_rows"),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "native host path of packkv_b200.ops", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
#define X(n) \
    if (!(names.n = PyUnicode_InternFromString(#n))) return nullptr;
    LAYER_NAMES(X)
#undef X
    return PyModule_Create(&module);
}
