// The checks and launches of the entry points that a step calls most, as functions of a Python module.
//
// A step of few tokens is bound by what the host does for a launch.  The same checks and the same call through Python's tensor attributes and ctypes took 6 to
// 11 us a launch where the CUDA call takes 3; here they take under one.  Every function checks what it is given at every call, with the errors of the functions
// in kernels/ops.py that call it, takes the current stream, lets go of the interpreter's lock for the launch, and returns the entry point's status.  Nothing is
// kept from call to call but the entry points' addresses.  An entry point is looked for by the first call that needs it and has passed its checks (binder), so that
// what is refused is refused before anything is compiled or loaded.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <initializer_list>
#include <sstream>
#include <string>

namespace {

struct Failed {};                      // a Python error is set
PyObject *kernel_error = nullptr, *binder = nullptr;

[[noreturn]] void fail(PyObject* type, const char* what) {
    PyErr_SetString(type, what);
    throw Failed{};
}
#define NEED(condition) do { if (!(condition)) fail(PyExc_AssertionError, #condition); } while (0)

typedef const at::Tensor* T;

T maybe(PyObject* o) {
    if (o == Py_None) return nullptr;
    if (!THPVariable_Check(o)) fail(PyExc_TypeError, "a tensor expected");
    return &THPVariable_Unpack(o);
}
T tensor(PyObject* o) {
    T t = maybe(o);
    if (!t) fail(PyExc_TypeError, "a tensor expected, not None");
    return t;
}
long long whole(PyObject* o) {
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw Failed{};
    return v;
}
int small(PyObject* o) { return static_cast<int>(whole(o)); }
float real(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw Failed{};
    return static_cast<float>(v);
}
bool truth(PyObject* o) {
    const int v = PyObject_IsTrue(o);
    if (v < 0) throw Failed{};
    return v;
}
void on_device(std::initializer_list<T> all) {
    for (T t : all)
        if (t && !t->is_cuda()) {
            const std::string where = "the engine's kernels run on a CUDA device only; got a tensor on " + t->device().str();
            fail(kernel_error, where.c_str());
        }
}
bool f32(T t) { return t->scalar_type() == at::kFloat; }
bool b16(T t) { return t->scalar_type() == at::kBFloat16; }
int type_of(T t) {
    if (f32(t)) return 0;
    if (b16(t)) return 1;
    const std::string what = std::string("element type ") + c10::toString(t->scalar_type()) + " not supported (float32 or bfloat16)";
    fail(kernel_error, what.c_str());
}
int type_or_f32(T t) { return t ? type_of(t) : 0; }
void* at_(T t) { return t ? t->data_ptr() : nullptr; }
const float* floats(T t) { return static_cast<const float*>(at_(t)); }
const int* ints(T t, const char* name) {
    if (t->scalar_type() != at::kInt || !t->is_contiguous()) {
        const std::string what = std::string(name) + " must be a contiguous int32 tensor";
        fail(kernel_error, what.c_str());
    }
    return static_cast<const int*>(t->data_ptr());
}
const int* maybe_ints(T t, const char* name) { return t ? ints(t, name) : nullptr; }
bool shaped(T t, std::initializer_list<int64_t> sizes) {
    if (t->dim() != static_cast<int64_t>(sizes.size())) return false;
    int64_t i = 0;
    for (int64_t s : sizes)
        if (t->size(i++) != s) return false;
    return true;
}
std::string sizes(T t) {
    std::ostringstream text;
    text << t->sizes() << " stride " << t->strides();
    return text.str();
}
void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// a fused projection [n, W] (parts 0), or float32 partial sums [parts, n, W]
struct Fused {
    void* p;
    int type, row_stride, parts;
    long long part_stride;
    int n;
    Fused(T t, int parts_) {
        if (parts_) NEED(t->dim() == 3 && t->size(0) == parts_ && t->stride(2) == 1 && f32(t));
        else NEED(t->dim() == 2 && t->stride(1) == 1);
        const int axis = parts_ ? 1 : 0;
        p = t->data_ptr();
        type = type_of(t);
        row_stride = static_cast<int>(t->stride(axis));
        parts = parts_ ? parts_ : 1;
        part_stride = parts_ ? t->stride(0) : 0;
        n = static_cast<int>(t->size(axis));
    }
};
// a branch output [n, H] (parts 0), or float32 partial sums [parts, n, H]; nothing: no branch
struct Branch {
    void* p = nullptr;
    int type = 0, parts = 1;
    long long stride = 0;
    Branch(T t, int parts_, int64_t n, int64_t H) {
        if (!t) return;
        NEED(t->is_contiguous() && t->dim() >= 2 && t->size(-2) == n && t->size(-1) == H);
        if (parts_) NEED(f32(t) && t->size(0) == parts_);
        p = t->data_ptr();
        type = type_of(t);
        parts = parts_ > 1 ? parts_ : 1;
        stride = parts_ ? n * H : 0;
    }
};

// -- the entry points (csrc/gemm_bf16_tc.cu, norm.cu, rope_cache.cu, attention_mma.cu) ---------------------------------------------------
typedef int (*GemmFn)(const void*, int, const void*, int, void*, int, int, int, int, int, int, int, int*, int, float, float, void*);
typedef int (*NormFn)(float*, const void*, int, int, long long, const void*, int, float, float, int, void*, int, const int*, int, int, void*);
typedef int (*SandwichFn)(float*, const void*, int, int, long long, const void*, const void*, int, int, long long, const void*, float, float, const void*, float,
                          int, float, const void*, float, int, float, int, void*, int, const int*, int, int, const float*, void*);
typedef int (*RopeFn)(const void*, int, int, int, long long, void*, int, int, const int*, const int*, const float*, void*, void*, int, int, int, int, int, int, int,
                      int, int, float, float, void*);
typedef int (*RopeRowFn)(const void*, int, int, int, long long, void*, int, int, const int*, const int*, const float*, void*, void*, int, int, int, int, int, int,
                         int, int, const void*, const void*, int, int, int, float, const float*, float*, const float*, int, float, void*);
typedef int (*DecodeFn)(const void*, int, void*, int, const void*, const void*, long long, const int*, const int*, const int*, const int*, int, int, int, int, int,
                        int, float, int, int, float*, int*, const float*, float, int, const float*, void*);
typedef int (*PrefillFn)(const void*, int, void*, int, const void*, const void*, long long, const int*, const int*, const int*, const int*, int, int, int, int, int,
                         int, int, float, int, int, int, float*, int*, const float*, float, int, const float*, void*);

GemmFn gemm_fn;
NormFn norm_fn;
SandwichFn sandwich_fn;
RopeFn rope_fn;
RopeRowFn rope_row_fn;
DecodeFn decode_fn[257];               // by head size
PrefillFn prefill_fn[257];

// the binder hands the addresses over: of one entry point (its name), or of a head size's two (the size)
PyObject* asked(const char* name) { return PyUnicode_FromString(name); }
PyObject* asked(int head_size) { return PyLong_FromLong(head_size); }

// (the arguments, and with them what is left to check in them, are worked out before this is entered)
template <typename Fn, typename Which, typename... Args>
PyObject* launch(Fn& fn, Which which, Args... args) {
    if (!fn) {
        PyObject* what = asked(which);
        PyObject* done = what && binder ? PyObject_CallOneArg(binder, what) : nullptr;
        Py_XDECREF(what);
        Py_XDECREF(done);
        if (PyErr_Occurred()) throw Failed{};
        if (!fn) fail(PyExc_RuntimeError, "the entry point is not bound");
    }
    int status;
    Py_BEGIN_ALLOW_THREADS
    status = fn(args...);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(status);
}

typedef PyObject* const* Args;
void count(Py_ssize_t n, Py_ssize_t want) {
    if (n != want) fail(PyExc_TypeError, "wrong number of arguments");
}

// shapes that the tensor-memory product takes
bool product_ok(T a, T w) {
    return b16(a) && b16(w) && a->dim() == 2 && w->dim() == 2 && a->stride(1) == 1 && w->stride(1) == 1 && a->size(1) % 8 == 0 && a->stride(0) % 8 == 0 &&
           w->stride(0) % 8 == 0 && reinterpret_cast<uintptr_t>(a->data_ptr()) % 16 == 0 && reinterpret_cast<uintptr_t>(w->data_ptr()) % 16 == 0;
}
PyObject* tc_gemm_ok(Args v, Py_ssize_t n) {
    count(n, 2);
    return PyBool_FromLong(product_ok(tensor(v[0]), tensor(v[1])));
}

// a, w, out, epilogue, gated, k_splits, half_rows, max_ctas, limit, slope, status, checked
PyObject* gemm(Args v, Py_ssize_t n) {
    count(n, 12);
    T a = tensor(v[0]), w = tensor(v[1]), out = tensor(v[2]), status = tensor(v[10]);
    on_device({a, w, out});
    if (!truth(v[11]) && !product_ok(a, w))
        fail(kernel_error, ("gemm_bf16_tc: bfloat16 operands with K and row pitches in steps of 8 elements, 16-byte aligned; got a" + sizes(a) + " w" +
                            sizes(w)).c_str());
    const int epilogue = small(v[3]), splits = small(v[5]);
    const int64_t M = a->size(0), K = a->size(1), N = w->size(0), cols = truth(v[4]) ? N / 2 : N;
    NEED(w->size(1) == K);
    NEED((splits == 1 ? shaped(out, {M, cols}) : shaped(out, {splits, M, cols})) && out->stride(-1) == 1 && (epilogue == 1 ? f32(out) : b16(out)));
    NEED(splits == 1 || (epilogue == 1 && out->is_contiguous()));
    return launch(gemm_fn, "wllm_gemm_bf16_tc_params",
                  at_(a), (int)a->stride(0), at_(w), (int)w->stride(0), at_(out), (int)out->stride(-2), (int)M, (int)N, (int)K, epilogue, splits,
                  small(v[6]), static_cast<int*>(at_(status)), small(v[7]), real(v[8]), real(v[9]), stream());
}

// resid, delta, weight, eps, offset, out, rows, delta_splits, center
PyObject* norm(Args v, Py_ssize_t n) {
    count(n, 9);
    T resid = tensor(v[0]), delta = maybe(v[1]), weight = maybe(v[2]), out = tensor(v[5]), rows = maybe(v[6]);
    on_device({resid, delta, weight, out, rows});
    const int splits = small(v[7]);
    const int64_t H = resid->size(1), n_out = rows ? rows->size(0) : resid->size(0);
    NEED(f32(resid) && resid->is_contiguous() && out->is_contiguous() && shaped(out, {n_out, H}));
    NEED(!weight || (shaped(weight, {H}) && weight->is_contiguous()));
    long long split_stride = 0;
    if (delta) {
        NEED(delta->is_contiguous());
        if (splits) {
            NEED(shaped(delta, {splits, resid->size(0), H}) && f32(delta));
            split_stride = resid->numel();
        } else NEED(shaped(delta, {resid->size(0), H}));
    }
    return launch(norm_fn, "wllm_norm",
                  static_cast<float*>(at_(resid)), at_(delta), type_or_f32(delta), splits > 1 ? splits : 1, split_stride, at_(weight),
                  type_or_f32(weight), real(v[3]), real(v[4]), truth(v[8]) ? 1 : 0, at_(out), type_of(out), maybe_ints(rows, "rows"), (int)n_out, (int)H, stream());
}

// resid, a, a_parts, out, post_weight, post_center, post_eps, weight, offset, center, eps, rows, gain_a, b, b_parts, gain_b, inner_eps, factor, post_offset, bias
PyObject* sandwich(Args v, Py_ssize_t n) {
    count(n, 20);
    T resid = tensor(v[0]), a = tensor(v[1]), out = tensor(v[3]), post = tensor(v[4]), weight = maybe(v[7]), rows = maybe(v[11]), gain_a = maybe(v[12]),
      b = maybe(v[13]), gain_b = maybe(v[15]), bias = maybe(v[19]);
    const int64_t N = resid->size(0), H = resid->size(1), n_out = rows ? rows->size(0) : N;
    on_device({resid, a, out, post, weight, rows, gain_a, gain_b, b});
    NEED(f32(resid) && resid->is_contiguous() && out->is_contiguous() && shaped(out, {n_out, H}));
    for (T g : {post, weight, gain_a, gain_b}) NEED(!g || (shaped(g, {H}) && g->is_contiguous() && g->scalar_type() == post->scalar_type()));
    NEED(!bias || (f32(bias) && shaped(bias, {H}) && bias->is_contiguous()));
    const Branch pa(a, small(v[2]), N, H), pb(b, small(v[14]), N, H);
    return launch(sandwich_fn, "wllm_sandwich_norm_offset",
                  static_cast<float*>(at_(resid)), pa.p, pa.type, pa.parts, pa.stride, at_(gain_a), pb.p, pb.type, pb.parts, pb.stride, at_(gain_b),
                  real(v[16]), real(v[17]), at_(post), real(v[18]), truth(v[5]) ? 1 : 0, real(v[6]), at_(weight), real(v[8]), truth(v[9]) ? 1 : 0, real(v[10]),
                  type_of(post), at_(out), type_of(out), maybe_ints(rows, "rows"), (int)n_out, (int)H, floats(bias), stream());
}

// what the rotating entry points share: the queries' rows out, frequencies, pages
void rotation(T q_out, int64_t n, int64_t nq, int64_t hd, T inv_freq, int64_t rot_dim, T slots, T k_pages, T v_pages) {
    NEED(shaped(q_out, {n, nq * hd}) && q_out->stride(1) == 1);
    NEED(f32(inv_freq) && inv_freq->numel() == rot_dim / 2 && inv_freq->is_contiguous());
    if (slots)
        NEED(k_pages && v_pages && k_pages->is_contiguous() && v_pages->is_contiguous() && k_pages->scalar_type() == q_out->scalar_type() &&
             v_pages->scalar_type() == q_out->scalar_type());
}

// qkv, q_out, positions, slots, inv_freq, k_pages, v_pages, nq, nkv, hd, rot_dim, page_size, in_splits, interleaved, vd, unit_norm_eps, turn_scale
PyObject* rope(Args v, Py_ssize_t n) {
    count(n, 17);
    T qkv = tensor(v[0]), q_out = tensor(v[1]), positions = tensor(v[2]), slots = maybe(v[3]), inv_freq = tensor(v[4]), kp = maybe(v[5]), vp = maybe(v[6]);
    on_device({qkv, q_out, positions, slots, inv_freq, kp, vp});
    const int nq = small(v[7]), nkv = small(v[8]), hd = small(v[9]), rot = small(v[10]), vd = v[14] == Py_None ? hd : small(v[14]);
    NEED(nkv > 0 || !slots);
    const Fused f(qkv, small(v[12]));
    NEED(qkv->size(-1) == (int64_t)(nq + nkv) * hd + (int64_t)nkv * vd);
    rotation(q_out, f.n, nq, hd, inv_freq, rot, slots, kp, vp);
    const bool unit = v[15] != Py_None;
    return launch(rope_fn, "wllm_rope_kv_write_general",
                  f.p, f.type, f.row_stride, f.parts, f.part_stride, at_(q_out), type_of(q_out), (int)q_out->stride(0), ints(positions, "positions"),
                  maybe_ints(slots, "slots"), floats(inv_freq), at_(kp), at_(vp), f.n, nq, nkv, hd, rot, small(v[11]), truth(v[13]) ? 1 : 0, vd, unit ? 1 : 0,
                  unit ? real(v[15]) : 0.f, real(v[16]), stream());
}

// qkv, q_out, positions, slots, inv_freq, k_pages, v_pages, nq, nkv, hd, rot_dim, page_size, q_gain, k_gain, eps, q_count, k_count, in_splits, interleaved, vd,
// bias, v_first, blend, mix (0, 1 first, 2 later), turn_scale
PyObject* rope_row(Args v, Py_ssize_t n) {
    count(n, 25);
    T qkv = tensor(v[0]), q_out = tensor(v[1]), positions = tensor(v[2]), slots = maybe(v[3]), inv_freq = tensor(v[4]), kp = maybe(v[5]), vp = maybe(v[6]),
      q_gain = tensor(v[12]), k_gain = maybe(v[13]), bias = maybe(v[20]), v_first = maybe(v[21]), blend = maybe(v[22]);
    on_device({qkv, q_out, positions, slots, inv_freq, kp, vp, q_gain, k_gain});
    const int nq = small(v[7]), nkv = small(v[8]), hd = small(v[9]), rot = small(v[10]), vd = v[19] == Py_None ? hd : small(v[19]), mix = small(v[23]);
    const Fused f(qkv, small(v[17]));
    const int64_t width = (int64_t)(nq + nkv) * hd + (int64_t)nkv * vd;
    NEED(qkv->size(-1) >= width);
    rotation(q_out, f.n, nq, hd, inv_freq, rot, slots, kp, vp);
    NEED(shaped(q_gain, {(int64_t)nq * hd}) && q_gain->is_contiguous() && (nkv > 0 || !slots));
    NEED(k_gain ? (shaped(k_gain, {(int64_t)nkv * hd}) && k_gain->scalar_type() == q_gain->scalar_type() && k_gain->is_contiguous()) : nkv == 0);
    on_device({bias, v_first, blend});
    NEED(!bias || (f32(bias) && shaped(bias, {width}) && bias->is_contiguous()));
    if (mix) {
        NEED(v_first && f32(v_first) && shaped(v_first, {f.n, (int64_t)nkv * vd}) && v_first->is_contiguous());
        NEED(mix == 1 || (blend && f32(blend) && blend->numel() == 1));
    }
    return launch(rope_row_fn, "wllm_rope_row_norm_kv_write",
                  f.p, f.type, f.row_stride, f.parts, f.part_stride, at_(q_out), type_of(q_out), (int)q_out->stride(0), ints(positions, "positions"),
                  maybe_ints(slots, "slots"), floats(inv_freq), at_(kp), at_(vp), f.n, nq, nkv, hd, rot, small(v[11]), truth(v[18]) ? 1 : 0, vd, at_(q_gain),
                  at_(k_gain), type_of(q_gain), small(v[15]), small(v[16]), real(v[14]), floats(bias), static_cast<float*>(mix ? at_(v_first) : nullptr),
                  mix == 2 ? floats(blend) : nullptr, mix, real(v[24]), stream());
}

void attention_operands(T q, T out, T kp, T vp, T sinks, T slopes, int64_t nq) {
    NEED(!slopes || (f32(slopes) && shaped(slopes, {nq}) && slopes->is_contiguous()));
    NEED(!sinks || (f32(sinks) && shaped(sinks, {nq}) && sinks->is_contiguous()));
    NEED(b16(q) && b16(out) && b16(kp) && q->stride(1) == 1 && out->stride(1) == 1);
    NEED(kp->is_contiguous() && vp->is_contiguous());
}

// q, out, k_pages, v_pages, req_q_start, req_q_len, req_ctx_len, block_table, nq, nkv, hd, page_size, window, scale, split_keys, max_splits, scratch, status,
// sinks, cap, keep, slopes
PyObject* attention_decode(Args v, Py_ssize_t n) {
    count(n, 22);
    T q = tensor(v[0]), out = tensor(v[1]), kp = tensor(v[2]), vp = tensor(v[3]), start = tensor(v[4]), len = tensor(v[5]), ctx = tensor(v[6]), table = tensor(v[7]),
      scratch = tensor(v[16]), status = tensor(v[17]), sinks = maybe(v[18]), slopes = maybe(v[21]);
    on_device({q, out, kp, vp, start, len, ctx, table, scratch, sinks, slopes});
    const int nq = small(v[8]), hd = small(v[10]), splits = small(v[15]), R = (int)len->size(0);
    attention_operands(q, out, kp, vp, sinks, slopes, nq);
    NEED(f32(scratch) && scratch->numel() >= (int64_t)R * nq * splits * (hd + 2));
    NEED(hd > 0 && hd <= 256);
    return launch(decode_fn[hd], hd,
                  at_(q), (int)q->stride(0), at_(out), (int)out->stride(0), at_(kp), at_(vp), (long long)kp->size(0), ints(start, "req_q_start"),
                  ints(len, "req_q_len"), ints(ctx, "req_ctx_len"), ints(table, "block_table"), (int)table->size(1), R, nq, small(v[9]), small(v[11]), small(v[12]),
                  real(v[13]), small(v[14]), splits, static_cast<float*>(at_(scratch)), static_cast<int*>(at_(status)), floats(sinks), real(v[19]), small(v[20]),
                  floats(slopes), stream());
}

// q, out, k_pages, v_pages, req_q_start, req_q_len, req_ctx_len, block_table, max_q_len, nq, nkv, hd, page_size, window, scale, skip_single, multi, split_above,
// halves, halves_floats, status, sinks, cap, keep, slopes
PyObject* attention_prefill(Args v, Py_ssize_t n) {
    count(n, 25);
    T q = tensor(v[0]), out = tensor(v[1]), kp = tensor(v[2]), vp = tensor(v[3]), start = tensor(v[4]), len = tensor(v[5]), ctx = tensor(v[6]), table = tensor(v[7]),
      halves = maybe(v[18]), status = tensor(v[20]), sinks = maybe(v[21]), slopes = maybe(v[24]);
    on_device({q, out, kp, vp, start, len, ctx, table, halves, sinks, slopes});
    const int nq = small(v[9]), hd = small(v[11]), split_above = small(v[17]), R = (int)len->size(0);
    attention_operands(q, out, kp, vp, sinks, slopes, nq);
    if (split_above > 0) {
        NEED(hd % 64 == 0 && halves && f32(halves) && halves->is_contiguous());
        NEED(halves->numel() >= whole(v[19]));
    }
    NEED(hd > 0 && hd <= 256);
    return launch(prefill_fn[hd], hd,
                  at_(q), (int)q->stride(0), at_(out), (int)out->stride(0), at_(kp), at_(vp), (long long)kp->size(0), ints(start, "req_q_start"),
                  ints(len, "req_q_len"), ints(ctx, "req_ctx_len"), ints(table, "block_table"), (int)table->size(1), R, small(v[8]), nq, small(v[10]), small(v[12]),
                  small(v[13]), real(v[14]), truth(v[15]) ? 1 : 0, small(v[16]), split_above, static_cast<float*>(split_above > 0 ? at_(halves) : nullptr),
                  static_cast<int*>(at_(status)), floats(sinks), real(v[22]), small(v[23]), floats(slopes), stream());
}

// -- the module ---------------------------------------------------------------------------------------------------------------------
PyObject* bind(Args v, Py_ssize_t n) {           // name, address
    count(n, 2);
    const char* name = PyUnicode_AsUTF8(v[0]);
    if (!name) throw Failed{};
    void* p = PyLong_AsVoidPtr(v[1]);
    if (!p) fail(PyExc_ValueError, "no address");
    const std::string which = name;
    if (which == "wllm_gemm_bf16_tc_params") gemm_fn = reinterpret_cast<GemmFn>(p);
    else if (which == "wllm_norm") norm_fn = reinterpret_cast<NormFn>(p);
    else if (which == "wllm_sandwich_norm_offset") sandwich_fn = reinterpret_cast<SandwichFn>(p);
    else if (which == "wllm_rope_kv_write_general") rope_fn = reinterpret_cast<RopeFn>(p);
    else if (which == "wllm_rope_row_norm_kv_write") rope_row_fn = reinterpret_cast<RopeRowFn>(p);
    else fail(PyExc_ValueError, "no such entry point");
    Py_RETURN_NONE;
}
PyObject* bind_attention(Args v, Py_ssize_t n) { // head size, address of decode, of prefill
    count(n, 3);
    const long long hd = whole(v[0]);
    if (hd < 1 || hd > 256) fail(PyExc_ValueError, "head sizes of 1 to 256");
    void *d = PyLong_AsVoidPtr(v[1]), *p = PyLong_AsVoidPtr(v[2]);
    if (!d || !p) fail(PyExc_ValueError, "no address");
    decode_fn[hd] = reinterpret_cast<DecodeFn>(d);
    prefill_fn[hd] = reinterpret_cast<PrefillFn>(p);
    Py_RETURN_NONE;
}
PyObject* errors(Args v, Py_ssize_t n) {         // the class that ops.KernelError is; what binds an entry point
    count(n, 2);
    Py_INCREF(v[0]);
    Py_INCREF(v[1]);
    Py_XDECREF(kernel_error);
    Py_XDECREF(binder);
    kernel_error = v[0];
    binder = v[1];
    Py_RETURN_NONE;
}

template <PyObject* (*F)(Args, Py_ssize_t)>
PyObject* guarded(PyObject*, Args v, Py_ssize_t n) {
    try {
        return F(v, n);
    } catch (const Failed&) {
    } catch (const std::exception& e) {          // what torch throws (a tensor without storage, too few dimensions)
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}
#define METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&guarded<name>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {METHOD(bind), METHOD(bind_attention), METHOD(errors), METHOD(tc_gemm_ok), METHOD(gemm), METHOD(norm), METHOD(sandwich), METHOD(rope),
                         METHOD(rope_row), METHOD(attention_decode), METHOD(attention_prefill), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "wllm_host_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_wllm_host_calls() { return PyModule_Create(&module); }
