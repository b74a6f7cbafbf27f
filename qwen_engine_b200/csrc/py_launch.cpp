// Python entry points of the launch functions: one builtin per launcher, straight from torch tensors to the C ABI.
//
// What bounds these calls is the host.  The kernels of a decode step take 1-4 us each, and a ctypes wrapper needs
// 5-6 us of interpreter time per call (a data_ptr() and a type conversion per tensor, the current stream, the foreign
// call itself) on top of the launch.  Here a call is one vectorcall: arguments are matched by position or interned
// name, tensors are read through THPVariable_Unpack, the current stream comes from c10.  Measured per call on B200:
// launch_gemv_w4a16 1536 x 1536, launched back to back, 8.7 -> 3.3 us; the 8 launches of a decode layer 71.5 -> 25.3 us.
//
// Argument rules, the same for every function: a tensor argument is a CUDA torch tensor or None, an integer anything
// with __index__, `stream` None (the current stream), an object with `cuda_stream`, or a raw handle.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <array>
#include <cstring>
#include <exception>
#include <tuple>
#include <type_traits>

#include "../../include/w4a16_b200.h"

namespace {

// One argument: its Python name and, for optional integers, the default.
struct Arg {
    const char* name;
    bool optional = false;
    int def = 0;
};
constexpr int kMaxArgs = 14;
struct Spec {
    const char* name;         // Python name
    const char* c_name;       // C ABI name, for error messages
    int n;
    Arg args[kMaxArgs];
    const char* doc;
};

constexpr int kHidden = 1536, kInter = 8960, kQHeads = 12, kKvHeads = 2, kHeadDim = 128, kVocab = 151936;

PyObject* g_str_cuda_stream = nullptr;
PyObject* g_check = nullptr;                                  // qwen_engine_b200._lib.check
PyObject* g_view_names[9] = {};                               // attributes of QKVProjectionView, in the C struct's order

// A torch call that may throw (a tensor without storage, as under vmap; the current stream where CUDA cannot start): a C++
// exception must not leave through the interpreter's C frames, which ends the process.
template <typename F>
bool torch_call(F&& f) {
    try {
        f();
        return true;
    } catch (const c10::Error& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return false;
}
bool not_on_device() {
    PyErr_SetString(PyExc_ValueError, "device pointer expected: tensor is not on a CUDA device");
    return false;
}
// Objects that are not torch tensors but offer is_cuda and data_ptr().
bool duck_pointer(PyObject* o, void** out) {
    PyObject* on_device = PyObject_GetAttrString(o, "is_cuda");
    if (on_device == nullptr) return false;
    const int yes = PyObject_IsTrue(on_device);
    Py_DECREF(on_device);
    if (yes < 0) return false;
    if (yes == 0) return not_on_device();
    PyObject* p = PyObject_CallMethod(o, "data_ptr", nullptr);
    if (p == nullptr) return false;
    *out = PyLong_AsVoidPtr(p);
    Py_DECREF(p);
    return *out != nullptr || !PyErr_Occurred();
}
bool to_pointer(PyObject* o, void** out) {
    if (o == Py_None) { *out = nullptr; return true; }
    if (!THPVariable_Check(o)) return duck_pointer(o, out);
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.is_cuda()) return not_on_device();
    return torch_call([&] { *out = t.data_ptr(); });
}
bool to_int(PyObject* o, int* out) {
    long v = PyLong_CheckExact(o) ? PyLong_AsLong(o) : -1;
    if (!PyLong_CheckExact(o)) {
        PyObject* i = PyNumber_Index(o);
        if (i == nullptr) return false;
        v = PyLong_AsLong(i);
        Py_DECREF(i);
    }
    if (v == -1 && PyErr_Occurred()) return false;
    if (v != static_cast<int>(v)) { PyErr_SetString(PyExc_OverflowError, "argument does not fit a C int"); return false; }
    *out = static_cast<int>(v);
    return true;
}
bool to_stream(PyObject* o, w4a16_stream_t* out) {
    if (o == nullptr || o == Py_None) {
        return torch_call([&] { *out = reinterpret_cast<w4a16_stream_t>(c10::cuda::getCurrentCUDAStream().stream()); });
    }
    PyObject* handle = nullptr;
    if (PyLong_Check(o)) {
        handle = Py_NewRef(o);
    } else if (PyObject_HasAttr(o, g_str_cuda_stream)) {
        handle = PyObject_GetAttr(o, g_str_cuda_stream);
    } else {
        handle = PyNumber_Long(o);
    }
    if (handle == nullptr) return false;
    void* p = PyLong_AsVoidPtr(handle);
    Py_DECREF(handle);
    if (p == nullptr && PyErr_Occurred()) return false;
    *out = reinterpret_cast<w4a16_stream_t>(p);
    return true;
}
bool to_view(PyObject* o, w4a16_qkv_view* v) {
    void* p[9];
    for (int i = 0; i < 9; ++i) {
        PyObject* t = PyObject_GetAttr(o, g_view_names[i]);
        if (t == nullptr) return false;
        const bool ok = to_pointer(t, &p[i]);
        Py_DECREF(t);               // the view object holds the tensor
        if (!ok) return false;
    }
    static_assert(sizeof(w4a16_qkv_view) == sizeof(p), "the view is nine pointers");
    std::memcpy(v, p, sizeof(p));
    return true;
}

// Storage and conversion of one C parameter.
template <typename T>
struct Slot {                        // any pointer but the two below
    static_assert(std::is_pointer_v<T>);
    void* p = nullptr;
    bool take(PyObject* o, const Arg&) { return to_pointer(o, &p); }
    T get() { return static_cast<T>(p); }
};
template <>
struct Slot<int> {
    int v = 0;
    bool take(PyObject* o, const Arg& a) {
        if (o == nullptr) { v = a.def; return true; }
        return to_int(o, &v);
    }
    int get() { return v; }
};
template <>
struct Slot<w4a16_stream_t> {
    w4a16_stream_t s = nullptr;
    bool take(PyObject* o, const Arg&) { return to_stream(o, &s); }
    w4a16_stream_t get() { return s; }
};
template <>
struct Slot<const w4a16_qkv_view*> {
    w4a16_qkv_view v{};
    bool take(PyObject* o, const Arg&) { return to_view(o, &v); }
    const w4a16_qkv_view* get() { return &v; }
};

// Positional and keyword arguments into `got` (borrowed, null where left out).
bool match_args(const Spec& s, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames, PyObject** got) {
    if (nargs > s.n) {
        PyErr_Format(PyExc_TypeError, "%s() takes at most %d arguments (%zd given)", s.name, s.n, nargs);
        return false;
    }
    for (int i = 0; i < s.n; ++i) got[i] = i < nargs ? args[i] : nullptr;
    const Py_ssize_t nkw = kwnames != nullptr ? PyTuple_GET_SIZE(kwnames) : 0;
    for (Py_ssize_t k = 0; k < nkw; ++k) {
        PyObject* key = PyTuple_GET_ITEM(kwnames, k);
        int i = 0;
        while (i < s.n && PyUnicode_CompareWithASCIIString(key, s.args[i].name) != 0) ++i;
        if (i == s.n) {
            PyErr_Format(PyExc_TypeError, "%s() got an unexpected keyword argument '%U'", s.name, key);
            return false;
        }
        if (got[i] != nullptr) {
            PyErr_Format(PyExc_TypeError, "%s() got multiple values for argument '%s'", s.name, s.args[i].name);
            return false;
        }
        got[i] = args[nargs + k];
    }
    for (int i = 0; i < s.n; ++i)
        if (got[i] == nullptr && !s.args[i].optional) {
            PyErr_Format(PyExc_TypeError, "%s() missing required argument '%s'", s.name, s.args[i].name);
            return false;
        }
    return true;
}

PyObject* finish(const char* c_name, int status) {
    if (__builtin_expect(status == 0, 1)) Py_RETURN_NONE;
    return PyObject_CallFunction(g_check, "si", c_name, status);      // raises W4A16Error
}

template <typename F>
struct Caller;
template <typename... P>
struct Caller<int (*)(P...)> {
    template <size_t... I>
    static PyObject* run(int (*fn)(P...), const Spec& s, PyObject** got, std::index_sequence<I...>) {
        std::tuple<Slot<P>...> slots;
        if (!(std::get<I>(slots).take(got[I], s.args[I]) && ...)) return nullptr;
        int status;
        Py_BEGIN_ALLOW_THREADS          // a full launch queue blocks: other Python threads go on meanwhile
        status = fn(std::get<I>(slots).get()...);
        Py_END_ALLOW_THREADS
        return finish(s.c_name, status);
    }
    static PyObject* call(int (*fn)(P...), const Spec& s, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
        PyObject* got[kMaxArgs];
        if (!match_args(s, args, nargs, kwnames, got)) return nullptr;
        return run(fn, s, got, std::index_sequence_for<P...>{});
    }
    static constexpr int count = sizeof...(P);
};

template <auto Fn, const Spec& S>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
    static_assert(Caller<decltype(Fn)>::count == S.n, "argument list does not match the C function");
    return Caller<decltype(Fn)>::call(Fn, S, args, nargs, kwnames);
}

constexpr Arg kStream{"stream", true, 0};
constexpr Arg opt(const char* name, int def) { return Arg{name, true, def}; }

#define W4_SPEC(py, c, doc, ...)                                                                     \
    constexpr Arg args_##py[] = {__VA_ARGS__};                                                       \
    constexpr Spec make_##py() {                                                                     \
        Spec s{#py, #c, static_cast<int>(std::size(args_##py)), {}, doc};                            \
        for (size_t i = 0; i < std::size(args_##py); ++i) s.args[i] = args_##py[i];                  \
        return s;                                                                                    \
    }                                                                                                \
    constexpr Spec spec_##py = make_##py();
#define W4_ENTRY(py, c) \
    {#py, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&entry<&c, spec_##py>)), METH_FASTCALL | METH_KEYWORDS, spec_##py.doc}

W4_SPEC(launch_quantize_fp16_to_q8_1, w4a16_quantize_fp16_to_q8_1,
        "Mirror of launch_quantize_fp16_to_q8_1 (reference include/kernels.cuh:39-153, as all launch_* below unless noted).",
        {"input_x"}, {"out_q8"}, {"out_scale"}, {"out_sum8"}, {"num_elements"}, kStream)
W4_SPEC(launch_rmsnorm_q8_1, w4a16_rmsnorm_q8_1, "RMSNorm and Q8_1 of a hidden state; the fp16 form too where output_fp16_opt is given.",
        {"input"}, {"gamma"}, {"output_fp16_opt"}, {"out_q8"}, {"out_scale"}, {"out_sum8"}, kStream, opt("hidden_size", kHidden))
W4_SPEC(quantize_attn_heads_f32_to_q8_1, w4a16_quantize_attn_heads_f32_to_q8_1,
        "Q8_1 of attention heads from their fp32 accumulators, with the rule of the reference's flash-decode\n"
        "combine step (src/kernels/attention_gqa.cu:258-310): per head, q = rn(acc / d).",
        {"attn_acc"}, {"attn_out_fp16_opt"}, {"out_q8"}, {"out_scale"}, {"out_sum8"}, {"num_heads"}, opt("head_dim", kHeadDim), kStream)
W4_SPEC(gemv_attn_heads_f32_w4a16, w4a16_gemv_attn_heads_f32_w4a16,
        "O projection straight from the fp32 attention accumulators (quantised per head in the GEMV's prologue).",
        {"qweight"}, {"scales"}, {"attn_acc"}, {"residual"}, {"output_y"}, {"out_features"}, {"in_features"}, kStream)
W4_SPEC(launch_gemv_w4a16, w4a16_gemv_w4a16, "y = W x (+ residual), fp16 activation quantised to Q8_1 inside the launch.",
        {"qweight"}, {"scales"}, {"input_x"}, {"residual"}, {"output_y"}, {"out_features"}, {"in_features"}, kStream)
W4_SPEC(gemv_w4a16_static_scratch, w4a16_gemv_w4a16_static_scratch,
        "launch_gemv_w4a16 for callers that can neither pass nor allocate scratch: the Q8_1 form of\n"
        "the activation goes into a fixed array inside the library (in_features <= 32768; calls that\n"
        "overlap on the GPU race on that array).",
        {"qweight"}, {"scales"}, {"input_x"}, {"residual"}, {"output_y"}, {"out_features"}, {"in_features"}, kStream)
W4_SPEC(launch_gemv_w4a8, w4a16_gemv_w4a8, "y = W x (+ residual), Q8_1 activation.",
        {"qweight"}, {"scales"}, {"input_q8"}, {"input_scale"}, {"input_sum8"}, {"residual"}, {"output_y"}, {"out_features"},
        {"in_features"}, kStream)
W4_SPEC(launch_embed_lookup_w4a16, w4a16_embed_lookup_w4a16,
        "Rows of the W4 embedding table for token ids (or for the control block's token); vocab_size bounds the ids.",
        {"embed_qweight"}, {"embed_scales"}, {"d_token_ids"}, {"out_hidden"}, {"d_control"}, {"num_tokens"}, kStream,
        opt("hidden_size", kHidden), opt("vocab_size", kVocab))
W4_SPEC(launch_sample_and_advance, w4a16_sample_and_advance,
        "Mirror of launch_sample_and_advance (reference include/kernels.cuh:210-219).",
        {"logits"}, {"sample_scratch_val"}, {"sample_scratch_idx"}, {"d_control"}, {"d_token_out"}, kStream, opt("vocab_size", kVocab))
W4_SPEC(launch_gemv_w4a8_sample_candidates, w4a16_gemv_w4a8_sample_candidates,
        "lm_head GEMV that leaves one (score, index) candidate per CTA; output_logits may be None.",
        {"qweight"}, {"scales"}, {"input_q8"}, {"input_scale"}, {"input_sum8"}, {"output_logits"}, {"candidate_val"},
        {"candidate_idx"}, {"d_control"}, {"index_offset"}, {"out_features"}, {"in_features"}, kStream)
W4_SPEC(launch_gemv_w4a8_sample_one_launch, w4a16_gemv_w4a8_sample_one_launch,
        "lm_head + token selection + control-block advance in one launch (d_counter: zero-initialised int32 [1]).",
        {"qweight"}, {"scales"}, {"input_q8"}, {"input_scale"}, {"input_sum8"}, {"output_logits"}, {"sample_scratch_val"},
        {"sample_scratch_idx"}, {"d_counter"}, {"d_control"}, {"d_token_out"}, {"out_features"}, {"in_features"}, kStream)
W4_SPEC(launch_sample_finish, w4a16_sample_finish, "Best of the candidates; writes the token and advances the control block.",
        {"candidate_val"}, {"candidate_idx"}, {"count"}, {"d_control"}, {"d_token_out"}, kStream)
W4_SPEC(launch_gemv_w4a8_sample_and_advance, w4a16_gemv_w4a8_sample_and_advance,
        "launch_gemv_w4a8 (lm_head) + launch_sample_and_advance in one pass over the weights.",
        {"qweight"}, {"scales"}, {"input_q8"}, {"input_scale"}, {"input_sum8"}, {"output_logits"}, {"sample_scratch_val"},
        {"sample_scratch_idx"}, {"d_control"}, {"d_token_out"}, {"out_features"}, {"in_features"}, kStream)
W4_SPEC(launch_gemv_qkv_w4a8, w4a16_gemv_qkv_w4a8, "Q, K and V projections of one Q8_1 activation in one launch.",
        {"view"}, {"input_q8"}, {"input_scale"}, {"input_sum8"}, kStream, opt("in_features", kHidden), opt("num_q_heads", kQHeads),
        opt("num_kv_heads", kKvHeads), opt("head_dim", kHeadDim))
W4_SPEC(launch_gemv_dual_gate_up_swiglu_w4a16, w4a16_gemv_dual_gate_up_swiglu_w4a16,
        "SwiGLU of the interleaved gate / up rows, fp16 activation.",
        {"gate_up_qweight"}, {"gate_up_scales"}, {"input_x"}, {"output_mlp"}, {"hidden_size"}, {"intermediate_size"}, kStream)
W4_SPEC(launch_gemv_dual_gate_up_swiglu_w4a8, w4a16_gemv_dual_gate_up_swiglu_w4a8,
        "SwiGLU of the interleaved gate / up rows, Q8_1 activation.",
        {"gate_up_qweight"}, {"gate_up_scales"}, {"input_q8"}, {"input_scale"}, {"input_sum8"}, {"output_mlp"}, {"hidden_size"},
        {"intermediate_size"}, kStream)
W4_SPEC(launch_gemv_rmsnorm_w4a16, w4a16_gemv_rmsnorm_w4a16,
        "launch_rmsnorm_q8_1 + launch_gemv_w4a8 in one launch (gamma None: quantise only).",
        {"qweight"}, {"scales"}, {"input_x"}, {"gamma"}, {"residual"}, {"output_y"}, {"out_features"}, {"in_features"}, kStream)
W4_SPEC(launch_gemv_qkv_rmsnorm_w4a16, w4a16_gemv_qkv_rmsnorm_w4a16, "launch_rmsnorm_q8_1 + launch_gemv_qkv_w4a8 in one launch.",
        {"view"}, {"input_x"}, {"gamma"}, kStream, opt("in_features", kHidden), opt("num_q_heads", kQHeads),
        opt("num_kv_heads", kKvHeads), opt("head_dim", kHeadDim))
W4_SPEC(launch_gemv_dual_gate_up_swiglu_rmsnorm_w4a16, w4a16_gemv_dual_gate_up_swiglu_rmsnorm_w4a16,
        "launch_rmsnorm_q8_1 + launch_gemv_dual_gate_up_swiglu_w4a8 in one launch.",
        {"gate_up_qweight"}, {"gate_up_scales"}, {"input_x"}, {"gamma"}, {"output_mlp"}, {"hidden_size"}, {"intermediate_size"}, kStream)
W4_SPEC(launch_gemv_dual_gate_up_swiglu_rmsnorm_w4a16_q8_1, w4a16_gemv_dual_gate_up_swiglu_rmsnorm_w4a16_q8_1,
        "The launch above, which also leaves the Q8_1 form of output_mlp (the down projection's input).",
        {"gate_up_qweight"}, {"gate_up_scales"}, {"input_x"}, {"gamma"}, {"output_mlp"}, {"output_q8"}, {"output_scale"},
        {"output_sum8"}, {"hidden_size"}, {"intermediate_size"}, kStream)
W4_SPEC(launch_gemm_prefill_w4a16, w4a16_gemm_prefill_w4a16, "Y = X W^T (+ residual) for M tokens.",
        {"qweight"}, {"scales"}, {"input_x"}, {"residual"}, {"output_y"}, {"M"}, {"N"}, {"K"}, kStream, opt("sm_count", 0))
W4_SPEC(launch_gemm_prefill_qkv_w4a16, w4a16_gemm_prefill_qkv_w4a16, "Q, K and V projections of M tokens in one launch.",
        {"view"}, {"input_x"}, {"M"}, kStream, opt("in_features", kHidden), opt("num_q_heads", kQHeads),
        opt("num_kv_heads", kKvHeads), opt("head_dim", kHeadDim), opt("sm_count", 0))
W4_SPEC(launch_gemm_prefill_dual_gate_up_swiglu_w4a16, w4a16_gemm_prefill_dual_gate_up_swiglu_w4a16,
        "SwiGLU of the interleaved gate / up rows for M tokens.",
        {"gate_up_qweight"}, {"gate_up_scales"}, {"input_x"}, {"output_mlp"}, {"M"}, kStream, opt("hidden_size", kHidden),
        opt("intermediate_size", kInter))
W4_SPEC(gemv_group_dots, w4a16_gemv_group_dots,
        "Diagnostic: int32 per-group partial sums of the decode GEMV (no reference launcher).",
        {"qweight"}, {"input_q8"}, {"input_sum8"}, {"out_dots"}, {"out_features"}, {"in_features"}, kStream)

// sweep_run_device(handle, h_in, h_out, stream)
PyObject* sweep_run_device(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    if (nargs != 4) {
        PyErr_SetString(PyExc_TypeError, "sweep_run_device(handle, h_in, h_out, stream)");
        return nullptr;
    }
    void* h = PyLong_AsVoidPtr(args[0]);
    if (h == nullptr && PyErr_Occurred()) return nullptr;
    void *in = nullptr, *out = nullptr;
    w4a16_stream_t s = nullptr;
    if (!to_pointer(args[1], &in) || !to_pointer(args[2], &out) || !to_stream(args[3], &s)) return nullptr;
    int status;
    Py_BEGIN_ALLOW_THREADS
    status = w4a16_sweep_run_device(static_cast<w4a16_sweep*>(h), in, out, s);
    Py_END_ALLOW_THREADS
    return finish("w4a16_sweep_run_device", status);
}

PyMethodDef g_methods[] = {
    W4_ENTRY(launch_quantize_fp16_to_q8_1, w4a16_quantize_fp16_to_q8_1),
    W4_ENTRY(launch_rmsnorm_q8_1, w4a16_rmsnorm_q8_1),
    W4_ENTRY(quantize_attn_heads_f32_to_q8_1, w4a16_quantize_attn_heads_f32_to_q8_1),
    W4_ENTRY(gemv_attn_heads_f32_w4a16, w4a16_gemv_attn_heads_f32_w4a16),
    W4_ENTRY(launch_gemv_w4a16, w4a16_gemv_w4a16),
    W4_ENTRY(gemv_w4a16_static_scratch, w4a16_gemv_w4a16_static_scratch),
    W4_ENTRY(launch_gemv_w4a8, w4a16_gemv_w4a8),
    W4_ENTRY(launch_embed_lookup_w4a16, w4a16_embed_lookup_w4a16),
    W4_ENTRY(launch_sample_and_advance, w4a16_sample_and_advance),
    W4_ENTRY(launch_gemv_w4a8_sample_candidates, w4a16_gemv_w4a8_sample_candidates),
    W4_ENTRY(launch_gemv_w4a8_sample_one_launch, w4a16_gemv_w4a8_sample_one_launch),
    W4_ENTRY(launch_sample_finish, w4a16_sample_finish),
    W4_ENTRY(launch_gemv_w4a8_sample_and_advance, w4a16_gemv_w4a8_sample_and_advance),
    W4_ENTRY(launch_gemv_qkv_w4a8, w4a16_gemv_qkv_w4a8),
    W4_ENTRY(launch_gemv_dual_gate_up_swiglu_w4a16, w4a16_gemv_dual_gate_up_swiglu_w4a16),
    W4_ENTRY(launch_gemv_dual_gate_up_swiglu_w4a8, w4a16_gemv_dual_gate_up_swiglu_w4a8),
    W4_ENTRY(launch_gemv_rmsnorm_w4a16, w4a16_gemv_rmsnorm_w4a16),
    W4_ENTRY(launch_gemv_qkv_rmsnorm_w4a16, w4a16_gemv_qkv_rmsnorm_w4a16),
    W4_ENTRY(launch_gemv_dual_gate_up_swiglu_rmsnorm_w4a16, w4a16_gemv_dual_gate_up_swiglu_rmsnorm_w4a16),
    W4_ENTRY(launch_gemv_dual_gate_up_swiglu_rmsnorm_w4a16_q8_1, w4a16_gemv_dual_gate_up_swiglu_rmsnorm_w4a16_q8_1),
    W4_ENTRY(launch_gemm_prefill_w4a16, w4a16_gemm_prefill_w4a16),
    W4_ENTRY(launch_gemm_prefill_qkv_w4a16, w4a16_gemm_prefill_qkv_w4a16),
    W4_ENTRY(launch_gemm_prefill_dual_gate_up_swiglu_w4a16, w4a16_gemm_prefill_dual_gate_up_swiglu_w4a16),
    W4_ENTRY(gemv_group_dots, w4a16_gemv_group_dots),
    {"sweep_run_device", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&sweep_run_device)), METH_FASTCALL,
     "One pass of a decode sweep (handle of w4a16_sweep_create) on device buffers."},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "qwen_engine_b200._launch",
                        "Launch functions of libw4a16_b200.so on torch CUDA tensors [" W4_BUILT_FOR "].", -1, g_methods,
                        nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__launch(void) {
    PyObject* lib = PyImport_ImportModule("qwen_engine_b200._lib");
    if (lib == nullptr) return nullptr;
    g_check = PyObject_GetAttrString(lib, "check");
    Py_DECREF(lib);
    if (g_check == nullptr) return nullptr;
    g_str_cuda_stream = PyUnicode_InternFromString("cuda_stream");
    const char* names[9] = {"q_weight", "q_scale", "d_q", "k_weight", "k_scale", "d_k", "v_weight", "v_scale", "d_v"};
    for (int i = 0; i < 9; ++i) g_view_names[i] = PyUnicode_InternFromString(names[i]);
    return PyModule_Create(&g_module);
}
