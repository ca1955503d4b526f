// The torch front end's call path in native code: argument checks, output allocation, stream look-up and the C-ABI call of one
// operation, without the interpreter in between. A decode call's kernel runs 4-15 us; the same steps in Python (tensor
// attribute look-ups, torch.cuda.current_stream, ctypes argument conversion) took 17-20 us of the host per call, here about 4.
//
// The module calls the C ABI through addresses handed over by bind() (the library that kernel_library.py found and checked), so
// there is one place that decides which library is used. Anything out of the ordinary (a wrong type, shape or device) makes a
// function return None instead of launching: the Python caller then takes its own path, which raises the proper error.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ops/_to_copy.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>  // C++ exceptions become the Python ones torch raises itself (OutOfMemoryError among them)
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <initializer_list>

namespace {

using at::Tensor;
using c10::ScalarType;

enum { TYPE_Q8_0 = 8, TYPE_Q4_K = 12, TYPE_Q6_K = 14 };
enum { ELEM_F32 = 0, ELEM_F16 = 1, ELEM_BF16 = 2 };
constexpr int ERR_UNSUPPORTED = -1;
constexpr int MATRIX_ROW_PADDING = 512;  // activation rows of the two-launch protocol are padded to this many values

// ---- the C ABI (include/inferencequant_b200.h) ----
using GemvFn = int (*)(int, int, const void*, const void*, void*, int, int, int, int, int, int, void*);
using GroupFn = int (*)(int, const int*, const void* const*, void* const*, const int*, int, int, const void*, int, void*);
using GemmWsFn = int (*)(int, int, const void*, const void*, void*, int, int, int, int, int, void*, int64_t, void*);
using MmqWsFn = int (*)(int, int, const void*, const void*, void*, int, int, int, int, void*, int64_t, void*);
using GemmBytesFn = int64_t (*)(int, int, int, int);
using GemvTcFn = int (*)(int, int, const void*, const void*, void*, int, int, int, int, int, void*, int64_t, void*);
using GemvTcBytesFn = int64_t (*)(int, int);
using QuantizeFn = int (*)(int, const void*, void*, int64_t, void*);
using DequantizeFn = int (*)(int, int, const void*, void*, int64_t, int, void*);
using GetRowsFn = int (*)(int, int, const void*, const int32_t*, void*, int64_t, int, int64_t, void*);
using StatusFn = int (*)();
using QuantQ8Fn = void (*)(const void*, void*, int, int, int, void*);
using PlainFn = void (*)(const void*, const void*, void*, int, int, int, int, int, void*);
using GluFn = void (*)(const void*, const void*, const void*, void*, int, int, int, int, int, int, void*);
using QuantMmqFn = void (*)(const void*, const int32_t*, void*, int, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, void*);
using MmqFn = void (*)(void*, const void*, const void*, void*, int64_t, int64_t, int64_t, int64_t, int64_t, int, int, int64_t, int, int, void*);

// indexed by type (0 q8_0, 1 q4_k, 2 q6_k) and element type
struct Abi {
    GemvFn gemv;
    GroupFn group;
    GemmWsFn gemm_ws;
    GemmBytesFn gemm_bytes, mmq_bytes;
    MmqWsFn mmq_ws;
    GemvTcFn gemv_tc;
    GemvTcBytesFn gemv_tc_bytes;
    QuantizeFn quantize;
    DequantizeFn dequantize;
    GetRowsFn get_rows;
    StatusFn take_status;
    QuantQ8Fn quant_q8[3];
    PlainFn plain[3][3];
    GluFn glu[3][3];
    QuantMmqFn quant_mmq[2];  // D4, DS4
    MmqFn mmq[3];
} abi{};
PyObject* check_fn = nullptr;          // kernel_library.check(rc, what): raises for a non-zero status
PyObject* launch_failed_fn = nullptr;  // raises for a status kept by a void launcher

struct AbiEntry {
    const char* name;
    void** slot;
};
const AbiEntry abi_entries[] = {
    {"b200q_gemv", (void**)&abi.gemv},
    {"b200q_gemv_group_act", (void**)&abi.group},
    {"b200q_gemm_ws", (void**)&abi.gemm_ws},
    {"b200q_mmq_ws", (void**)&abi.mmq_ws},
    {"b200q_mmq_workspace_bytes", (void**)&abi.mmq_bytes},
    {"b200q_gemm_workspace_bytes", (void**)&abi.gemm_bytes},
    {"b200q_gemv_tc", (void**)&abi.gemv_tc},
    {"b200q_gemv_tc_workspace_bytes", (void**)&abi.gemv_tc_bytes},
    {"b200q_quantize", (void**)&abi.quantize},
    {"b200q_dequantize", (void**)&abi.dequantize},
    {"b200q_get_rows", (void**)&abi.get_rows},
    {"b200q_take_launch_status", (void**)&abi.take_status},
    {"launch_mmvq_gguf_quantize_q8_1_f32", (void**)&abi.quant_q8[ELEM_F32]},
    {"launch_mmvq_gguf_quantize_q8_1_f16", (void**)&abi.quant_q8[ELEM_F16]},
    {"launch_mmvq_gguf_quantize_q8_1_bf16", (void**)&abi.quant_q8[ELEM_BF16]},
#define B200Q_HOST_TYPE(i, tag)                                              \
    {"launch_mmvq_gguf_" tag "_f32_plain", (void**)&abi.plain[i][ELEM_F32]},     \
    {"launch_mmvq_gguf_" tag "_f16_plain", (void**)&abi.plain[i][ELEM_F16]},     \
    {"launch_mmvq_gguf_" tag "_bf16_plain", (void**)&abi.plain[i][ELEM_BF16]},   \
    {"launch_mmvq_gguf_" tag "_f32_fused_glu", (void**)&abi.glu[i][ELEM_F32]},   \
    {"launch_mmvq_gguf_" tag "_f16_fused_glu", (void**)&abi.glu[i][ELEM_F16]},   \
    {"launch_mmvq_gguf_" tag "_bf16_fused_glu", (void**)&abi.glu[i][ELEM_BF16]}, \
    {"launch_mmq_gguf_" tag, (void**)&abi.mmq[i]},
    B200Q_HOST_TYPE(0, "q8_0") B200Q_HOST_TYPE(1, "q4_k") B200Q_HOST_TYPE(2, "q6_k")
#undef B200Q_HOST_TYPE
    {"launch_mmq_quantize_q8_1_D4", (void**)&abi.quant_mmq[0]},
    {"launch_mmq_quantize_q8_1_DS4", (void**)&abi.quant_mmq[1]},
};

int type_index(long type) { return type == TYPE_Q8_0 ? 0 : (type == TYPE_Q4_K ? 1 : (type == TYPE_Q6_K ? 2 : -1)); }
int64_t block_elems(int ti) { return ti == 0 ? 32 : 256; }
int64_t block_bytes(int ti) { return ti == 0 ? 34 : (ti == 1 ? 144 : 210); }
int elem_of(ScalarType t) {
    return t == ScalarType::Float ? ELEM_F32 : (t == ScalarType::Half ? ELEM_F16 : (t == ScalarType::BFloat16 ? ELEM_BF16 : -1));
}
int mmq_type_x(int elem) { return elem == ELEM_F32 ? 0 : (elem == ELEM_F16 ? 1 : 30); }
int64_t pad(int64_t k, int64_t to) { return (k + to - 1) / to * to; }

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// ---- arguments ----
const Tensor* tensor_arg(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }
bool cuda_contiguous(const Tensor* t) { return t != nullptr && t->is_cuda() && t->is_contiguous(); }
// anything that counts as an integer (a numpy integer has an index too)
bool int_arg(PyObject* o, long& v) {
    PyObject* i = PyNumber_Index(o);
    if (i != nullptr) {
        v = PyLong_AsLong(i);
        Py_DECREF(i);
    }
    if (i != nullptr && !(v == -1 && PyErr_Occurred())) return true;
    PyErr_Clear();
    return false;
}
bool int_args(PyObject* const* args, std::initializer_list<std::pair<int, long*>> list) {
    for (const auto& [i, v] : list)
        if (!int_arg(args[i], *v)) return false;
    return true;
}
Tensor empty(at::IntArrayRef size, ScalarType t, const Tensor& like) { return at::detail::empty_cuda(size, t, like.device(), std::nullopt); }
PyObject* none() { Py_RETURN_NONE; }
// launches may block (a full queue, a first load of a kernel): other Python threads go on meanwhile
struct NoGil {
    PyThreadState* state = PyEval_SaveThread();
    ~NoGil() { PyEval_RestoreThread(state); }
};
template <typename Fn, typename... Args> auto call(Fn fn, Args... args) {
    NoGil nogil;
    return fn(args...);
}

// 0: fine; otherwise a Python exception is set (kernel_library.check raises)
int failed(int rc, const char* what) {
    if (rc == 0) return 0;
    PyObject* r = PyObject_CallFunction(check_fn, "is", rc, what);
    Py_XDECREF(r);
    return 1;
}
int launcher_failed(const char* what) {
    const int rc = abi.take_status();
    if (rc == 0) return 0;
    PyObject* r = PyObject_CallFunction(launch_failed_fn, "is", rc, what);
    Py_XDECREF(r);
    return 1;
}

// ---- matmul ----
// quantize to Q8_1, then the reference's own matvec: shapes the one-launch kernel declines
int two_launches(int ti, int elem, const Tensor& w, const Tensor& x, Tensor& y, int64_t n, int64_t k, int64_t rows) {
    const int64_t kp = pad(k, MATRIX_ROW_PADDING);
    Tensor vy = empty({rows, kp / 32 * 36}, ScalarType::Byte, x);
    call(abi.quant_q8[elem], x.data_ptr(), vy.data_ptr(), (int)k, (int)kp, (int)rows, stream());
    call(abi.plain[ti][elem], w.data_ptr(), vy.data_ptr(), y.data_ptr(), (int)k, (int)n, (int)(kp / 32), (int)n, (int)rows, stream());
    return launcher_failed("launch_mmvq_gguf_*_plain");
}

// A workspace from the caching allocator for the duration of a call (given back in stream order); undefined if none is needed or the
// memory is not there, where the caller has a form that needs none.
Tensor workspace(int64_t bytes, const Tensor& like) {
    if (bytes <= 0) return Tensor();
    try {
        return empty({bytes}, ScalarType::Byte, like);
    } catch (const c10::OutOfMemoryError&) {
        return Tensor();
    }
}

// the tile GEMM
int gemm(long type, int elem, const Tensor& w, const Tensor& x, Tensor& y, int64_t m, int64_t n, int64_t k, int64_t ldx, int64_t ldy) {
    const int64_t bytes = abi.gemm_bytes((int)type, (int)m, (int)n, (int)k);
    const Tensor ws = workspace(bytes, x);
    return call(abi.gemm_ws, (int)type, elem, w.data_ptr(), x.data_ptr(), y.data_ptr(), (int)m, (int)n, (int)k, (int)ldx, (int)ldy,
                ws.defined() ? ws.data_ptr() : nullptr, bytes, stream());
}

// forward(type, w, n, k, x, act_quant, tier): y = x . W^T for contiguous x [..., k]; `tier` is what the caller's routing chose for
// the row count: 0 decode matvec, 1 small-batch tensor-core kernel, 2 tile GEMM, 3 as 1 or, where that refuses the weights or finds no room for its workspace, as 0
PyObject* py_forward(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    long type, n, k, act_quant, tier;
    if (nargs != 7 || !int_args(args, {{0, &type}, {2, &n}, {3, &k}, {5, &act_quant}, {6, &tier}})) return none();
    const Tensor *w = tensor_arg(args[1]), *x = tensor_arg(args[4]);
    const int ti = type_index(type);
    if (ti < 0 || !cuda_contiguous(w) || !cuda_contiguous(x) || x->dim() < 2 || x->size(-1) != k || x->device() != w->device()) return none();
    const int elem = elem_of(x->scalar_type());
    if (elem < 0) return none();
    const int64_t rows = x->numel() / k;
    if (rows == 0) return none();
    c10::SmallVector<int64_t, 6> shape(x->sizes().begin(), x->sizes().end());
    shape.back() = n;
    if (tier == 2) {
        if (k % 64 != 0) return none();
        // the tensor-core path takes 16-bit activations; f32 inputs are narrowed and the result widened again
        const Tensor x16 = elem == ELEM_F32 ? at::_to_copy(*x, ScalarType::BFloat16) : *x;
        Tensor y = empty(shape, x16.scalar_type(), *x);
        if (failed(gemm(type, elem == ELEM_F32 ? ELEM_BF16 : elem, *w, x16, y, rows, n, k, k, n), "b200q_gemm"))
            return nullptr;
        return THPVariable_Wrap(elem == ELEM_F32 ? at::_to_copy(y, ScalarType::Float) : y);
    }
    Tensor y = empty(shape, x->scalar_type(), *x);
    if (tier == 1 || tier == 3) {
        const int64_t bytes = abi.gemv_tc_bytes((int)type, (int)k);
        if (bytes <= 0) return none();
        const Tensor ws = tier == 1 ? empty({bytes}, ScalarType::Byte, *x) : workspace(bytes, *x);
        const int rc = !ws.defined() ? ERR_UNSUPPORTED
                                     : call(abi.gemv_tc, (int)type, elem, w->data_ptr(), x->data_ptr(), y.data_ptr(), (int)rows, (int)n, (int)k, (int)k, (int)n,
                                            ws.data_ptr(), bytes, stream());
        if (rc != ERR_UNSUPPORTED || tier == 1) return failed(rc, "b200q_gemv_tc") ? nullptr : THPVariable_Wrap(std::move(y));
    }
    if (k % 128 == 0) {
        const int rc = call(abi.gemv, (int)type, elem, w->data_ptr(), x->data_ptr(), y.data_ptr(), (int)k, (int)n, (int)k, (int)n, (int)rows, (int)act_quant, stream());
        // no staged plan for this call (unaligned weights, no ring that fits): the two-launch protocol serves Q8_1 activations
        if (rc != ERR_UNSUPPORTED || act_quant != 0) return failed(rc, "b200q_gemv") ? nullptr : THPVariable_Wrap(std::move(y));
    } else if (act_quant != 0) {
        return none();
    }
    return two_launches(ti, elem, *w, *x, y, n, k, rows) ? nullptr : THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

// gemv(type, w, x, n, out or None, act_quant)
PyObject* py_gemv(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    long type, n, act_quant;
    if (nargs != 6 || !int_args(args, {{0, &type}, {3, &n}, {5, &act_quant}})) return none();
    const Tensor *w = tensor_arg(args[1]), *x = tensor_arg(args[2]), *out = args[4] == Py_None ? nullptr : tensor_arg(args[4]);
    if (!cuda_contiguous(w) || !cuda_contiguous(x) || x->dim() != 2 || (args[4] != Py_None && (out == nullptr || out->dim() != 2))) return none();
    const int elem = elem_of(x->scalar_type());
    if (elem < 0) return none();
    const int64_t b = x->size(0), k = x->size(1);
    Tensor y = out != nullptr ? *out : empty({b, n}, x->scalar_type(), *x);
    if (failed(call(abi.gemv, (int)type, elem, w->data_ptr(), x->data_ptr(), y.data_ptr(), (int)k, (int)n, (int)x->stride(0), (int)y.stride(0), (int)b, (int)act_quant,
                        stream()),
               "b200q_gemv"))
        return nullptr;
    return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

// gemm(type, w, x, n, out or None)
PyObject* py_gemm(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    long type, n;
    if (nargs != 5 || !int_args(args, {{0, &type}, {3, &n}})) return none();
    const Tensor *w = tensor_arg(args[1]), *x = tensor_arg(args[2]), *out = args[4] == Py_None ? nullptr : tensor_arg(args[4]);
    if (!cuda_contiguous(w) || !cuda_contiguous(x) || x->dim() != 2 || (args[4] != Py_None && (out == nullptr || out->dim() != 2))) return none();
    const int elem = elem_of(x->scalar_type());
    if (elem < 0) return none();
    Tensor y = out != nullptr ? *out : empty({x->size(0), n}, x->scalar_type(), *x);
    if (failed(gemm(type, elem, *w, *x, y, x->size(0), n, x->size(1), x->stride(0), y.stride(0)), "b200q_gemm")) return nullptr;
    return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

// gemv_group(types, ws, x, ns, outs or None, act_quant): lists of 1..4
PyObject* py_gemv_group(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    constexpr int MAX = 4;
    long act_quant;
    if (nargs != 6 || !int_arg(args[5], act_quant)) return none();
    for (int i : {0, 1, 3})
        if (!PyList_Check(args[i]) && !PyTuple_Check(args[i])) return none();
    const Tensor* x = tensor_arg(args[2]);
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(args[1]);
    const bool have_outs = args[4] != Py_None;
    if (n < 1 || n > MAX || PySequence_Fast_GET_SIZE(args[0]) != n || PySequence_Fast_GET_SIZE(args[3]) != n || !cuda_contiguous(x) || x->dim() != 2 ||
        x->size(0) != 1 || (have_outs && ((!PyList_Check(args[4]) && !PyTuple_Check(args[4])) || PySequence_Fast_GET_SIZE(args[4]) != n)))
        return none();
    const int elem = elem_of(x->scalar_type());
    if (elem < 0) return none();
    int types[MAX], ns[MAX];
    const void* ws[MAX];
    void* dsts[MAX];
    Tensor outs[MAX];
    for (Py_ssize_t i = 0; i < n; ++i) {
        long t, rows;
        if (!int_arg(PySequence_Fast_GET_ITEM(args[0], i), t) || !int_arg(PySequence_Fast_GET_ITEM(args[3], i), rows)) return none();
        const Tensor* w = tensor_arg(PySequence_Fast_GET_ITEM(args[1], i));
        if (!cuda_contiguous(w)) return none();
        types[i] = (int)t;
        ns[i] = (int)rows;
        ws[i] = w->data_ptr();
        if (have_outs) {
            const Tensor* o = tensor_arg(PySequence_Fast_GET_ITEM(args[4], i));
            if (o == nullptr) return none();
            dsts[i] = o->data_ptr();
        }
    }
    if (!have_outs)
        for (Py_ssize_t i = 0; i < n; ++i) {
            outs[i] = empty({1, (int64_t)ns[i]}, x->scalar_type(), *x);
            dsts[i] = outs[i].data_ptr();
        }
    const int rc = call(abi.group, (int)n, types, ws, dsts, ns, (int)x->size(1), elem, x->data_ptr(), (int)act_quant, stream());
    if (failed(rc, act_quant ? "b200q_gemv_group_act" : "b200q_gemv_group")) return nullptr;
    if (have_outs) {
        Py_INCREF(args[4]);
        return args[4];
    }
    PyObject* list = PyList_New(n);
    for (Py_ssize_t i = 0; list != nullptr && i < n; ++i) PyList_SET_ITEM(list, i, THPVariable_Wrap(std::move(outs[i])));
    return list;
    END_HANDLE_TH_ERRORS
}

// ---- the reference host's own sequence ----
// quantize_q8_1(x, k_padded)
PyObject* py_quantize_q8_1(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    long kp;
    if (nargs != 2 || !int_arg(args[1], kp)) return none();
    const Tensor* x = tensor_arg(args[0]);
    if (!cuda_contiguous(x) || x->dim() != 2 || elem_of(x->scalar_type()) < 0) return none();
    Tensor out = empty({x->size(0), kp / 32 * 36}, ScalarType::Byte, *x);
    call(abi.quant_q8[elem_of(x->scalar_type())], x->data_ptr(), out.data_ptr(), (int)x->size(1), (int)kp, (int)x->size(0), stream());
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// elem code of an output type given as its code
bool elem_scalar(long elem, ScalarType& t) {
    if (elem < 0 || elem > 2) return false;
    t = elem == ELEM_F32 ? ScalarType::Float : (elem == ELEM_F16 ? ScalarType::Half : ScalarType::BFloat16);
    return true;
}

// mmvq_plain(type, w, vy, n, k, b, elem, k_padded)
PyObject* py_mmvq_plain(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    long type, n, k, b, elem, kp;
    ScalarType t;
    if (nargs != 8 || !int_args(args, {{0, &type}, {3, &n}, {4, &k}, {5, &b}, {6, &elem}, {7, &kp}}) || !elem_scalar(elem, t)) return none();
    const Tensor *w = tensor_arg(args[1]), *vy = tensor_arg(args[2]);
    const int ti = type_index(type);
    if (ti < 0 || !cuda_contiguous(w) || !cuda_contiguous(vy)) return none();
    Tensor y = empty({b, n}, t, *w);
    call(abi.plain[ti][elem], w->data_ptr(), vy->data_ptr(), y.data_ptr(), (int)k, (int)n, (int)(kp / 32), (int)n, (int)b, stream());
    return launcher_failed("launch_mmvq_gguf_*_plain") ? nullptr : THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

// mmvq_fused_glu(type, w_gate, w_up, vy, n, k, b, elem, k_padded, activation)
PyObject* py_mmvq_fused_glu(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    long type, n, k, b, elem, kp, act;
    ScalarType t;
    if (nargs != 10 || !int_args(args, {{0, &type}, {4, &n}, {5, &k}, {6, &b}, {7, &elem}, {8, &kp}, {9, &act}}) || !elem_scalar(elem, t)) return none();
    const Tensor *wg = tensor_arg(args[1]), *wu = tensor_arg(args[2]), *vy = tensor_arg(args[3]);
    const int ti = type_index(type);
    if (ti < 0 || !cuda_contiguous(wg) || !cuda_contiguous(wu) || !cuda_contiguous(vy)) return none();
    Tensor y = empty({b, n}, t, *vy);
    call(abi.glu[ti][elem], wg->data_ptr(), wu->data_ptr(), vy->data_ptr(), y.data_ptr(), (int)k, (int)n, (int)(kp / 32), (int)n, (int)b, (int)act, stream());
    return launcher_failed("launch_mmvq_gguf_*_fused_glu") ? nullptr : THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

// quantize_mmq_q8_1(x, ds4, k_padded)
PyObject* py_quantize_mmq_q8_1(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    long ds4, kp;
    if (nargs != 3 || !int_args(args, {{1, &ds4}, {2, &kp}})) return none();
    const Tensor* x = tensor_arg(args[0]);
    if (!cuda_contiguous(x) || x->dim() != 2 || elem_of(x->scalar_type()) < 0) return none();
    const int64_t rows = x->size(0), k = x->size(1);
    Tensor out = empty({kp / 128, rows, 144}, ScalarType::Byte, *x);
    call(abi.quant_mmq[ds4 ? 1 : 0], x->data_ptr(), nullptr, out.data_ptr(), mmq_type_x(elem_of(x->scalar_type())), k, k, 0, 0, kp, rows, 1, 1, stream());
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// mmq(type, w, vy, m, n, k, elem, cc, nsm)
PyObject* py_mmq(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    long type, m, n, k, elem, cc, nsm;
    ScalarType t;
    if (nargs != 9 || !int_args(args, {{0, &type}, {3, &m}, {4, &n}, {5, &k}, {6, &elem}, {7, &cc}, {8, &nsm}}) || !elem_scalar(elem, t)) return none();
    const Tensor *w = tensor_arg(args[1]), *vy = tensor_arg(args[2]);
    const int ti = type_index(type);
    if (ti < 0 || !cuda_contiguous(w) || !cuda_contiguous(vy)) return none();
    Tensor y = empty({m, n}, t, *w);
    const int64_t bytes = abi.mmq_bytes((int)type, (int)m, (int)n, (int)k);
    if (const Tensor ws = workspace(bytes, *w); ws.defined()) {
        const int rc = call(abi.mmq_ws, (int)type, (int)elem, w->data_ptr(), vy->data_ptr(), y.data_ptr(), (int)m, (int)n, (int)k, (int)n, ws.data_ptr(), bytes,
                            stream());
        if (rc != ERR_UNSUPPORTED) return failed(rc, "b200q_mmq_ws") ? nullptr : THPVariable_Wrap(std::move(y));
    }
    call(abi.mmq[ti], nullptr, w->data_ptr(), vy->data_ptr(), y.data_ptr(), k, n, m, k / block_elems(ti), n, (int)cc, (int)nsm, 232448, 32, mmq_type_x((int)elem),
                stream());
    return launcher_failed("launch_mmq_gguf_*") ? nullptr : THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

// ---- weights ----
// quantize(type, x): f32 [n, k] -> packed blocks, then the padding, zeroed
PyObject* py_quantize(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    long type;
    if (nargs != 2 || !int_arg(args[0], type)) return none();
    const Tensor* x = tensor_arg(args[1]);
    const int ti = type_index(type);
    if (ti < 0 || !cuda_contiguous(x) || x->dim() != 2 || x->scalar_type() != ScalarType::Float || x->size(1) % block_elems(ti) != 0) return none();
    const int64_t bytes = x->numel() / block_elems(ti) * block_bytes(ti), padding = MATRIX_ROW_PADDING / block_elems(ti) * block_bytes(ti);
    Tensor buf = empty({bytes + padding}, ScalarType::Byte, *x);
    buf.narrow(0, bytes, padding).zero_();
    if (failed(call(abi.quantize, (int)type, x->data_ptr(), buf.data_ptr(), x->numel(), stream()), "b200q_quantize")) return nullptr;
    return THPVariable_Wrap(std::move(buf));
    END_HANDLE_TH_ERRORS
}

// dequantize(type, w, n, k, elem)
PyObject* py_dequantize(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    long type, n, k, elem;
    ScalarType t;
    if (nargs != 5 || !int_args(args, {{0, &type}, {2, &n}, {3, &k}, {4, &elem}}) || !elem_scalar(elem, t)) return none();
    const Tensor* w = tensor_arg(args[1]);
    if (!cuda_contiguous(w)) return none();
    Tensor out = empty({n, k}, t, *w);
    if (failed(call(abi.dequantize, (int)type, (int)elem, w->data_ptr(), out.data_ptr(), n, (int)k, stream()), "b200q_dequantize")) return nullptr;
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// get_rows(type, w, ids, n, k, elem): ids int32, contiguous, on the device
PyObject* py_get_rows(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    long type, n, k, elem;
    ScalarType t;
    if (nargs != 6 || !int_args(args, {{0, &type}, {3, &n}, {4, &k}, {5, &elem}}) || !elem_scalar(elem, t)) return none();
    const Tensor *w = tensor_arg(args[1]), *ids = tensor_arg(args[2]);
    if (!cuda_contiguous(w) || !cuda_contiguous(ids) || ids->scalar_type() != ScalarType::Int || ids->device() != w->device()) return none();
    c10::SmallVector<int64_t, 6> shape(ids->sizes().begin(), ids->sizes().end());
    shape.push_back(k);
    Tensor out = empty(shape, t, *w);
    if (failed(call(abi.get_rows, (int)type, (int)elem, w->data_ptr(), static_cast<const int32_t*>(ids->data_ptr()), out.data_ptr(), ids->numel(), (int)k, n, stream()),
               "b200q_get_rows"))
        return nullptr;
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// bind(names, addresses, check, launch_failed)
PyObject* py_bind(PyObject*, PyObject* args) {
    PyObject *addresses, *check, *launch_failed;
    if (!PyArg_ParseTuple(args, "O!OO", &PyDict_Type, &addresses, &check, &launch_failed)) return nullptr;
    for (const AbiEntry& e : abi_entries) {
        PyObject* v = PyDict_GetItemString(addresses, e.name);
        if (v == nullptr) return PyErr_Format(PyExc_KeyError, "no address for %s", e.name);
        *e.slot = PyLong_AsVoidPtr(v);
        if (PyErr_Occurred()) return nullptr;
    }
    Py_INCREF(check);
    Py_INCREF(launch_failed);
    Py_XSETREF(check_fn, check);
    Py_XSETREF(launch_failed_fn, launch_failed);
    Py_RETURN_NONE;
}

PyObject* py_symbols(PyObject*, PyObject*) {
    PyObject* list = PyList_New(0);
    for (const AbiEntry& e : abi_entries) {
        PyObject* s = PyUnicode_FromString(e.name);
        if (list == nullptr || s == nullptr || PyList_Append(list, s) != 0) return nullptr;
        Py_DECREF(s);
    }
    return list;
}

#define B200Q_FAST(name, fn) {name, (PyCFunction)(void (*)(void))fn, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"bind", py_bind, METH_VARARGS, nullptr},
    {"symbols", py_symbols, METH_NOARGS, nullptr},
    B200Q_FAST("forward", py_forward),
    B200Q_FAST("gemv", py_gemv),
    B200Q_FAST("gemv_group", py_gemv_group),
    B200Q_FAST("gemm", py_gemm),
    B200Q_FAST("quantize_q8_1", py_quantize_q8_1),
    B200Q_FAST("mmvq_plain", py_mmvq_plain),
    B200Q_FAST("mmvq_fused_glu", py_mmvq_fused_glu),
    B200Q_FAST("quantize_mmq_q8_1", py_quantize_mmq_q8_1),
    B200Q_FAST("mmq", py_mmq),
    B200Q_FAST("quantize", py_quantize),
    B200Q_FAST("dequantize", py_dequantize),
    B200Q_FAST("get_rows", py_get_rows),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "b200q_torch_host", "Native call path of the torch front end.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_b200q_torch_host(void) { return PyModule_Create(&module_def); }
