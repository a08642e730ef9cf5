// CPython binding of the rfk.h operators that take device tensors: tensors, integers and floats in, C ABI call on torch's
// current stream out.
//
// Most operators last 3 to 15 us on the device, and a call through ctypes (argument checks in Python, one foreign-function
// conversion per argument, the stream looked up through Python objects) took 6 to 8 us, so a run of them was bound by the
// host: 45 us for the six operators of a view's front end at any size. Here the conversions are generated from the C
// prototypes: a call with seven arguments costs about 0.4 us plus the launch itself.
//
// The binding has no argument errors of its own: whatever it does not recognise at once (a keyword, a wrong dtype, a CPU
// tensor, an integer type that is not Python's) goes to the Python function it was made for, which checks every argument
// and raises or calls.
#include <Python.h>
#include <structmember.h>

#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <climits>
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <tuple>
#include <type_traits>
#include <utility>

#include "rfk.h"

namespace {

// the dtypes a C pointer type stands for: uint8_t is a byte mask (bool or uint8), void a byte buffer
template <class T> bool takes(at::ScalarType t) {
    if constexpr (std::is_same_v<T, rfk_half>) return t == at::kHalf;
    else if constexpr (std::is_same_v<T, float>) return t == at::kFloat;
    else if constexpr (std::is_same_v<T, uint8_t>) return t == at::kByte || t == at::kBool;
    else if constexpr (std::is_same_v<T, void>) return t == at::kByte;
    else return false;
}

template <class T> bool convert(PyObject* o, T& v) {
    if constexpr (std::is_pointer_v<T>) {
        if (o == Py_None) { v = nullptr; return true; }
        if (!THPVariable_Check(o)) return false;
        const at::Tensor& t = THPVariable_Unpack(o);
        if (!t.is_cuda() || !takes<std::remove_cv_t<std::remove_pointer_t<T>>>(t.scalar_type()) || !t.is_contiguous()) return false;
        v = static_cast<T>(t.data_ptr());
        return true;
    } else if constexpr (std::is_floating_point_v<T>) {
        if (PyFloat_Check(o)) v = static_cast<T>(PyFloat_AS_DOUBLE(o));
        else if (PyLong_CheckExact(o)) {
            const double x = PyLong_AsDouble(o);
            if (x == -1.0 && PyErr_Occurred()) { PyErr_Clear(); return false; }
            v = static_cast<T>(x);
        } else return false;
        return true;
    } else {
        if (!PyLong_Check(o)) return false;
        int overflow = 0;
        const long long x = PyLong_AsLongLongAndOverflow(o, &overflow);
        if (overflow || (sizeof(T) == sizeof(int) && (x < INT_MIN || x > INT_MAX))) return false;
        v = static_cast<T>(x);
        return true;
    }
}

// Converts the arguments and calls; false (nothing called) when one of them is not taken.
using Invoke = bool (*)(PyObject* const* args, int* status);

template <auto Fn> struct Bound;
template <class... A, int (*Fn)(A...)> struct Bound<Fn> {
    static constexpr size_t kArgs = sizeof...(A) - 1;  // all but the stream
    using Values = std::tuple<A...>;
    template <size_t... I> static bool invoke_(PyObject* const* args, int* status, std::index_sequence<I...>) {
        Values v{};
        if (!(convert(args[I], std::get<I>(v)) && ...)) return false;
        const auto stream = static_cast<rfk_stream_t>(c10::cuda::getCurrentCUDAStream().stream());
        Py_BEGIN_ALLOW_THREADS
        *status = Fn(std::get<I>(v)..., stream);
        Py_END_ALLOW_THREADS
        return true;
    }
    static bool invoke(PyObject* const* args, int* status) {
        try {
            return invoke_(args, status, std::make_index_sequence<kArgs>{});
        } catch (...) {  // torch refused before the call was made (no device, a tensor without storage): not taken
            return false;
        }
    }
};

struct Entry { const char* name; Invoke invoke; size_t nargs; };
#define RFK_OP(fn) {#fn, Bound<fn>::invoke, Bound<fn>::kArgs}
const Entry kEntries[] = {
    RFK_OP(rfk_rmsnorm), RFK_OP(rfk_rmsnorm_f32), RFK_OP(rfk_rmsnorm_residual_f32_cast16),
    RFK_OP(rfk_rmsnorm_residual_mixed_cast16), RFK_OP(rfk_rmsnorm_residual_f16), RFK_OP(rfk_rmsnorm_residual_f16_windows),
    RFK_OP(rfk_residual_add), RFK_OP(rfk_residual_add_f32), RFK_OP(rfk_residual_add_mixed),
    RFK_OP(rfk_cast_fp32_to_fp16), RFK_OP(rfk_cast_fp16_to_fp32), RFK_OP(rfk_broadcast_add),
    RFK_OP(rfk_triangle_rope_freqs), RFK_OP(rfk_apply_rope), RFK_OP(rfk_apply_rope_one), RFK_OP(rfk_apply_rope_f32),
    RFK_OP(rfk_apply_rope_one_f32), RFK_OP(rfk_transpose_bshd_to_bhsd), RFK_OP(rfk_transpose_bhsd_to_bsd),
    RFK_OP(rfk_nerf_pe), RFK_OP(rfk_nerf_pe_f32),
    RFK_OP(rfk_softmax_inplace), RFK_OP(rfk_masked_softmax_inplace), RFK_OP(rfk_swin_masked_softmax_inplace),
    RFK_OP(rfk_softmax_cast_fp16), RFK_OP(rfk_softmax_cast_fp16_masked), RFK_OP(rfk_softmax_cast_fp16_scaled),
    RFK_OP(rfk_softmax_probs_inplace), RFK_OP(rfk_swin_softmax_probs_inplace), RFK_OP(rfk_swin_softmax_cast_fp16),
    RFK_OP(rfk_fused_silu_mul), RFK_OP(rfk_fused_silu_mul_f32), RFK_OP(rfk_swiglu), RFK_OP(rfk_swiglu_inplace),
    RFK_OP(rfk_elu), RFK_OP(rfk_pow10_minus1), RFK_OP(rfk_bilinear_upsample), RFK_OP(rfk_silu_inplace),
    RFK_OP(rfk_add_bias_nchw), RFK_OP(rfk_permute_bsd_to_nchw), RFK_OP(rfk_bias_act_residual_nhwc), RFK_OP(rfk_silu),
    RFK_OP(rfk_bilinear_upsample_nhwc), RFK_OP(rfk_depth_to_space_bias_nhwc), RFK_OP(rfk_permute_nhwc_to_nchw),
    RFK_OP(rfk_pointwise_conv_to_planar), RFK_OP(rfk_permute_filter), RFK_OP(rfk_post_elu_pow10),
    RFK_OP(rfk_ray_gen), RFK_OP(rfk_ray_gen_patchify), RFK_OP(rfk_patchify), RFK_OP(rfk_world_to_cam),
    RFK_OP(rfk_world_to_cam_f32), RFK_OP(rfk_view_geometry), RFK_OP(rfk_window_gather), RFK_OP(rfk_window_scatter),
};

// One bound operator: callable(args...) -> None; `checked` is the Python function behind it, `failed(symbol, status)` is
// called for a non-zero status.
constexpr size_t kMaxArgs = 24;
struct Op {
    PyObject_HEAD
    vectorcallfunc vectorcall;
    PyObject* dict;
    const Entry* entry;
    PyObject *checked, *failed, *defaults;  // defaults: tuple of the trailing parameters' defaults
};

PyObject* op_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
    Op* op = reinterpret_cast<Op*>(self);
    const size_t n = PyVectorcall_NARGS(nargsf), want = op->entry->nargs, nd = (size_t)PyTuple_GET_SIZE(op->defaults);
    if (!kwnames && n <= want && n + nd >= want) {
        PyObject* filled[kMaxArgs];
        PyObject* const* a = args;
        if (n < want) {
            std::memcpy(filled, args, n * sizeof(PyObject*));
            for (size_t i = n; i < want; ++i) filled[i] = PyTuple_GET_ITEM(op->defaults, nd - (want - i));
            a = filled;
        }
        int status = 0;
        if (op->entry->invoke(a, &status)) {
            if (status == RFK_OK) Py_RETURN_NONE;
            return PyObject_CallFunction(op->failed, "si", op->entry->name, status);
        }
    }
    return PyObject_Vectorcall(op->checked, args, nargsf, kwnames);
}

int op_traverse(PyObject* self, visitproc visit, void* arg) {
    Op* op = reinterpret_cast<Op*>(self);
    Py_VISIT(op->dict); Py_VISIT(op->checked); Py_VISIT(op->failed); Py_VISIT(op->defaults);
    return 0;
}
int op_clear(PyObject* self) {
    Op* op = reinterpret_cast<Op*>(self);
    Py_CLEAR(op->dict); Py_CLEAR(op->checked); Py_CLEAR(op->failed); Py_CLEAR(op->defaults);
    return 0;
}
void op_dealloc(PyObject* self) {
    PyObject_GC_UnTrack(self);
    op_clear(self);
    Py_TYPE(self)->tp_free(self);
}

// An operator is copied and pickled as the module's function that it stands for: by name.
PyObject* op_reduce(PyObject* self, PyObject*) { return PyObject_GetAttrString(self, "__qualname__"); }

PyMethodDef op_methods[] = {{"__reduce__", op_reduce, METH_NOARGS, "the operator's name in its module"},
                            {nullptr, nullptr, 0, nullptr}};
PyMemberDef op_members[] = {
    {"__dictoffset__", T_PYSSIZET, offsetof(Op, dict), READONLY, nullptr},
    {"__vectorcalloffset__", T_PYSSIZET, offsetof(Op, vectorcall), READONLY, nullptr},
    {nullptr, 0, 0, 0, nullptr}};
PyGetSetDef op_getset[] = {{"__dict__", PyObject_GenericGetDict, PyObject_GenericSetDict, nullptr, nullptr},
                           {nullptr, nullptr, nullptr, nullptr, nullptr}};
PyType_Slot op_slots[] = {
    {Py_tp_dealloc, reinterpret_cast<void*>(op_dealloc)}, {Py_tp_traverse, reinterpret_cast<void*>(op_traverse)},
    {Py_tp_clear, reinterpret_cast<void*>(op_clear)},     {Py_tp_call, reinterpret_cast<void*>(PyVectorcall_Call)},
    {Py_tp_members, op_members},                          {Py_tp_getset, op_getset},
    {Py_tp_methods, op_methods},                          {0, nullptr}};
PyType_Spec op_spec = {"rfk.Op", sizeof(Op), 0,
                       Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC | Py_TPFLAGS_HAVE_VECTORCALL | Py_TPFLAGS_DISALLOW_INSTANTIATION,
                       op_slots};
PyObject* op_type = nullptr;

// bind(symbol, checked, failed, defaults) -> Op
PyObject* bind(PyObject*, PyObject* args) {
    const char* symbol;
    PyObject *checked, *failed, *defaults;
    if (!PyArg_ParseTuple(args, "sOOO!", &symbol, &checked, &failed, &PyTuple_Type, &defaults)) return nullptr;
    for (const Entry& e : kEntries) {
        if (std::strcmp(e.name, symbol)) continue;
        if (e.nargs > kMaxArgs) break;
        Op* op = reinterpret_cast<Op*>(PyType_GenericAlloc(reinterpret_cast<PyTypeObject*>(op_type), 0));
        if (!op) return nullptr;
        op->vectorcall = op_call;
        op->entry = &e;
        op->checked = Py_NewRef(checked);
        op->failed = Py_NewRef(failed);
        op->defaults = Py_NewRef(defaults);
        return reinterpret_cast<PyObject*>(op);
    }
    return PyErr_Format(PyExc_KeyError, "no operator %s", symbol);
}

PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, "bind(symbol, checked, failed, defaults) -> callable"},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_native", "Operators of librfk.so as Python callables", -1, methods,
                          nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() {
    op_type = PyType_FromSpec(&op_spec);
    if (!op_type) return nullptr;
    PyObject* module = PyModule_Create(&module_def);
    // what it was compiled against (build.py); torch's C++ interface is only the same within a version
    if (module && PyModule_AddStringConstant(module, "built_for", RFK_BUILT_FOR) < 0) Py_CLEAR(module);
    return module;
}
