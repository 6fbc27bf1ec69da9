// CPython module `binarybrain_b200._native`: the bbcu_* operators of libbbcu_b200.so as functions on torch tensors.
//
// The operators take about 2 us of host time per kernel; called through ctypes with the current stream looked up in Python they took
// 6-9 us more, which is what bounded small networks (the training step of a 1024-420-70 MLP: 134 us of kernels in 390 us).
// Here a call parses its arguments straight into the C signature: tensors give their data pointer, None is a null pointer, numbers
// pass as they are, and a trailing stream argument that is left out is torch's current stream.  A status other than 0 raises
// binarybrain_b200.abi.BbcuError.  The functions are looked up in the library that binarybrain_b200.abi has loaded.
#include <Python.h>

#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/autograd/python_variable.h>

#include <climits>
#include <cstdint>
#include <exception>
#include <tuple>
#include <type_traits>
#include <utility>

#include "bbcu_b200.h"

namespace {

void *g_library = nullptr;

// the library handle of binarybrain_b200.abi (loads it on first use); false with a Python error set
bool bind_library()
{
    if (g_library) return true;
    PyObject *abi = PyImport_ImportModule("binarybrain_b200.abi");
    if (!abi) return false;
    PyObject *lib = PyObject_CallMethod(abi, "lib", nullptr);
    Py_DECREF(abi);
    if (!lib) return false;
    PyObject *handle = PyObject_GetAttrString(lib, "_handle");
    Py_DECREF(lib);
    if (!handle) return false;
    g_library = PyLong_AsVoidPtr(handle);
    Py_DECREF(handle);
    return g_library != nullptr;
}

PyObject *raise_status(const char *name, int status)
{
    using Text = const char *(*)(int);
    Text text = reinterpret_cast<Text>(dlsym(g_library, "bbcu_b200_error_string"));
    PyObject *abi = PyImport_ImportModule("binarybrain_b200.abi");
    if (!abi) return nullptr;
    PyObject *cls = PyObject_GetAttrString(abi, "BbcuError");
    Py_DECREF(abi);
    if (!cls) return nullptr;
    PyObject *e = PyObject_CallFunction(cls, "sis", name, status, text ? text(status) : "");
    if (e) { PyErr_SetObject(cls, e); Py_DECREF(e); }
    Py_DECREF(cls);
    return nullptr;
}

// one argument of type T; false with a Python error set when the object does not fit
template <class T> bool parse(PyObject *o, T &v)
{
    if constexpr (std::is_pointer_v<T>) {
        if (o == Py_None) { v = nullptr; return true; }
        if (THPVariable_Check(o)) {
            // an operator that may write through the pointer needs the tensor's own memory: mutable_data_ptr() gives a lazily cloned
            // tensor its copy, where const_data_ptr() would have the operator write into the tensor it was cloned from
            const at::Tensor &t = THPVariable_Unpack(o);
            try {
                if constexpr (std::is_const_v<std::remove_pointer_t<T>>) v = static_cast<T>(t.const_data_ptr());
                else v = static_cast<T>(t.mutable_data_ptr());
            } catch (const std::exception &e) {
                PyErr_SetString(PyExc_RuntimeError, e.what());
                return false;
            }
            return true;
        }
        v = reinterpret_cast<T>(PyLong_AsVoidPtr(o));
    } else if constexpr (std::is_floating_point_v<T>) {
        v = static_cast<T>(PyFloat_AsDouble(o));
    } else {
        const long long n = PyLong_AsLongLong(o);
        if (n == -1 && PyErr_Occurred()) return false;
        v = static_cast<T>(n);
        if (static_cast<long long>(v) != n) { PyErr_Format(PyExc_OverflowError, "%lld does not fit the argument", n); return false; }
        return true;
    }
    return !PyErr_Occurred();
}

template <class F> struct Operator;
template <class... A> struct Operator<int(A...)> {
    using Fn = int (*)(A...);
    static constexpr Py_ssize_t kArgs = sizeof...(A);
    using Args = std::tuple<A...>;
    static constexpr bool kStream = std::is_same_v<std::tuple_element_t<kArgs - 1, Args>, bbcu_stream_t>;

    template <std::size_t... I> static bool parse_all(PyObject *const *o, Py_ssize_t n, Args &a, std::index_sequence<I...>)
    {
        return (((Py_ssize_t)I >= n || parse(o[I], std::get<I>(a))) && ...);
    }
    static PyObject *call(Fn &fn, const char *name, PyObject *const *o, Py_ssize_t n)
    {
        if (!fn) {
            if (!bind_library()) return nullptr;
            fn = reinterpret_cast<Fn>(dlsym(g_library, name));
            if (!fn) { PyErr_Format(PyExc_AttributeError, "the library lacks %s", name); return nullptr; }
        }
        if (n != kArgs && !(kStream && n == kArgs - 1)) {
            PyErr_Format(PyExc_TypeError, "%s takes %zd arguments, got %zd", name, kArgs - kStream, n);
            return nullptr;
        }
        Args a{};
        if (!parse_all(o, n, a, std::make_index_sequence<sizeof...(A)>())) return nullptr;
        int status = 0;
        try {
            if constexpr (kStream) {
                if (n == kArgs - 1) std::get<kArgs - 1>(a) = reinterpret_cast<bbcu_stream_t>(c10::cuda::getCurrentCUDAStream().stream());
            }
            Py_BEGIN_ALLOW_THREADS
            status = std::apply(fn, a);
            Py_END_ALLOW_THREADS
        } catch (const std::exception &e) {
            PyErr_SetString(PyExc_RuntimeError, e.what());
            return nullptr;
        }
        if (status != 0) return raise_status(name, status);
        Py_RETURN_NONE;
    }
};

// A new uninitialised tensor on the device of `like`: empty_f32 / empty_i32(like, rows, cols), vector_f32(like, n), scalar_f64(like)
template <int DIM> PyObject *empty(at::ScalarType type, PyObject *const *o, Py_ssize_t n)
{
    constexpr Py_ssize_t want = DIM + 1;
    if (n != want || !THPVariable_Check(o[0])) { PyErr_SetString(PyExc_TypeError, "expected (tensor, size...)"); return nullptr; }
    int64_t size[2] = {0, 0};
    for (Py_ssize_t i = 1; i < n; ++i)
        if (!parse(o[i], size[i - 1])) return nullptr;
    try {
        const at::Tensor &like = THPVariable_Unpack(o[0]);
        return THPVariable_Wrap(at::empty(at::IntArrayRef(size, (size_t)DIM), at::TensorOptions().dtype(type).device(like.device())));
    } catch (const std::exception &e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

PyObject *empty_f32(PyObject *, PyObject *const *o, Py_ssize_t n)  { return empty<2>(at::kFloat, o, n); }
PyObject *empty_i32(PyObject *, PyObject *const *o, Py_ssize_t n)  { return empty<2>(at::kInt, o, n); }
PyObject *vector_f32(PyObject *, PyObject *const *o, Py_ssize_t n) { return empty<1>(at::kFloat, o, n); }
PyObject *scalar_f64(PyObject *, PyObject *const *o, Py_ssize_t n) { return empty<0>(at::kDouble, o, n); }

#define BB200_OPERATORS(X)                                                                                                                    \
    X(bbcu_fp32_StochasticLut6_Forward) X(bbcu_bit_fp32_StochasticLut6_Forward) X(bbcu_bit_bit_fp32_StochasticLut6_Forward)                   \
    X(bbcu_fp32_StochasticLut6_Backward) X(bbcu_bit_fp32_StochasticLut6_Backward) X(bbcu_fp32_DifferentiableLut6_ForwardTrainingRows)         \
    X(bbcu_bit_fp32_DifferentiableLut6_ForwardTraining) X(bbcu_fp32_DifferentiableLut6_ForwardInference)                                      \
    X(bbcu_bit_fp32_DifferentiableLut6_ForwardInference) X(bbcu_fp32_DifferentiableLut6_Backward) X(bbcu_bit_fp32_DifferentiableLut6_Backward) \
    X(bbcu_fp32_DifferentiableLut6_ForwardStats) X(bbcu_fp32_DifferentiableLut6_ForwardNormalize) X(bbcu_fp32_DifferentiableLut6_BackwardStats) \
    X(bbcu_fp32_DifferentiableLut6_BackwardStatsFromOutput) X(bbcu_fp32_DifferentiableLut6_BackwardApply)                                     \
    X(bbcu_fp32_StochasticBatchNormalization_ForwardTraining) X(bbcu_fp32_StochasticBatchNormalization_ReForward)                             \
    X(bbcu_fp32_StochasticBatchNormalization_ForwardInference) X(bbcu_fp32_StochasticBatchNormalization_Backward)                             \
    X(bbcu_bit_BinaryLut6_Forward) X(bbcu_bit_BinaryLut6_Forward_Lop3Immediate) X(bbcu_host_bit_BinaryLut6_Forward)                           \
    X(bbcu_fp32_Vector_clamp) X(bbcu_fp32_OptimizerAdam) X(bbcu_fp32_OptimizerAdamUpdate) X(bbcu_fp32_LossSoftmaxCrossEntropyMean)             \
    X(bbcu_fp32_LossMeanSquaredError)                                                                                                         \
    X(bbcu_fp32_Reduce_Forward) X(bbcu_fp32_Reduce_Backward) X(bbcu_bit_fp32_RealToBinary_Forward) X(bbcu_bit_fp32_BinaryToReal_Forward)      \
    X(bbcu_fp32_BinaryToReal_Forward) X(bbcu_fp32_BinaryToReal_Backward) X(bbcu_fp32_Im2Col_Forward) X(bbcu_bit_Im2Col_Forward)               \
    X(bbcu_fp32_Im2Col_Backward) X(bbcu_fp32_Col2Im_Forward) X(bbcu_bit_Col2Im_Forward) X(bbcu_fp32_Col2Im_Backward)                          \
    X(bbcu_fp32_MaxPooling_Forward) X(bbcu_bit_MaxPooling_Forward) X(bbcu_fp32_MaxPooling_Backward) X(bbcu_bit_fp32_MaxPooling_Backward)

#define BB200_DEFINE(name)                                                          \
    PyObject *py_##name(PyObject *, PyObject *const *o, Py_ssize_t n)               \
    {                                                                               \
        static Operator<decltype(name)>::Fn fn = nullptr;                           \
        return Operator<decltype(name)>::call(fn, #name, o, n);                     \
    }
BB200_OPERATORS(BB200_DEFINE)
#undef BB200_DEFINE

// ---- a layer's training step on fp32 frames: the tensors that are not given are made here and the sizes are read off the tensors, which in Python took
// 1.5 us a call (the optimizer step of a small MLP is some 65 us of host time)

template <class F> F *bound(F *&fn, const char *name)
{
    if (fn || !bind_library()) return fn;
    fn = reinterpret_cast<F *>(dlsym(g_library, name));
    if (!fn) PyErr_Format(PyExc_AttributeError, "the library lacks %s", name);
    return fn;
}

// the tensor in `o`, which has to have `dims` dimensions at least; null with a Python error set
const at::Tensor *tensor_of(PyObject *o, int64_t dims, const char *name)
{
    if (!THPVariable_Check(o)) { PyErr_Format(PyExc_TypeError, "%s: expected a tensor", name); return nullptr; }
    const at::Tensor &t = THPVariable_Unpack(o);
    if (t.dim() < dims) { PyErr_Format(PyExc_IndexError, "%s: expected %d dimensions", name, (int)dims); return nullptr; }
    return &t;
}

// a flag, or any number that int() takes
bool parse_flag(PyObject *o, int &v)
{
    if (PyLong_Check(o)) return parse(o, v);
    PyObject *n = PyNumber_Long(o);
    if (!n) return false;
    const bool ok = parse(n, v);
    Py_DECREF(n);
    return ok;
}

// an fp32 output: memory of the given tensor, the given address, or, for None, a new tensor beside `like`; false with a Python error set
struct Output {
    PyObject *given;
    at::Tensor made;
    float *data = nullptr;

    bool take(PyObject *o, const at::Tensor &like, at::IntArrayRef size)
    {
        given = o;
        if (o != Py_None) return parse(o, data);
        made = at::empty(size, at::TensorOptions().dtype(at::kFloat).device(like.device()));
        data = static_cast<float *>(made.mutable_data_ptr());
        return true;
    }
    PyObject *result() const { return given != Py_None ? Py_NewRef(given) : THPVariable_Wrap(made); }
};

// train_forward(x, y, idx, W, mean, rstd, running_mean, running_var, gamma, beta, momentum, bias, frames, lut_binarize, binary) -> (y, mean, rstd)
PyObject *train_forward(PyObject *, PyObject *const *o, Py_ssize_t n)
{
    static decltype(&bbcu_fp32_DifferentiableLut6_ForwardTrainingRows) fn = nullptr;
    if (n != 15) { PyErr_SetString(PyExc_TypeError, "train_forward takes 15 arguments"); return nullptr; }
    float gamma, beta, momentum, bias, *running_mean, *running_var;
    const float *x, *W;
    const int *index;
    int frames, lut_binarize, binary;
    try {
        const at::Tensor *xt = tensor_of(o[0], 2, "x"), *idx = xt ? tensor_of(o[2], 1, "idx") : nullptr;
        if (!idx || !parse(o[0], x) || !parse(o[2], index) || !parse(o[3], W) || !parse(o[6], running_mean) || !parse(o[7], running_var) ||
            !parse(o[8], gamma) || !parse(o[9], beta) || !parse(o[10], momentum) || !parse(o[11], bias) || !parse(o[12], frames) ||
            !parse_flag(o[13], lut_binarize) || !parse_flag(o[14], binary) || !bound(fn, "bbcu_fp32_DifferentiableLut6_ForwardTrainingRows")) return nullptr;
        const int64_t rows = xt->size(0), stride = xt->size(1), nodes = idx->size(0);
        if (rows > INT_MAX || stride > INT_MAX || nodes > INT_MAX) { PyErr_SetString(PyExc_OverflowError, "a size does not fit the operator"); return nullptr; }
        Output y, mean, rstd;
        if (!y.take(o[1], *xt, {nodes, stride}) || !mean.take(o[4], *xt, {nodes}) || !rstd.take(o[5], *xt, {nodes})) return nullptr;
        const auto stream = reinterpret_cast<bbcu_stream_t>(c10::cuda::getCurrentCUDAStream().stream());
        int status = 0;
        Py_BEGIN_ALLOW_THREADS
        status = fn(x, y.data, index, W, mean.data, rstd.data, running_mean, running_var, gamma, beta, momentum, bias, (int)rows, (int)nodes, frames, (int)stride,
                    lut_binarize, binary, stream);
        Py_END_ALLOW_THREADS
        if (status != 0) return raise_status("bbcu_fp32_DifferentiableLut6_ForwardTrainingRows", status);
        PyObject *r = PyTuple_New(3);
        if (!r) return nullptr;
        PyTuple_SET_ITEM(r, 0, y.result());
        PyTuple_SET_ITEM(r, 1, mean.result());
        PyTuple_SET_ITEM(r, 2, rstd.result());
        return r;
    } catch (const std::exception &e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

// train_backward(x, dy, dx, idx, W, dW, mean, rstd, gamma, beta, bias, n_in, frames, lut_binarize, binary) -> dx; dmean and dvar go to scratch
PyObject *train_backward(PyObject *, PyObject *const *o, Py_ssize_t n)
{
    static decltype(&bbcu_fp32_DifferentiableLut6_Backward) fn = nullptr;
    if (n != 15) { PyErr_SetString(PyExc_TypeError, "train_backward takes 15 arguments"); return nullptr; }
    float gamma, beta, bias, *dW;
    const float *x, *dy, *W, *mean, *rstd;
    const int *index;
    int n_in, frames, lut_binarize, binary;
    try {
        const at::Tensor *xt = tensor_of(o[0], 2, "x"), *dyt = xt ? tensor_of(o[1], 2, "dy") : nullptr, *idx = dyt ? tensor_of(o[3], 1, "idx") : nullptr;
        if (!idx || !parse(o[0], x) || !parse(o[1], dy) || !parse(o[3], index) || !parse(o[4], W) || !parse(o[5], dW) || !parse(o[6], mean) ||
            !parse(o[7], rstd) || !parse(o[8], gamma) || !parse(o[9], beta) || !parse(o[10], bias) || !parse(o[11], n_in) || !parse(o[12], frames) ||
            !parse_flag(o[13], lut_binarize) || !parse_flag(o[14], binary) || !bound(fn, "bbcu_fp32_DifferentiableLut6_Backward")) return nullptr;
        const int64_t stride = dyt->size(1), nodes = idx->size(0);
        if (xt->size(1) != stride) { PyErr_SetString(PyExc_AssertionError, "x and dy differ in their stride"); return nullptr; }
        if (stride > INT_MAX || nodes > INT_MAX) { PyErr_SetString(PyExc_OverflowError, "a size does not fit the operator"); return nullptr; }
        Output dx, scratch;
        if (!dx.take(o[2], *dyt, {n_in, stride}) || !scratch.take(Py_None, *dyt, {2 * nodes})) return nullptr;
        const auto stream = reinterpret_cast<bbcu_stream_t>(c10::cuda::getCurrentCUDAStream().stream());
        int status = 0;
        Py_BEGIN_ALLOW_THREADS
        status = fn(x, dy, dx.data, nullptr, index, nullptr, W, dW, mean, rstd, scratch.data, scratch.data + nodes, gamma, beta, bias, 0, n_in, (int)nodes, frames,
                    (int)stride, 0, 0, lut_binarize, binary, stream);
        Py_END_ALLOW_THREADS
        if (status != 0) return raise_status("bbcu_fp32_DifferentiableLut6_Backward", status);
        return dx.result();
    } catch (const std::exception &e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

#define BB200_METHOD(name, function) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(function)), METH_FASTCALL, nullptr},
#define BB200_OPERATOR_METHOD(name) BB200_METHOD(#name, py_##name)
PyMethodDef g_methods[] = {
    BB200_OPERATORS(BB200_OPERATOR_METHOD)
    BB200_METHOD("empty_f32", empty_f32) BB200_METHOD("empty_i32", empty_i32) BB200_METHOD("vector_f32", vector_f32) BB200_METHOD("scalar_f64", scalar_f64)
    BB200_METHOD("train_forward", train_forward) BB200_METHOD("train_backward", train_backward)
    {nullptr, nullptr, 0, nullptr}};
#undef BB200_METHOD

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", "bbcu_* operators on torch tensors", -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}   // namespace

PyMODINIT_FUNC PyInit__native()
{
    PyObject *m = PyModule_Create(&g_module);
    if (!m) return nullptr;
    if (PyModule_AddIntConstant(m, "SMALL_NODE_FRAMES", BBCU_B200_SMALL_NODE_FRAMES) || PyModule_AddIntConstant(m, "SMALL_FRAMES", BBCU_B200_SMALL_FRAMES)) {
        Py_DECREF(m);
        return nullptr;
    }
    return m;
}
