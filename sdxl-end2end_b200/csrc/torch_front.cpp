// Native front of the Python mirror: takes torch tensors and the mirror's Weight / LinearCall objects,
// allocates the outputs and calls the C ABI (include/sdxlq.h) without building ctypes structures.
//
// What bounds it: host time. A projection of few rows runs for 5 to 15 us on the GPU; checking its arguments,
// allocating its output and filling a ctypes descriptor in Python cost more than that again. Measured per call
// with its launches (B200): FP8 of two rows 15.3 -> 10.3 us, FP16 of 154 rows 11.1 -> 9.9 us (now the
// kernels), the ten calls of a transformer block's weight packing 113 -> 68 us.
//
// Every function answers with
//   a result          the call was issued,
//   an int            the C ABI refused it (status; the message is in the context),
//   None              the arguments are not those of an ordinary call: the caller's Python path looks at
//                     them, with its own checks and messages, and issues the call or raises.
// So this file states no error message, and accepts a call only where that path would accept it.
//
// The C ABI's functions arrive as addresses (bind), so that whichever libsdxlq.so the package has loaded
// is the one that runs.

#include "../../include/sdxlq.h"

#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <limits>
#include <utility>

namespace {

int (*g_linear)(sdxlq_context*, const sdxlq_linear_desc*) = nullptr;
int (*g_linear_grouped)(sdxlq_context*, const sdxlq_linear_desc*, size_t) = nullptr;
int (*g_layer_norm)(sdxlq_context*, const sdxlq_layer_norm_desc*) = nullptr;
int (*g_quantize_int8)(sdxlq_context*, const void*, int32_t, uint64_t, uint64_t, uint32_t, int8_t*, float*) = nullptr;
int (*g_quantize_fp8)(sdxlq_context*, const void*, uint64_t, int32_t, uint8_t*, float*) = nullptr;
int (*g_pack_int8)(sdxlq_context*, const void*, int32_t, uint64_t, uint64_t, uint32_t, int8_t*, float*) = nullptr;
int (*g_pack_fp8)(sdxlq_context*, const void*, int32_t, uint64_t, uint64_t, int32_t, int32_t, int32_t, uint8_t*, float*) = nullptr;

// Attribute names of Weight and LinearCall, interned once.
struct Names {
    PyObject *data, *type, *n, *k, *scales, *scale_mode, *layout, *convrot_group_size;
    PyObject *x, *weight, *bias, *activation, *y, *xq, *xq_scales, *acc_out, *residual, *y_amax, *x_amax;
} g_names;

sdxlq_context* context_of(PyObject* handle) {
    return reinterpret_cast<sdxlq_context*>(PyLong_AsVoidPtr(handle));
}

// A reference to an attribute, released at the end of the scope.
class Attribute {
public:
    Attribute(PyObject* object, PyObject* name) : value_(PyObject_GetAttr(object, name)) {
        if (value_ == nullptr) PyErr_Clear();
    }
    ~Attribute() { Py_XDECREF(value_); }
    Attribute(const Attribute&) = delete;
    Attribute& operator=(const Attribute&) = delete;
    PyObject* get() const { return value_; }
    bool integer(uint64_t& out) const {
        if (value_ == nullptr || !PyLong_Check(value_)) return false;
        out = PyLong_AsUnsignedLongLong(value_);
        if (out == static_cast<uint64_t>(-1) && PyErr_Occurred()) { PyErr_Clear(); return false; }
        return true;
    }

private:
    PyObject* value_;
};

// A reference that is released at the end of the scope, by an exception too, unless it was handed on.
class Owned {
public:
    explicit Owned(PyObject* object) : object_(object) {}
    ~Owned() { Py_XDECREF(object_); }
    Owned(const Owned&) = delete;
    Owned& operator=(const Owned&) = delete;
    PyObject* get() const { return object_; }
    PyObject* release() { return std::exchange(object_, nullptr); }

private:
    PyObject* object_;
};

bool is_none(PyObject* object) { return object == Py_None; }

// The tensor behind `object` (an input): false when it is not a CUDA tensor, or an attribute that does not exist. `pointer`
// stays null for None.
bool optional_input(PyObject* object, const void*& pointer) {
    pointer = nullptr;
    if (is_none(object)) return true;
    if (object == nullptr || !THPVariable_Check(object)) return false;
    const at::Tensor& tensor = THPVariable_Unpack(object);
    if (!tensor.is_cuda()) return false;
    pointer = tensor.const_data_ptr();
    return true;
}

// The same for a tensor that the call writes. A copy-on-write tensor gets its own memory here.
bool optional_output(PyObject* object, void*& pointer) {
    pointer = nullptr;
    if (is_none(object)) return true;
    if (object == nullptr || !THPVariable_Check(object)) return false;
    const at::Tensor& tensor = THPVariable_Unpack(object);
    if (!tensor.is_cuda()) return false;
    pointer = tensor.mutable_data_ptr();
    return true;
}

bool ordinary(PyObject* object) { return object != nullptr && THPVariable_Check(object) && THPVariable_Unpack(object).is_cuda(); }

bool half_vector(PyObject* object, int64_t width) {
    if (!ordinary(object)) return false;
    const at::Tensor& t = THPVariable_Unpack(object);
    return t.scalar_type() == at::kHalf && t.dim() == 1 && t.size(0) == width && t.is_contiguous();
}

// Goes through the dispatcher where somebody may listen: a dispatch mode or a transform is active on this thread, or new
// memory is filled for determinism. Otherwise straight to the allocator.
at::Tensor empty(at::IntArrayRef sizes, at::ScalarType type, const at::Tensor& like) {
    const bool filled = at::globalContext().deterministicAlgorithms() && at::globalContext().deterministicFillUninitializedMemory();
    if (filled || !(c10::impl::tls_local_dispatch_key_set().included_ == c10::default_included_set)) {
        return at::empty(sizes, at::TensorOptions().dtype(type).device(like.device()));
    }
    return at::Tensor(at::detail::empty_cuda(sizes, type, like.device(), std::nullopt));
}

bool read_weight(PyObject* object, sdxlq_weight& w) {
    uint64_t type, layout, mode, group;
    {
        const Attribute data(object, g_names.data);
        const void* pointer = nullptr;
        if (is_none(data.get()) || !optional_input(data.get(), pointer)) return false;
        w.data = pointer;
    }
    {
        const Attribute scales(object, g_names.scales);
        const void* pointer = nullptr;
        if (!optional_input(scales.get(), pointer)) return false;
        w.scales = static_cast<const float*>(pointer);
        w.scale_count = pointer == nullptr ? 0 : static_cast<uint64_t>(THPVariable_Unpack(scales.get()).numel());
    }
    if (!Attribute(object, g_names.type).integer(type) || !Attribute(object, g_names.n).integer(w.n) ||
        !Attribute(object, g_names.k).integer(w.k) || !Attribute(object, g_names.layout).integer(layout) ||
        !Attribute(object, g_names.scale_mode).integer(mode) || !Attribute(object, g_names.convrot_group_size).integer(group)) {
        return false;
    }
    w.dtype = static_cast<int32_t>(type);
    w.layout = static_cast<int32_t>(layout);
    w.scale_mode = static_cast<int32_t>(mode);
    w.convrot_group_size = static_cast<uint32_t>(group);
    return w.n != 0 && w.k != 0;
}

struct LinearArguments {
    PyObject *input, *weight, *bias, *out, *xq, *xq_scales, *acc_out, *residual, *y_amax, *x_amax;
    uint64_t activation;
};

// Fills the descriptor of one projection and allocates its output when the caller gave none. False: not an
// ordinary call.
bool describe(const LinearArguments& a, bool poison, sdxlq_linear_desc& d, at::Tensor& allocated) {
    d = sdxlq_linear_desc{};
    if (!read_weight(a.weight, d.weight)) return false;
    const int64_t k = static_cast<int64_t>(d.weight.k), n = static_cast<int64_t>(d.weight.n);
    const void* input = nullptr;
    void* output = nullptr;
    PyObject* const leading = is_none(a.input) ? a.xq : a.input;
    if (!ordinary(leading)) return false;
    const at::Tensor& lead = THPVariable_Unpack(leading);
    if (lead.dim() < 1) return false;
    if (leading == a.input) {
        if (lead.scalar_type() != at::kHalf || lead.dim() < 2 || !lead.is_contiguous() || lead.size(-1) != k) return false;
        d.x = lead.const_data_ptr();
    }
    const int64_t m = lead.numel() / k;
    d.m = static_cast<uint64_t>(m);
    if (!is_none(a.bias)) {
        if (!ordinary(a.bias)) return false;
        const at::Tensor& bias = THPVariable_Unpack(a.bias);
        if (bias.scalar_type() != at::kHalf || bias.dim() != 1 || bias.size(0) != n) return false;
        d.bias = bias.const_data_ptr();
    }
    const int64_t n_out = a.activation == SDXLQ_ACT_GEGLU ? n / 2 : n;
    if (!is_none(a.residual)) {
        if (!ordinary(a.residual)) return false;
        const at::Tensor& residual = THPVariable_Unpack(a.residual);
        if (residual.scalar_type() != at::kHalf || !residual.is_contiguous() || residual.numel() != m * n_out) return false;
        d.residual = residual.const_data_ptr();
    }
    d.activation = static_cast<int32_t>(a.activation);
    if (!optional_input(a.xq, input)) return false;
    d.xq = input;
    if (!optional_input(a.xq_scales, input)) return false;
    d.xq_scales = static_cast<const float*>(input);
    if (!optional_output(a.acc_out, output)) return false;
    d.acc_out = static_cast<int32_t*>(output);
    if (!optional_output(a.y_amax, output)) return false;
    d.y_amax = output;
    if (!optional_output(a.x_amax, output)) return false;          // put back to zero by the call
    d.x_amax = output;
    if (is_none(a.out)) {
        c10::SmallVector<int64_t, 5> sizes(lead.sizes().begin(), lead.sizes().end());
        sizes.back() = n_out;
        allocated = empty(sizes, at::kHalf, lead);
        if (poison) allocated.fill_(std::numeric_limits<double>::quiet_NaN());
        d.y = allocated.mutable_data_ptr();
    } else {
        if (!optional_output(a.out, output)) return false;
        d.y = output;
    }
    return true;
}

// A call into the C ABI, which may wait for room in the stream's launch queue: other Python threads run meanwhile.
template <typename Function, typename... Arguments>
int unlocked(Function function, Arguments... arguments) {
    int status;
    Py_BEGIN_ALLOW_THREADS
    status = function(arguments...);
    Py_END_ALLOW_THREADS
    return status;
}

PyObject* answer(int status, PyObject* result) {
    if (status == SDXLQ_OK) return result;
    Py_XDECREF(result);
    return PyLong_FromLong(status);
}

PyObject* tensor_or(PyObject* given, at::Tensor& allocated) {
    if (!is_none(given)) return Py_NewRef(given);
    return THPVariable_Wrap(std::move(allocated));
}

// linear(handle, input, weight, bias, activation, out, xq, xq_scales, acc_out, residual, y_amax, x_amax, poison)
PyObject* linear(PyObject*, PyObject* const* args, Py_ssize_t count) {
    if (count != 13) Py_RETURN_NONE;
    LinearArguments a{args[1], args[2], args[3], args[5], args[6], args[7], args[8], args[9], args[10], args[11], 0};
    if (!PyLong_Check(args[4])) Py_RETURN_NONE;
    a.activation = PyLong_AsUnsignedLongLongMask(args[4]);
    sdxlq_linear_desc desc;
    at::Tensor allocated;
    if (!describe(a, args[12] == Py_True, desc, allocated)) Py_RETURN_NONE;
    return answer(unlocked(g_linear, context_of(args[0]), &desc), tensor_or(a.out, allocated));
}

// linear_grouped(handle, calls, poison): a list of outputs; the calls' `y` is set like the Python path does.
PyObject* linear_grouped(PyObject*, PyObject* const* args, Py_ssize_t count) {
    constexpr Py_ssize_t kMost = 16;          // small groups; larger ones go through the Python path
    if (count != 3 || !PyList_Check(args[1])) Py_RETURN_NONE;
    const Py_ssize_t calls = PyList_GET_SIZE(args[1]);
    if (calls == 0 || calls > kMost) Py_RETURN_NONE;
    for (Py_ssize_t i = 1; i < calls; ++i) {
        for (Py_ssize_t j = 0; j < i; ++j) {
            if (PyList_GET_ITEM(args[1], i) == PyList_GET_ITEM(args[1], j)) Py_RETURN_NONE;      // one output for both
        }
    }
    sdxlq_linear_desc descs[kMost];
    at::Tensor allocated[kMost];
    Owned outputs(PyList_New(calls));
    if (outputs.get() == nullptr) return nullptr;
    for (Py_ssize_t i = 0; i < calls; ++i) {
        PyObject* const call = PyList_GET_ITEM(args[1], i);
        const Attribute x(call, g_names.x), weight(call, g_names.weight), bias(call, g_names.bias), y(call, g_names.y),
            xq(call, g_names.xq), xq_scales(call, g_names.xq_scales), acc_out(call, g_names.acc_out),
            residual(call, g_names.residual), y_amax(call, g_names.y_amax), x_amax(call, g_names.x_amax);
        LinearArguments a{x.get(), weight.get(), bias.get(), y.get(), xq.get(), xq_scales.get(), acc_out.get(),
                          residual.get(), y_amax.get(), x_amax.get(), 0};
        if (weight.get() == nullptr || !Attribute(call, g_names.activation).integer(a.activation) ||
            !describe(a, args[2] == Py_True, descs[i], allocated[i])) {
            Py_RETURN_NONE;
        }
        PyList_SET_ITEM(outputs.get(), i, Py_NewRef(is_none(y.get()) ? Py_None : y.get()));
    }
    const int status = unlocked(g_linear_grouped, context_of(args[0]), descs, static_cast<size_t>(calls));
    if (status != SDXLQ_OK) return PyLong_FromLong(status);
    for (Py_ssize_t i = 0; i < calls; ++i) {
        if (!allocated[i].defined()) continue;
        Owned y(THPVariable_Wrap(std::move(allocated[i])));
        if (y.get() == nullptr || PyObject_SetAttr(PyList_GET_ITEM(args[1], i), g_names.y, y.get()) != 0) return nullptr;
        PyObject* const placeholder = PyList_GET_ITEM(outputs.get(), i);
        PyList_SET_ITEM(outputs.get(), i, y.release());
        Py_DECREF(placeholder);
    }
    return outputs.release();
}

PyObject* pair_of(at::Tensor& first, at::Tensor& second) {
    PyObject* const a = THPVariable_Wrap(std::move(first));
    PyObject* const b = THPVariable_Wrap(std::move(second));
    PyObject* const pair = PyTuple_New(2);
    if (a == nullptr || b == nullptr || pair == nullptr) {
        Py_XDECREF(a); Py_XDECREF(b); Py_XDECREF(pair);
        return nullptr;
    }
    PyTuple_SET_ITEM(pair, 0, a);
    PyTuple_SET_ITEM(pair, 1, b);
    return pair;
}

// layer_norm(handle, input, gamma, beta, epsilon, out, consumer): `consumer` None for the FP16 form.
PyObject* layer_norm(PyObject*, PyObject* const* args, Py_ssize_t count) {
    if (count != 7 || !ordinary(args[1])) Py_RETURN_NONE;
    const at::Tensor& x = THPVariable_Unpack(args[1]);
    if (x.scalar_type() != at::kHalf || x.dim() < 1 || !x.is_contiguous()) Py_RETURN_NONE;
    const int64_t width = x.size(-1);
    if (width == 0 || !half_vector(args[2], width) || !half_vector(args[3], width)) Py_RETURN_NONE;
    const double epsilon = PyFloat_AsDouble(args[4]);
    if (epsilon == -1.0 && PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }
    sdxlq_layer_norm_desc d{};
    d.x = x.const_data_ptr();
    d.rows = static_cast<uint64_t>(x.numel() / width);
    d.width = static_cast<uint64_t>(width);
    d.gamma = THPVariable_Unpack(args[2]).const_data_ptr();
    d.beta = THPVariable_Unpack(args[3]).const_data_ptr();
    d.epsilon = static_cast<float>(epsilon);
    if (is_none(args[6])) {
        d.out_dtype = SDXLQ_FP16;
        at::Tensor allocated;
        if (is_none(args[5])) {
            allocated = empty(x.sizes(), at::kHalf, x);
            d.y = allocated.mutable_data_ptr();
        } else if (!optional_output(args[5], d.y)) {
            Py_RETURN_NONE;
        }
        return answer(unlocked(g_layer_norm, context_of(args[0]), &d), tensor_or(args[5], allocated));
    }
    sdxlq_weight w{};
    if (!read_weight(args[6], w) || w.k != d.width) Py_RETURN_NONE;
    const bool int8 = w.dtype == SDXLQ_INT8;
    if (!int8 && w.dtype != SDXLQ_FP8_E4M3 && w.dtype != SDXLQ_FP8_E5M2) Py_RETURN_NONE;
    at::Tensor xq = empty(x.sizes(), int8 ? at::kChar : at::kByte, x);
    at::Tensor scales = empty({int8 ? static_cast<int64_t>(d.rows) : 1}, at::kFloat, x);
    d.out_dtype = w.dtype;
    d.convrot_group_size = int8 ? w.convrot_group_size : 0;
    d.xq = xq.mutable_data_ptr();
    d.xq_scales = static_cast<float*>(scales.mutable_data_ptr());
    const int status = unlocked(g_layer_norm, context_of(args[0]), &d);
    return status == SDXLQ_OK ? pair_of(xq, scales) : PyLong_FromLong(status);
}

bool small_integer(PyObject* object, int64_t& out) {
    if (!PyLong_Check(object)) return false;
    out = PyLong_AsLongLong(object);
    if (out == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
    return true;
}

// quantize_int8(handle, source, group, rank_2): (int8 like the source, FP32 scale per row). `rank_2` asks for the
// weight packer (rank-2 sources only) instead of the activation quantiser.
PyObject* quantize_int8(PyObject*, PyObject* const* args, Py_ssize_t count) {
    int64_t group;
    if (count != 4 || !ordinary(args[1]) || !small_integer(args[2], group) || group < 0) Py_RETURN_NONE;
    const at::Tensor& x = THPVariable_Unpack(args[1]);
    const bool half = x.scalar_type() == at::kHalf, weight = args[3] == Py_True;
    if ((!half && x.scalar_type() != at::kFloat) || x.dim() < 2 || (weight && x.dim() != 2) || !x.is_contiguous() || x.numel() == 0) Py_RETURN_NONE;
    const int64_t k = x.size(-1), m = x.numel() / k;
    at::Tensor xq = empty(x.sizes(), at::kChar, x);
    at::Tensor scales = empty({m}, at::kFloat, x);
    const auto call = weight ? g_pack_int8 : g_quantize_int8;
    const int status = unlocked(call, context_of(args[0]), x.const_data_ptr(), half ? SDXLQ_FP16 : SDXLQ_FP32, static_cast<uint64_t>(m),
                            static_cast<uint64_t>(k), static_cast<uint32_t>(group), static_cast<int8_t*>(xq.mutable_data_ptr()),
                            static_cast<float*>(scales.mutable_data_ptr()));
    return status == SDXLQ_OK ? pair_of(xq, scales) : PyLong_FromLong(status);
}

// quantize_fp8(handle, source, format): (bytes like the source, FP32 scale)
PyObject* quantize_fp8(PyObject*, PyObject* const* args, Py_ssize_t count) {
    int64_t format;
    if (count != 3 || !ordinary(args[1]) || !small_integer(args[2], format)) Py_RETURN_NONE;
    const at::Tensor& x = THPVariable_Unpack(args[1]);
    if (x.scalar_type() != at::kHalf || x.dim() < 1 || !x.is_contiguous()) Py_RETURN_NONE;
    at::Tensor q = empty(x.sizes(), at::kByte, x);
    at::Tensor scale = empty({1}, at::kFloat, x);
    const int status = unlocked(g_quantize_fp8, context_of(args[0]), x.const_data_ptr(), static_cast<uint64_t>(x.numel()),
                                      static_cast<int32_t>(format), static_cast<uint8_t*>(q.mutable_data_ptr()),
                                      static_cast<float*>(scale.mutable_data_ptr()));
    return status == SDXLQ_OK ? pair_of(q, scale) : PyLong_FromLong(status);
}

// pack_fp8(handle, source, source_dtype, format, scale_mode, layout): (bytes, FP32 scales) of a rank-2 weight
PyObject* pack_fp8(PyObject*, PyObject* const* args, Py_ssize_t count) {
    int64_t source_dtype, format, mode, layout;
    if (count != 6 || !ordinary(args[1]) || !small_integer(args[2], source_dtype) || !small_integer(args[3], format) ||
        !small_integer(args[4], mode) || !small_integer(args[5], layout)) {
        Py_RETURN_NONE;
    }
    const at::Tensor& x = THPVariable_Unpack(args[1]);
    if (x.dim() != 2 || !x.is_contiguous()) Py_RETURN_NONE;
    const int64_t n = x.size(0), k = x.size(1);
    const bool k_major = layout == SDXLQ_K_MAJOR_KN;
    at::Tensor packed = empty({k_major ? k : n, k_major ? n : k}, at::kByte, x);
    at::Tensor scales = empty({mode == SDXLQ_SCALE_PER_OUTPUT_CHANNEL ? n : 1}, at::kFloat, x);
    const int status = unlocked(g_pack_fp8, context_of(args[0]), x.const_data_ptr(), static_cast<int32_t>(source_dtype),
                                  static_cast<uint64_t>(n), static_cast<uint64_t>(k), static_cast<int32_t>(format),
                                  static_cast<int32_t>(mode), static_cast<int32_t>(layout),
                                  static_cast<uint8_t*>(packed.mutable_data_ptr()), static_cast<float*>(scales.mutable_data_ptr()));
    return status == SDXLQ_OK ? pair_of(packed, scales) : PyLong_FromLong(status);
}

// bind(addresses): the C ABI's functions, in the order below.
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t count) {
    void* addresses[7];
    if (count != 7) { PyErr_SetString(PyExc_ValueError, "bind wants seven addresses"); return nullptr; }
    for (int i = 0; i < 7; ++i) {
        addresses[i] = PyLong_AsVoidPtr(args[i]);
        if (addresses[i] == nullptr) {
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "null function address");
            return nullptr;
        }
    }
    g_linear = reinterpret_cast<decltype(g_linear)>(addresses[0]);
    g_linear_grouped = reinterpret_cast<decltype(g_linear_grouped)>(addresses[1]);
    g_layer_norm = reinterpret_cast<decltype(g_layer_norm)>(addresses[2]);
    g_quantize_int8 = reinterpret_cast<decltype(g_quantize_int8)>(addresses[3]);
    g_quantize_fp8 = reinterpret_cast<decltype(g_quantize_fp8)>(addresses[4]);
    g_pack_int8 = reinterpret_cast<decltype(g_pack_int8)>(addresses[5]);
    g_pack_fp8 = reinterpret_cast<decltype(g_pack_fp8)>(addresses[6]);
    Py_RETURN_NONE;
}

template <PyObject* (*Function)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* args, Py_ssize_t count) {
    HANDLE_TH_ERRORS                                  // out of memory in the allocator, for one
    return Function(self, args, count);
    END_HANDLE_TH_ERRORS
}

template <PyObject* (*Function)(PyObject*, PyObject* const*, Py_ssize_t)>
PyCFunction entry() { return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&guarded<Function>)); }

PyMethodDef g_methods[] = {
    {"bind", entry<bind>(), METH_FASTCALL, nullptr},
    {"linear", entry<linear>(), METH_FASTCALL, nullptr},
    {"linear_grouped", entry<linear_grouped>(), METH_FASTCALL, nullptr},
    {"layer_norm", entry<layer_norm>(), METH_FASTCALL, nullptr},
    {"quantize_int8", entry<quantize_int8>(), METH_FASTCALL, nullptr},
    {"quantize_fp8", entry<quantize_fp8>(), METH_FASTCALL, nullptr},
    {"pack_fp8", entry<pack_fp8>(), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_front", "Native front of the quantized-Linear operator.", -1, g_methods,
                        nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__front() {
    const struct { PyObject** slot; const char* text; } names[] = {
        {&g_names.data, "data"}, {&g_names.type, "type"}, {&g_names.n, "n"}, {&g_names.k, "k"}, {&g_names.scales, "scales"},
        {&g_names.scale_mode, "scale_mode"}, {&g_names.layout, "layout"}, {&g_names.convrot_group_size, "convrot_group_size"},
        {&g_names.x, "x"}, {&g_names.weight, "weight"}, {&g_names.bias, "bias"}, {&g_names.activation, "activation"},
        {&g_names.y, "y"}, {&g_names.xq, "xq"}, {&g_names.xq_scales, "xq_scales"}, {&g_names.acc_out, "acc_out"},
        {&g_names.residual, "residual"}, {&g_names.y_amax, "y_amax"}, {&g_names.x_amax, "x_amax"}};
    for (const auto& name : names) {
        *name.slot = PyUnicode_InternFromString(name.text);
        if (*name.slot == nullptr) return nullptr;
    }
    return PyModule_Create(&g_module);
}
