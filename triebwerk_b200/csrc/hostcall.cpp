// Python -> C calls of the decode and prefill path without ctypes.
//
// A decode step of a small batch is a few dozen kernels of a few microseconds each, so what Python spends per call is
// what the GPU waits for: through ctypes one Engine.decode_layer call cost 8.4 us of host time (attribute look-ups of
// four tensors, the stream object, argument conversion), of which the launch itself is about 2.  Here a call is one
// METH_FASTCALL function that reads tensors and the current stream through torch's C++ interface and calls the library
// function with the interpreter lock released, as ctypes does.
//
// Every function is made by one template from the declaration in triebwerk_b200.h: pointer parameters take a tensor
// (CUDA, contiguous), None or an address, int parameters a number; a trailing tq_stream_t is torch's current stream.
// They return the status (launchers: that of tq_last_compat_status()).  No C++ exception leaves them.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <exception>
#include <tuple>
#include <type_traits>
#include <utility>

#include "../../include/triebwerk_b200.h"

namespace {

// What the tensors of a call must be beside CUDA and contiguous.
enum class Need { Any, Half };

bool tensor_address(PyObject* o, Need need, void** out) {
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.is_cuda() || !t.is_contiguous() || (need == Need::Half && t.scalar_type() != at::kHalf)) {
        PyErr_SetString(PyExc_AssertionError, need == Need::Half ? "device, contiguous fp16 tensors only" : "device, contiguous tensors only");
        return false;
    }
    *out = t.data_ptr();
    return true;
}

template <typename T>
bool convert(PyObject* o, Need need, T* out) {
    if constexpr (std::is_pointer_v<T>) {
        void* p = nullptr;
        if (THPVariable_Check(o)) {
            if (!tensor_address(o, need, &p)) return false;
        } else if (o != Py_None) {
            p = PyLong_AsVoidPtr(o);
            if (PyErr_Occurred()) return false;
        }
        *out = (T)p;
        return true;
    } else {
        const long long v = PyLong_AsLongLong(o);
        if (v == -1 && PyErr_Occurred()) return false;
        *out = (T)v;
        return true;
    }
}

template <auto Fn, Need need>
struct Call;

template <typename R, typename... A, R (*Fn)(A...), Need need>
struct Call<Fn, need> {
    static constexpr size_t N = sizeof...(A) - 1;  // the last parameter is the stream

    template <size_t... I>
    static PyObject* go(PyObject* const* args, std::index_sequence<I...>) {
        std::tuple<std::decay_t<A>...> v{};
        try {
            if (!(convert(args[I], need, &std::get<I>(v)) && ...)) return nullptr;
            std::get<N>(v) = (tq_stream_t)c10::cuda::getCurrentCUDAStream().stream();
        } catch (const std::exception& e) {  // torch throws: a machine without a GPU, a tensor without memory of its own
            PyErr_SetString(PyExc_RuntimeError, e.what());
            return nullptr;
        }
        int status = 0;
        Py_BEGIN_ALLOW_THREADS
        try {
            if constexpr (std::is_void_v<R>) {
                std::apply(Fn, v);
                status = tq_last_compat_status();
            } else {
                status = std::apply(Fn, v);
            }
        } catch (const std::exception&) {  // (the library's own containers)
            status = TQ_ERR_NOMEM;
        }
        Py_END_ALLOW_THREADS
        return PyLong_FromLong(status);
    }
    static PyObject* py(PyObject*, PyObject* const* args, Py_ssize_t n) {
        if (n != (Py_ssize_t)N) {
            PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", (Py_ssize_t)N, n);
            return nullptr;
        }
        return go(args, std::make_index_sequence<N>{});
    }
};

#define TQ_CALL(name, need) {#name, (PyCFunction)(void (*)(void))Call<&name, need>::py, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    TQ_CALL(tq_engine_decode_layer, Need::Half),
    TQ_CALL(tq_engine_decode_step, Need::Half),
    TQ_CALL(tq_engine_prefill_layer, Need::Half),
    TQ_CALL(tq_engine_prefill_layer_batch, Need::Half),
    TQ_CALL(tq_engine_prefill_append, Need::Any),
    TQ_CALL(tq_engine_prefill_append_batch, Need::Any),
    TQ_CALL(launch_turbo_kv_quantize, Need::Any),
    TQ_CALL(launch_turbo_kv_quantize_batch, Need::Any),
    TQ_CALL(launch_turbo_gqa_attention_batch, Need::Any),
    TQ_CALL(launch_turbo_gqa_attention, Need::Any),
    TQ_CALL(launch_turbo_gqa_prefill_attention, Need::Any),
    TQ_CALL(launch_kv_cache_write_batch, Need::Any),
    TQ_CALL(launch_gqa_attention_batch, Need::Any),
    TQ_CALL(launch_gqa_attention, Need::Any),
    TQ_CALL(launch_gqa_prefill_attention, Need::Any),
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_hostcall", "Library calls on tensors and the current stream.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__hostcall(void) { return PyModule_Create(&module); }
