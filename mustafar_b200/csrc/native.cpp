// CPython binding of the entry points that run once or more per decode step.  The C ABI is the interface; ctypes serves
// it everywhere else, but converts arguments one by one through Python objects: 9 us for the 37 arguments of a fused
// attention call, more than the launch itself.  Here each function is called through the vectorcall protocol (under 1 us).
// Integers and addresses (None = null) must fit their C type: OverflowError instead of a silent truncation.  The GIL is
// released around the call, as ctypes does.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <limits>
#include <tuple>
#include <type_traits>
#include <utility>

#include "../../include/mustafar_b200.h"

namespace {

template <typename T>
bool convert(PyObject* o, T& v) {
    if constexpr (std::is_pointer_v<T>) {
        if (o == Py_None) {
            v = nullptr;
            return true;
        }
        void* p = PyLong_AsVoidPtr(o);
        if (p == nullptr && PyErr_Occurred()) return false;
        v = static_cast<T>(p);
    } else if constexpr (std::is_floating_point_v<T>) {
        const double d = PyFloat_AsDouble(o);
        if (d == -1.0 && PyErr_Occurred()) return false;
        v = static_cast<T>(d);
    } else if constexpr (std::is_unsigned_v<T>) {
        const size_t n = PyLong_AsSize_t(o);
        if (n == static_cast<size_t>(-1) && PyErr_Occurred()) return false;
        v = static_cast<T>(n);
    } else {
        const long long n = PyLong_AsLongLong(o);
        if (n == -1 && PyErr_Occurred()) return false;
        if (n < std::numeric_limits<T>::min() || n > std::numeric_limits<T>::max()) {
            PyErr_SetString(PyExc_OverflowError, "argument does not fit its C type");
            return false;
        }
        v = static_cast<T>(n);
    }
    return true;
}

template <auto Fn>
struct Wrap;

template <typename... Args, int (*Fn)(Args...)>
struct Wrap<Fn> {
    template <size_t... I>
    static PyObject* run(PyObject* const* args, std::index_sequence<I...>) {
        std::tuple<Args...> v;
        if (!(convert(args[I], std::get<I>(v)) && ...)) return nullptr;
        int status;
        Py_BEGIN_ALLOW_THREADS
        status = Fn(std::get<I>(v)...);
        Py_END_ALLOW_THREADS
        return PyLong_FromLong(status);
    }
    static PyObject* call(PyObject*, PyObject* const* args, Py_ssize_t n) {
        if (n != static_cast<Py_ssize_t>(sizeof...(Args))) {
            PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", static_cast<Py_ssize_t>(sizeof...(Args)), n);
            return nullptr;
        }
        return run(args, std::index_sequence_for<Args...>{});
    }
};

#define MFAR_METHOD(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&Wrap<&f>::call)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    MFAR_METHOD(mfar_compress_fp16),
    MFAR_METHOD(mfar_compact_heads_fp16),
    MFAR_METHOD(mfar_compress_quant),
    MFAR_METHOD(mfar_decode_attention_fp16),
    MFAR_METHOD(mfar_decode_attention_fp16_dyn),
    MFAR_METHOD(mfar_decode_attention_quant),
    MFAR_METHOD(mfar_key_scores_rows_fp16),
    MFAR_METHOD(mfar_value_output_rows_fp16),
    MFAR_METHOD(mfar_key_scores_rows_quant),
    MFAR_METHOD(mfar_value_output_rows_quant),
    MFAR_METHOD(mfar_add_rmsnorm_f16),
    MFAR_METHOD(mfar_rope_append_f16),
    MFAR_METHOD(mfar_silu_mul_f16),
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, 0, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() { return PyModule_Create(&module); }
