// Native host path of the operator and model API: argument checks, output allocation and the launches of one call in
// C++, so that a call costs a few microseconds of host time instead of tens (a ctypes call with thirty arguments and
// its Python-side checks took 29 us around a 4 us kernel).  The kernels stay behind the C ABI of libcdssm_b200.so.
#pragma once
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <array>
#include <mutex>
#include <string>

#include "../../../include/cdssm_b200.h"

namespace cdssm_host {

using at::Tensor;

// Raised as the package's CdssmError.
struct Error : std::runtime_error {
    using std::runtime_error::runtime_error;
};

void check(int rc, const char* what);   // throws Error unless rc is CDSSM_OK

inline int dtype_code(const Tensor& t) {
    if (t.scalar_type() == at::kBFloat16) return CDSSM_BF16;
    if (t.scalar_type() == at::kFloat) return CDSSM_F32;
    throw Error(std::string("unsupported dtype ") + c10::toString(t.scalar_type()) +
                ": use bfloat16 (the reference's type) or float32");
}

inline void need_cuda(const Tensor& t, const char* name) {
    if (!t.is_cuda()) throw Error(std::string(name) + " must be a CUDA tensor (no CPU fallback exists)");
}

// A dense CUDA tensor of the wanted type, or an error (the reference launchers check neither).
inline Tensor dense(const Tensor& t, at::ScalarType dt, const char* name) {
    need_cuda(t, name);
    if (t.scalar_type() != dt)
        throw Error(std::string(name) + " has dtype " + c10::toString(t.scalar_type()) + ", expected " + c10::toString(dt));
    return t.is_contiguous() ? t : t.contiguous();
}

// Per-head float32 vectors; a bf16 buffer (a model cast with .bfloat16()) is converted.
inline Tensor f32_vector(const Tensor& t, const char* name) {
    need_cuda(t, name);
    if (t.scalar_type() == at::kFloat && t.is_contiguous()) return t;
    return t.detach().to(at::kFloat).contiguous();
}

// (sizes are read by position below: another rank would be taken for a batch of its first dimensions)
inline void need_dims(const Tensor& t, int64_t n, const char* name) {
    if (t.dim() != n) throw Error(std::string(name) + " must have " + std::to_string(n) + " dimensions, not " + std::to_string(t.dim()));
}

inline const void* cptr(const Tensor& t) { return t.defined() ? t.const_data_ptr() : nullptr; }
inline void* mptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
inline const float* fptr(const Tensor& t) { return t.defined() ? static_cast<const float*>(t.const_data_ptr()) : nullptr; }
inline float* fmut(const Tensor& t) { return t.defined() ? static_cast<float*>(t.data_ptr()) : nullptr; }

inline void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// Outputs straight from the framework's CUDA allocator: by way of the dispatcher an allocation took 0.4 us more, of the 4.5 that a one-token
// step's call takes.  Not where somebody looks on (dispatch modes and transforms are keys beside the default ones) or wants memory filled
// (deterministic algorithms).
inline Tensor empty_cuda(at::IntArrayRef sizes, at::ScalarType dt, const Tensor& like) {
    const bool watched = !(c10::impl::tls_local_dispatch_key_set().included_ - c10::default_included_set).empty();
    if (watched || at::globalContext().deterministicAlgorithms()) return at::empty(sizes, like.options().dtype(dt));
    return at::detail::empty_cuda(sizes, dt, like.device(), std::nullopt);
}
inline Tensor empty_like_dims(at::IntArrayRef sizes, const Tensor& like) { return empty_cuda(sizes, like.scalar_type(), like); }
inline Tensor empty_f32(at::IntArrayRef sizes, const Tensor& like) { return empty_cuda(sizes, at::kFloat, like); }

struct Dyn {   // the five scalars of the dynamics
    float c[5];
};

// The grow-only scratch buffer of a (device, current stream): 256-byte aligned start and usable bytes.
// While it lives, no other thread launches with that buffer.
struct Workspace {
    void* ptr;
    size_t bytes;
    std::unique_lock<std::mutex> hold;
};
Workspace workspace(const Tensor& on, size_t bytes);
void* workspace_if_any(int device);   // start of the buffer of (device, its current stream), or nullptr

// ---- operators (ops.cpp)
struct ScanOut {
    Tensor y, final_state, tail;
};
ScanOut scan_fused(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gate, const Tensor& lds,
                   const Tensor& rope, const Dyn& dyn, int64_t H, int64_t N, int64_t C, const Tensor& h0, double shortcut,
                   int64_t pos0, bool want_tail, int64_t flags, const Tensor& out, int64_t segs);
Tensor decode_step(const Tensor& state, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gate,
                   const Tensor& lds, const Tensor& rope, const Dyn& dyn, int64_t H, int64_t N, int64_t pos,
                   const Tensor& pos_dev, double shortcut, const Tensor& out, const Tensor& v_first, const Tensor& mix);
Tensor rms_norm(const Tensor& x, const Tensor& w, double eps);
Tensor groupnorm_gate(const Tensor& y, const Tensor& gw, const Tensor& gb, const Tensor& z, const Tensor& skip,
                      const Tensor& x_conv, int64_t groups, double eps, bool per_token);
Tensor conv1d_silu(const Tensor& x, const Tensor& w, const Tensor& b);
Tensor conv1d_silu_step(const Tensor& x, const Tensor& hist, const Tensor& w, const Tensor& b);

// ---- library products (gemm.cpp)
constexpr size_t kGemmWorkspace = 32u << 20;   // what the library is given by default on this architecture
Tensor gemm_workspace(const Tensor& on);
void gemm_raw(int device, void* out, int64_t ldo, const void* x, int64_t ldx, const void* w, const void* bias, int64_t rows, int64_t M,
              int64_t K, bool accumulate, void* workspace, void* stream);
void gemm(const Tensor& out, const Tensor& x, const Tensor& w, const Tensor& bias, bool accumulate, const Tensor& workspace);
Tensor linear(const Tensor& x, const Tensor& w, const Tensor& bias, const Tensor& workspace);

// ---- Python side helpers
struct Args {   // positional arguments of a METH_FASTCALL function
    PyObject* const* a;
    Py_ssize_t n, at = 0;
    PyObject* next() {
        if (at >= n) throw Error("too few arguments");
        return a[at++];
    }
    Tensor tensor(const char* name) {
        PyObject* o = next();
        if (!THPVariable_Check(o)) throw Error(std::string(name) + " must be a tensor");
        return THPVariable_Unpack(o);
    }
    Tensor tensor_or_none(const char* name) {
        PyObject* o = next();
        if (o == Py_None) return Tensor();
        if (!THPVariable_Check(o)) throw Error(std::string(name) + " must be a tensor or None");
        return THPVariable_Unpack(o);
    }
    double number() {
        const double v = PyFloat_AsDouble(next());
        if (v == -1.0 && PyErr_Occurred()) throw std::invalid_argument("number");
        return v;
    }
    int64_t integer() {
        PyObject* o = next();
        PyObject* i = PyLong_Check(o) ? (Py_INCREF(o), o) : PyNumber_Long(o);
        if (!i) throw std::invalid_argument("integer");
        const int64_t v = PyLong_AsLongLong(i);
        Py_DECREF(i);
        if (v == -1 && PyErr_Occurred()) throw std::invalid_argument("integer");
        return v;
    }
    bool flag() { return PyObject_IsTrue(next()) == 1; }
    Dyn dyn() {
        Dyn d;
        for (float& x : d.c) x = (float)number();
        return d;
    }
};

extern PyObject* g_error_type;
// Runs fn and turns C++ exceptions into Python ones.
template <typename F>
PyObject* guarded(F&& fn) {
    try {
        return fn();
    } catch (const Error& e) {
        PyErr_SetString(g_error_type ? g_error_type : PyExc_RuntimeError, e.what());
    } catch (const c10::OutOfMemoryError& e) {
        PyObject* t = PyObject_GetAttrString(PyImport_AddModule("torch"), "OutOfMemoryError");
        PyErr_SetString(t ? t : PyExc_RuntimeError, e.what_without_backtrace());
        Py_XDECREF(t);
    } catch (const c10::IndexError& e) {
        PyErr_SetString(PyExc_IndexError, e.what_without_backtrace());
    } catch (const c10::ValueError& e) {
        PyErr_SetString(PyExc_ValueError, e.what_without_backtrace());
    } catch (const c10::TypeError& e) {
        PyErr_SetString(PyExc_TypeError, e.what_without_backtrace());
    } catch (const c10::Error& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
    } catch (const std::exception& e) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}
// Runs fn without the interpreter's lock, so that other threads of the program go on while a pass is launched.
template <typename F>
auto without_gil(F&& fn) {
    struct Released {
        PyThreadState* state = PyEval_SaveThread();
        ~Released() { PyEval_RestoreThread(state); }
    } released;
    return fn();
}
inline PyObject* wrap(Tensor t) { return THPVariable_Wrap(std::move(t)); }

PyMethodDef* model_methods();   // lm.cpp
PyMethodDef* train_methods();   // train.cpp

}  // namespace cdssm_host
