// The operator's path from a Python call to the kernels' launches, natively: argument checks,
// the output and scratch tensors, the stream, the launch.  A call of a dozen microseconds of GPU
// work is bound by this path when calls are issued back to back; through torch's Python API and
// ctypes it took 17 us a call, here it takes about 5.
//
// Every entry returns None for arguments it does not take (wrong shapes, types, devices, a
// library that is not bound yet): the Python wrapper then finds out what is wrong and raises the
// documented error.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/DeviceGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <dlfcn.h>

#include <cmath>
#include <exception>
#include <vector>

#include "../../include/flash_colsum_b200.h"
#include "host_api.h"

namespace {

FcsRunCallFn g_run_call = nullptr;
FcsRunHostCallFn g_run_host_call = nullptr;
FcsSelectTopkFn g_select_topk = nullptr;
FcsSelectThresholdFn g_select_threshold = nullptr;
FcsLastErrorFn g_last_error = nullptr;

constexpr int MAX_DEVICES = 64;
int* g_status[MAX_DEVICES] = {nullptr};   // the device status words (owned by the Python package)

// The launches run without the interpreter lock: they may wait for room in the launch queue.
struct WithoutGil {
    PyThreadState* state;
    WithoutGil() : state(PyEval_SaveThread()) {}
    ~WithoutGil() { PyEval_RestoreThread(state); }
};

PyObject* raise_library_error(int rc) {
    PyErr_Format(PyExc_RuntimeError, "flash_colsum_b200: %s (code %d)", g_last_error ? g_last_error() : "", rc);
    return nullptr;
}

at::Tensor empty_f32(int64_t rows, int64_t cols, c10::Device dev) {
    const int64_t size[2] = {rows, cols};
    return at::detail::empty_cuda(c10::IntArrayRef(size, 2), at::kFloat, dev, std::nullopt);
}

// Scratch of one call; freed when the call returns (the caching allocator hands it out again in
// stream order only).  What the allocator throws does not pass through the library, which has copies
// in flight to wait for: it is kept, and thrown again by `rethrow` once the library has returned.
struct Scratch {
    c10::Device dev;
    std::vector<at::Tensor> held;
    std::exception_ptr error;
    static void* alloc(void* ctx, size_t bytes) noexcept {
        Scratch* s = static_cast<Scratch*>(ctx);
        try {
            const int64_t size[1] = {static_cast<int64_t>(bytes)};
            s->held.push_back(at::detail::empty_cuda(c10::IntArrayRef(size, 1), at::kByte, s->dev, std::nullopt));
            return s->held.back().mutable_data_ptr();
        } catch (...) {
            s->error = std::current_exception();
            return nullptr;
        }
    }
    void rethrow() const {
        if (error) std::rethrow_exception(error);
    }
};

int dtype_code(at::ScalarType t) {
    return t == at::kHalf ? FCS_DTYPE_FP16 : t == at::kBFloat16 ? FCS_DTYPE_BF16 : t == at::kFloat ? FCS_DTYPE_FP32 : -1;
}

// Unit inner stride, positive outer strides in multiples of 16 bytes, 16-byte aligned base.  The
// stride of an axis of one entry says nothing; the contiguous one stands in for it.
void kernel_strides(const at::Tensor& t, int64_t (&st)[3]) {
    int64_t dense = t.size(3);
    for (int i = 2; i >= 0; --i) {
        st[i] = t.size(i) > 1 ? t.stride(i) : dense;
        dense *= t.size(i);
    }
}
bool kernel_ready(const at::Tensor& t) {
    int64_t st[3];
    kernel_strides(t, st);
    const int64_t granule = 16 / t.element_size();
    return t.stride(3) == 1 && st[0] > 0 && st[1] > 0 && st[2] > 0 && ((st[0] | st[1] | st[2]) & (granule - 1)) == 0 &&
           (reinterpret_cast<uintptr_t>(t.const_data_ptr()) & 15) == 0;
}

bool usable(PyObject* o) { return THPVariable_Check(o); }

// One call on checked operands.  Returns a new reference, or NULL with an exception set.
PyObject* run(at::Tensor q, at::Tensor k, double scale, bool causal, int k_past, int cls_n, int h_norm) {
    const c10::Device dev = q.device();
    at::Tensor out;
    int rc;
    {
        WithoutGil nogil;
        const c10::DeviceGuard guard(dev);
        if (!kernel_ready(q)) q = q.contiguous();
        if (!kernel_ready(k)) k = k.contiguous();
        FcsCall c;
        c.B = (int)q.size(0);
        c.H = (int)q.size(1);
        c.Sq = (int)q.size(2);
        c.Sk = (int)k.size(2);
        c.D = (int)q.size(3);
        out = empty_f32(c.B, c.Sk, dev);
        c.q = q.const_data_ptr();
        c.k = k.const_data_ptr();
        c.out = static_cast<float*>(out.mutable_data_ptr());
        c.out_ld = c.Sk;
        c.dtype = dtype_code(q.scalar_type());
        kernel_strides(q, c.q_stride);
        kernel_strides(k, c.k_stride);
        c.scale = (float)scale;
        c.causal = causal ? 1 : 0;
        c.k_past = k_past;
        c.cls_n = cls_n;
        c.h_norm = h_norm;
        c.status = g_status[dev.index()];
        c.stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
        Scratch scratch{dev, {}, nullptr};
        c.alloc = &Scratch::alloc;
        c.alloc_ctx = &scratch;
        rc = g_run_call(&c);
        scratch.rethrow();
    }
    if (rc != FCS_OK) return raise_library_error(rc);
    return THPVariable_Wrap(std::move(out));
}

// Whether the kernels take this pair of operands: CUDA tensors of one device whose status word is
// known, 4-D, no empty axis, one supported type, matching batch, heads and head dimension.
bool operands_ok(const at::Tensor& q, const at::Tensor& k) {
    if (q.dim() != 4 || k.dim() != 4 || !q.is_cuda() || q.device() != k.device()) return false;
    const int idx = q.device().index();
    if (idx < 0 || idx >= MAX_DEVICES || !g_status[idx]) return false;
    if (q.scalar_type() != k.scalar_type() || dtype_code(q.scalar_type()) < 0) return false;
    const auto a = q.sizes(), b = k.sizes();
    if (a[0] != b[0] || a[1] != b[1] || a[3] != b[3] || a[3] < 8 || a[3] > 128 || a[3] % 8) return false;
    for (int i = 0; i < 4; ++i)
        if (a[i] <= 0 || b[i] <= 0 || a[i] > 0x7fffffffLL || b[i] > 0x7fffffffLL) return false;
    return g_run_call != nullptr;
}

double scale_or_default(PyObject* o, const at::Tensor& q) {
    return o == Py_None ? 1.0 / std::pow((double)q.size(3), 0.5) : PyFloat_AsDouble(o);
}

// colsum(query, key, scale, is_causal, cls_len): `flash_colsum`'s rules
PyObject* py_colsum(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 5 || !usable(args[0]) || !usable(args[1])) Py_RETURN_NONE;
    const at::Tensor& q = THPVariable_Unpack(args[0]);
    const at::Tensor& k = THPVariable_Unpack(args[1]);
    if (!operands_ok(q, k)) Py_RETURN_NONE;
    const int causal = PyObject_IsTrue(args[3]);
    if (causal < 0) return nullptr;
    int cls_n = -1;
    if (args[4] != Py_None) {
        if (causal || !PyLong_CheckExact(args[4])) Py_RETURN_NONE;
        int overflow = 0;
        const long long v = PyLong_AsLongLongAndOverflow(args[4], &overflow);
        if (overflow || v <= 0 || v > 0x7fffffffLL) Py_RETURN_NONE;
        cls_n = (int)v;
    }
    if (causal ? q.size(0) != 1 : q.size(2) != k.size(2)) Py_RETURN_NONE;
    const double scale = scale_or_default(args[2], q);
    if (PyErr_Occurred()) return nullptr;
    return run(q, k, scale, causal != 0, -1, cls_n, 0);
    END_HANDLE_TH_ERRORS
}

// launch(query, key, scale, is_causal, k_past, cls_n, h_norm): checked arguments, -1 / 0 for defaults
PyObject* py_launch(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 7 || !usable(args[0]) || !usable(args[1])) Py_RETURN_NONE;
    const at::Tensor& q = THPVariable_Unpack(args[0]);
    const at::Tensor& k = THPVariable_Unpack(args[1]);
    if (!operands_ok(q, k)) Py_RETURN_NONE;
    const double scale = scale_or_default(args[2], q);
    const int causal = PyObject_IsTrue(args[3]);
    const long k_past = PyLong_AsLong(args[4]), cls_n = PyLong_AsLong(args[5]), h_norm = PyLong_AsLong(args[6]);
    if (PyErr_Occurred()) return nullptr;
    if (!causal && q.size(2) != k.size(2)) Py_RETURN_NONE;
    const long most = 0x7fffffffL;
    return run(q, k, scale, causal != 0, (int)(k_past < most ? k_past : most), (int)(cls_n < most ? cls_n : most),
               (int)h_norm);
    END_HANDLE_TH_ERRORS
}

// host(query, key, scale, is_causal, cls_len, device index, batch_chunk or 0) -> host tensor
PyObject* py_host(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 7 || !g_run_host_call || !usable(args[0]) || !usable(args[1])) Py_RETURN_NONE;
    const at::Tensor& q = THPVariable_Unpack(args[0]);
    const at::Tensor& k = THPVariable_Unpack(args[1]);
    const int causal = PyObject_IsTrue(args[3]);
    const long idx = PyLong_AsLong(args[5]), batch_chunk = PyLong_AsLong(args[6]);
    if (PyErr_Occurred()) return nullptr;
    if (idx < 0 || idx >= MAX_DEVICES || !g_status[idx] || batch_chunk < 0) Py_RETURN_NONE;
    if (q.dim() != 4 || k.dim() != 4 || !q.is_cpu() || !k.is_cpu() || !q.is_contiguous() || !k.is_contiguous()) Py_RETURN_NONE;
    if (q.scalar_type() != k.scalar_type() || dtype_code(q.scalar_type()) < 0) Py_RETURN_NONE;
    const auto a = q.sizes(), b = k.sizes();
    if (a[0] != b[0] || a[1] != b[1] || a[3] != b[3] || a[3] < 8 || a[3] > 128 || a[3] % 8) Py_RETURN_NONE;
    for (int i = 0; i < 4; ++i)
        if (a[i] <= 0 || b[i] <= 0 || a[i] > 0x7fffffffLL || b[i] > 0x7fffffffLL) Py_RETURN_NONE;
    if (causal ? a[0] != 1 : a[2] != b[2]) Py_RETURN_NONE;
    int cls_n = -1;
    if (args[4] != Py_None) {
        if (causal || !PyLong_CheckExact(args[4])) Py_RETURN_NONE;
        int overflow = 0;
        const long long v = PyLong_AsLongLongAndOverflow(args[4], &overflow);
        if (overflow || v <= 0 || v > 0x7fffffffLL) Py_RETURN_NONE;
        cls_n = (int)v;
    }
    const double scale = scale_or_default(args[2], q);
    if (PyErr_Occurred()) return nullptr;
    at::Tensor host_out;
    int rc;
    {
        WithoutGil nogil;
        const c10::Device dev(c10::kCUDA, (c10::DeviceIndex)idx);
        const c10::DeviceGuard guard(dev);
        const at::Tensor dq = at::detail::empty_cuda(a, q.scalar_type(), dev, std::nullopt);
        const at::Tensor dk = at::detail::empty_cuda(b, k.scalar_type(), dev, std::nullopt);
        const at::Tensor out = empty_f32(a[0], b[2], dev);
        host_out = at::empty({a[0], b[2]}, at::TensorOptions().dtype(at::kFloat).device(at::kCPU));
        FcsHostCall hc;
        FcsCall& c = hc.call;
        c.B = (int)a[0];
        c.H = (int)a[1];
        c.Sq = (int)a[2];
        c.Sk = (int)b[2];
        c.D = (int)a[3];
        c.q = dq.const_data_ptr();
        c.k = dk.const_data_ptr();
        c.out = static_cast<float*>(out.mutable_data_ptr());
        c.out_ld = c.Sk;
        c.dtype = dtype_code(q.scalar_type());
        kernel_strides(dq, c.q_stride);
        kernel_strides(dk, c.k_stride);
        c.scale = (float)scale;
        c.causal = causal;
        c.k_past = -1;
        c.cls_n = cls_n;
        c.h_norm = 0;
        c.status = g_status[idx];
        c.stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)idx).stream();
        Scratch scratch{dev, {}, nullptr};
        c.alloc = &Scratch::alloc;
        c.alloc_ctx = &scratch;
        hc.host_q = q.const_data_ptr();
        hc.host_k = k.const_data_ptr();
        hc.host_out = static_cast<float*>(host_out.mutable_data_ptr());
        hc.batch_chunk = (int)(batch_chunk < 0x7fffffffL ? batch_chunk : 0x7fffffffL);
        rc = g_run_host_call(&hc);
        scratch.rethrow();
    }
    if (rc != FCS_OK) return raise_library_error(rc);
    return THPVariable_Wrap(std::move(host_out));
    END_HANDLE_TH_ERRORS
}

bool means_ok(const at::Tensor& t) {
    return t.dim() == 2 && t.scalar_type() == at::kFloat && t.is_cuda();
}

PyObject* pair(at::Tensor a, at::Tensor b) {
    PyObject* t = PyTuple_New(2);
    if (!t) return nullptr;
    PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(a)));
    PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(std::move(b)));
    return t;
}

// topk(colsum, k) -> (values, indices)
PyObject* py_topk(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 2 || !g_select_topk || !usable(args[0]) || !PyLong_Check(args[1])) Py_RETURN_NONE;
    at::Tensor x = THPVariable_Unpack(args[0]);
    if (!means_ok(x)) Py_RETURN_NONE;
    const long long k = PyLong_AsLongLong(args[1]);
    if (PyErr_Occurred() || k < 1 || k > x.size(1)) { PyErr_Clear(); Py_RETURN_NONE; }
    const c10::Device dev = x.device();
    at::Tensor idx, val;
    int rc;
    {
        WithoutGil nogil;
        const c10::DeviceGuard guard(dev);
        if (x.stride(1) != 1 || x.stride(0) < x.size(1)) x = x.contiguous();
        const int64_t size[2] = {x.size(0), (int64_t)k};
        idx = at::detail::empty_cuda(c10::IntArrayRef(size, 2), at::kInt, dev, std::nullopt);
        val = empty_f32(size[0], size[1], dev);
        rc = g_select_topk(static_cast<const float*>(x.const_data_ptr()), x.size(0) > 1 ? x.stride(0) : x.size(1),
                           (int)x.size(0), (int)x.size(1), (int)k, static_cast<int*>(idx.mutable_data_ptr()),
                           static_cast<float*>(val.mutable_data_ptr()),
                           c10::cuda::getCurrentCUDAStream(dev.index()).stream());
    }
    if (rc != FCS_OK) return raise_library_error(rc);
    return pair(std::move(val), std::move(idx));
    END_HANDLE_TH_ERRORS
}

// threshold(colsum, threshold, relative) -> (indices, counts)
PyObject* py_threshold(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 3 || !g_select_threshold || !usable(args[0])) Py_RETURN_NONE;
    at::Tensor x = THPVariable_Unpack(args[0]);
    if (!means_ok(x)) Py_RETURN_NONE;
    const double thr = PyFloat_AsDouble(args[1]);
    const int relative = PyObject_IsTrue(args[2]);
    if (PyErr_Occurred()) return nullptr;
    if (std::isnan(thr)) Py_RETURN_NONE;
    const c10::Device dev = x.device();
    at::Tensor idx, cnt;
    int rc;
    {
        WithoutGil nogil;
        const c10::DeviceGuard guard(dev);
        if (x.stride(1) != 1 || x.stride(0) < x.size(1)) x = x.contiguous();
        const int64_t size[2] = {x.size(0), x.size(1)};
        idx = at::detail::empty_cuda(c10::IntArrayRef(size, 2), at::kInt, dev, std::nullopt);
        cnt = at::detail::empty_cuda(c10::IntArrayRef(size, 1), at::kInt, dev, std::nullopt);
        rc = g_select_threshold(static_cast<const float*>(x.const_data_ptr()),
                                x.size(0) > 1 ? x.stride(0) : x.size(1), (int)x.size(0), (int)x.size(1), (float)thr,
                                relative, static_cast<int*>(idx.mutable_data_ptr()),
                                static_cast<int*>(cnt.mutable_data_ptr()),
                                c10::cuda::getCurrentCUDAStream(dev.index()).stream());
    }
    if (rc != FCS_OK) return raise_library_error(rc);
    return pair(std::move(idx), std::move(cnt));
    END_HANDLE_TH_ERRORS
}

// bind(handle): the entry points of the loaded CUDA library (a dlopen handle)
PyObject* py_bind(PyObject*, PyObject* arg) {
    void* h = PyLong_AsVoidPtr(arg);
    if (PyErr_Occurred()) return nullptr;
    auto sym = [&](const char* name) { return dlsym(h, name); };
    g_last_error = reinterpret_cast<FcsLastErrorFn>(sym("fcs_last_error"));
    g_select_topk = reinterpret_cast<FcsSelectTopkFn>(sym("fcs_select_topk"));
    g_select_threshold = reinterpret_cast<FcsSelectThresholdFn>(sym("fcs_select_threshold"));
    g_run_call = reinterpret_cast<FcsRunCallFn>(sym("fcs_run_call"));
    g_run_host_call = reinterpret_cast<FcsRunHostCallFn>(sym("fcs_run_host_call"));
    if (!g_last_error || !g_select_topk || !g_select_threshold || !g_run_call || !g_run_host_call) {
        PyErr_SetString(PyExc_RuntimeError, "flash_colsum_b200: the CUDA library lacks an entry point of this binding");
        return nullptr;
    }
    Py_RETURN_NONE;
}

// set_status(device_index, address): the status word that this device's calls report into
PyObject* py_set_status(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 2) { PyErr_SetString(PyExc_TypeError, "set_status(device_index, address)"); return nullptr; }
    const long idx = PyLong_AsLong(args[0]);
    void* p = PyLong_AsVoidPtr(args[1]);
    if (PyErr_Occurred()) return nullptr;
    if (idx >= 0 && idx < MAX_DEVICES) g_status[idx] = static_cast<int*>(p);
    Py_RETURN_NONE;
}

template <typename F>
constexpr PyCFunction fast(F f) { return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(f)); }

PyMethodDef g_methods[] = {
    {"colsum", fast(py_colsum), METH_FASTCALL, nullptr},
    {"launch", fast(py_launch), METH_FASTCALL, nullptr},
    {"host", fast(py_host), METH_FASTCALL, nullptr},
    {"topk", fast(py_topk), METH_FASTCALL, nullptr},
    {"threshold", fast(py_threshold), METH_FASTCALL, nullptr},
    {"bind", py_bind, METH_O, nullptr},
    {"set_status", fast(py_set_status), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_fcs_torch", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fcs_torch(void) { return PyModule_Create(&g_module); }
