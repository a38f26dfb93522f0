// CPython face of the call path a program takes once per transform: turbofft_b200.fft / ifft,
// Plan.__call__ on ordinary CUDA tensors, Plan.ft_status.
//
// A 16 x 1024-point transform keeps the GPU busy for 2.5 us; the interpreted form of this path
// (attribute reads, a key tuple, reshape, ctypes argument conversion) kept the caller busy for 15.
// Here a call reads the tensor's fields through ATen, looks the plan up in the SAME dictionary the
// Python side keeps, allocates the output and calls tfft_exec (Plan.__call__) or tfft_exec_ws (fft, ifft).  Whatever is not an ordinary call --
// a plan that does not exist yet, a tensor that is not on a GPU, not contiguous, lazily conjugated, of
// another type or length -- returns None, and the Python code does what it always did, errors included.
// What torch raises on the way (no memory for the output) leaves as torch's own exception.
// The module links nothing of the library: it is handed the addresses of the entries that _lib.py loaded.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>

#include <cstdint>
#include <vector>

namespace {

typedef int (*ExecFn)(void*, const void*, void*, void*);
typedef int (*ExecWsFn)(void*, const void*, void*, void*, void*);
typedef size_t (*ScratchFn)(void*);
typedef int (*StatusFn)(void*, int*, int*, int, int*, int, int*);
typedef int (*InfoFn)(void*, int*);
typedef int (*ShapeFn)(void*, int*, long long*, int*, int*);

ExecFn g_exec = nullptr;
ExecWsFn g_exec_ws = nullptr;
ScratchFn g_scratch_bytes = nullptr;
StatusFn g_status = nullptr;
InfoFn g_info = nullptr;
ShapeFn g_shape = nullptr;
PyObject* g_plans = nullptr;  // turbofft_b200._plan_cache
PyObject *s_h, *s_value, *s_strided;

// complex64 -> 0, complex128 -> 1 (the C ABI's dtype codes), anything else -> -1
int type_code(const at::Tensor& x) {
    const auto t = x.scalar_type();
    return t == at::kComplexFloat ? 0 : (t == at::kComplexDouble ? 1 : -1);
}

// A plain torch.Tensor whose memory is its value: no subclass, no lazy conjugate or negative bit (x.conj() is a
// contiguous view of x's memory; the Python path applies the bit first)
bool ordinary(PyObject* o) {
    if (!THPVariable_CheckExact(o)) return false;
    const at::Tensor& t = THPVariable_Unpack(o);
    return !t.is_conj() && !t.is_neg();
}

// the tfft_plan behind a Plan object, null for a destroyed one
void* plan_handle(PyObject* plan) {
    PyObject* h = PyObject_GetAttr(plan, s_h);
    PyObject* v = h ? PyObject_GetAttr(h, s_value) : nullptr;
    void* p = v && PyLong_Check(v) ? PyLong_AsVoidPtr(v) : nullptr;
    Py_XDECREF(v);
    Py_XDECREF(h);
    if (PyErr_Occurred()) PyErr_Clear();
    return p;
}

// Allocates the output (unless the caller brought one) and runs the plan on the current stream of the
// tensor's device.  None when the library reports an error: the Python path repeats the call and raises.
// shared: a plan of the cache, which callers on several streams and threads run at the same time; the intermediate
// buffer is this call's own, from the caching allocator.  It goes back when the launches are queued and can then only
// be given to later work of the same stream (and, inside a capture, of the same graph).
PyObject* execute(void* plan, bool shared, const at::Tensor& x, PyObject* out_obj) {
    at::Tensor y;
    if (out_obj == Py_None) y = at::detail::empty_cuda(x.sizes(), x.scalar_type(), x.device(), c10::nullopt);
    else y = THPVariable_Unpack(out_obj);
    void* stream = c10::cuda::getCurrentCUDAStream(x.device().index()).stream();
    int rc;
    const void* in = x.const_data_ptr();
    void* out = y.mutable_data_ptr();
    at::DataPtr ws;
    if (const size_t bytes = shared ? g_scratch_bytes(plan) : 0) {
        c10::cuda::CUDAGuard guard(x.device());
        ws = c10::cuda::CUDACachingAllocator::get()->allocate(bytes);
    }
    Py_BEGIN_ALLOW_THREADS
    rc = shared ? g_exec_ws(plan, in, out, ws.get(), stream) : g_exec(plan, in, out, stream);
    Py_END_ALLOW_THREADS
    if (rc != 0) Py_RETURN_NONE;
    if (out_obj != Py_None) {
        Py_INCREF(out_obj);
        return out_obj;
    }
    return THPVariable_Wrap(std::move(y));
}

struct KeyFields {
    int64_t device, logn, batch, inner, thread_bs;  // inner: 0 for the last axis
    double expo;
    int64_t flags;
    bool operator==(const KeyFields& o) const {
        return device == o.device && logn == o.logn && batch == o.batch && inner == o.inner && thread_bs == o.thread_bs &&
               expo == o.expo && flags == o.flags;
    }
};
struct KeySlot {
    KeyFields fields;
    PyObject* key;
};
constexpr int kKeySlots = 64;
KeySlot g_keys[kKeySlots];  // under the interpreter lock

// The key turbofft_b200.fft files this call's plan under, kept in `slot`
PyObject* make_key(PyObject* const* a, const KeyFields& f, int64_t outer, int code, int ft, int err, int inverse, KeySlot& slot) {
    PyObject* key = f.inner ? Py_BuildValue("(OLLLLiOO)", s_strided, (long long)f.device, (long long)f.logn, (long long)f.inner,
                                            (long long)outer, code, inverse ? Py_True : Py_False, a[5])
                            : Py_BuildValue("(LLLiOOOOO)", (long long)f.device, (long long)f.logn, (long long)f.batch, code,
                                            ft ? Py_True : Py_False, err ? Py_True : Py_False, a[3], inverse ? Py_True : Py_False, a[5]);
    if (!key) return nullptr;
    Py_XDECREF(slot.key);
    slot.fields = f;
    slot.key = key;
    return key;
}

// torch's own translation, without the buffer for warnings that its macro sets up on every call
PyObject* raise_as_torch_does() {
    torch::translate_exception_to_python(std::current_exception());
    return nullptr;
}

// fft(x, ft, err, thread_bs, out, norm_exponent, inverse, dim): the transform along one axis, or None
PyObject* fast_fft(PyObject*, PyObject* const* a, Py_ssize_t n) {
    try {
        if (n != 8 || !g_exec || !ordinary(a[0]) || !PyLong_Check(a[7])) Py_RETURN_NONE;
        const at::Tensor& x = THPVariable_Unpack(a[0]);
        const int code = type_code(x);
        const int64_t rank = x.dim();
        int overflow = 0;  // the Python path takes an axis of any size modulo the rank
        int64_t dim = PyLong_AsLongLongAndOverflow(a[7], &overflow);
        if (overflow) Py_RETURN_NONE;
        if (dim < 0) dim += rank;
        if (code < 0 || !x.is_cuda() || dim < 0 || dim >= rank || x.numel() == 0 || !x.is_contiguous()) Py_RETURN_NONE;
        const int64_t len = x.size(dim);
        if (len < 2 || (len & (len - 1))) Py_RETURN_NONE;
        const int logn = __builtin_ctzll((unsigned long long)len);
        if (a[4] != Py_None) {
            if (!ordinary(a[4])) Py_RETURN_NONE;
            const at::Tensor& y = THPVariable_Unpack(a[4]);
            if (!y.is_cuda() || !y.is_contiguous() || y.scalar_type() != x.scalar_type() || y.sizes() != x.sizes()) Py_RETURN_NONE;
        }
        const int ft = PyObject_IsTrue(a[1]), err = PyObject_IsTrue(a[2]), inverse = PyObject_IsTrue(a[6]);
        if (ft < 0 || err < 0 || inverse < 0) return nullptr;
        const bool strided = dim != rank - 1;
        if (strided && (ft || err || a[4] != Py_None)) Py_RETURN_NONE;
        int64_t inner = 1;
        for (int64_t d = dim + 1; d < rank; ++d) inner *= x.size(d);
        // a program repeats a handful of shapes: their key tuples are kept, the plans stay the dictionary's
        const int64_t thread_bs = PyLong_Check(a[3]) ? PyLong_AsLongLong(a[3]) : -1;
        const double expo = PyFloat_Check(a[5]) ? PyFloat_AS_DOUBLE(a[5]) : 2.0;
        if (thread_bs < 0 || expo > 1.0) {
            PyErr_Clear();
            Py_RETURN_NONE;
        }
        const KeyFields fields = {x.device().index(), logn, x.numel() / len, strided ? inner : 0, thread_bs, expo,
                                  code | ft << 1 | err << 2 | inverse << 3};
        KeySlot& slot = g_keys[(fields.batch * 31 + fields.logn * 7 + fields.flags) & (kKeySlots - 1)];
        PyObject* key = slot.key && slot.fields == fields ? slot.key : nullptr;
        if (!key) key = make_key(a, fields, x.numel() / (len * inner), code, ft, err, inverse, slot);
        if (!key) return nullptr;
        PyObject* found = PyDict_GetItemWithError(g_plans, key);  // borrowed
        if (!found) {
            if (PyErr_Occurred()) return nullptr;
            Py_RETURN_NONE;
        }
        Py_INCREF(found);
        THPObjectPtr plan(found);  // held while the interpreter lock is released
        void* h = plan_handle(found);
        if (!h) Py_RETURN_NONE;
        return execute(h, true, x, a[4]);
    } catch (...) {
        return raise_as_torch_does();
    }
}

// exec(plan, x, out): Plan.__call__, or None
PyObject* fast_exec(PyObject*, PyObject* const* a, Py_ssize_t n) {
    try {
        if (n != 3 || !g_exec || !ordinary(a[1]) || (a[2] != Py_None && !ordinary(a[2]))) Py_RETURN_NONE;
        const at::Tensor& x = THPVariable_Unpack(a[1]);
        void* h = plan_handle(a[0]);
        int logn, dtype, device;
        long long batch;
        if (!h || g_shape(h, &logn, &batch, &dtype, &device) != 0) Py_RETURN_NONE;
        if (!x.is_cuda() || type_code(x) != dtype || x.numel() != (batch << logn) || x.device().index() != device || !x.is_contiguous())
            Py_RETURN_NONE;
        if (a[2] != Py_None) {
            const at::Tensor& y = THPVariable_Unpack(a[2]);
            if (!y.is_cuda() || !y.is_contiguous() || y.scalar_type() != x.scalar_type() || y.numel() != x.numel()) Py_RETURN_NONE;
        }
        return execute(h, false, x, a[2]);
    } catch (...) {
        return raise_as_torch_does();
    }
}

// ft_status(plan, launch): (detected, corrected, [located per block]) with one library call, or the negative status
PyObject* ft_status(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 2 || !PyLong_Check(a[1])) {
        PyErr_SetString(PyExc_TypeError, "ft_status(plan, launch)");
        return nullptr;
    }
    void* h = plan_handle(a[0]);
    const int launch = (int)PyLong_AsUnsignedLongLongMask(a[1]);  // as ctypes passes a C int
    int info[19] = {0}, nd = 0, nc = 0, nb = 0, rc = h ? g_info(h, info) : -1;
    if (rc == 0) {
        const int last = launch < 0 ? info[0] - 1 : launch;
        std::vector<int> located(last < info[0] ? (size_t)info[1 + 6 * last + 3] : 0);  // the launch's grid
        Py_BEGIN_ALLOW_THREADS
        rc = g_status(h, &nd, &nc, launch, located.data(), (int)located.size(), &nb);
        Py_END_ALLOW_THREADS
        if (rc == 0) {
            PyObject* list = PyList_New(nb);
            if (!list) return nullptr;
            for (int i = 0; i < nb; ++i) PyList_SET_ITEM(list, i, PyLong_FromLong(located[i]));
            return Py_BuildValue("iiN", nd, nc, list);
        }
    }
    return PyLong_FromLong(rc);
}

// bind(addresses of tfft_exec, _ft_status, _plan_info, _plan_shape, _exec_ws and _scratch_bytes, plan dictionary)
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 7 || !PyDict_Check(a[6])) {
        PyErr_SetString(PyExc_TypeError, "bind(exec, ft_status, plan_info, plan_shape, exec_ws, scratch_bytes, dict)");
        return nullptr;
    }
    void* p[6];
    for (int i = 0; i < 6; ++i) {
        p[i] = PyLong_AsVoidPtr(a[i]);
        if (!p[i] && PyErr_Occurred()) return nullptr;
    }
    Py_INCREF(a[6]);
    Py_XDECREF(g_plans);
    g_plans = a[6];
    g_exec = (ExecFn)p[0];
    g_status = (StatusFn)p[1];
    g_info = (InfoFn)p[2];
    g_shape = (ShapeFn)p[3];
    g_exec_ws = (ExecWsFn)p[4];
    g_scratch_bytes = (ScratchFn)p[5];
    Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"fft", (PyCFunction)(void (*)(void))fast_fft, METH_FASTCALL, nullptr},
    {"exec", (PyCFunction)(void (*)(void))fast_exec, METH_FASTCALL, nullptr},
    {"ft_status", (PyCFunction)(void (*)(void))ft_status, METH_FASTCALL, nullptr},
    {"bind", (PyCFunction)(void (*)(void))bind, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_torch_binding", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_binding(void) {
    s_h = PyUnicode_InternFromString("_h");
    s_value = PyUnicode_InternFromString("value");
    s_strided = PyUnicode_InternFromString("strided");
    return PyModule_Create(&kModule);
}
