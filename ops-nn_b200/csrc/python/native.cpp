// CPython module behind aclnn.py and torch_api.py: tensor descriptors made straight from torch tensors, and both phases of a call with
// its output and workspace in one native step.
//
// What bounds a small call is the host: through ctypes, a W4A16 call on a 4096 x 4096 weight spent 52 us of Python on 12 us of GPU work
// (five descriptors with three ctypes arrays each, two argument conversions of eleven pointers, two torch.empty); here it is 5 us. The
// descriptors live on the stack, the output comes from torch's CUDA allocator without the dispatcher, and the workspace is a block of
// the same allocator on the call's stream that goes back to it when the launches are enqueued - the lifetime a torch.empty in the
// wrapper would have.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <structmember.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include "aclnnop/aclnn_dynamic_mx_quant.h"
#include "aclnnop/aclnn_quant_matmul_v5.h"
#include "aclnnop/aclnn_quant_matmul_weight_nz.h"
#include "aclnnop/aclnn_weight_quant_batch_matmul_nz.h"
#include "aclnnop/aclnn_weight_quant_batch_matmul_v2.h"
#include "aclnnop/aclnn_weight_quant_batch_matmul_v3.h"
#include "internal.h"

namespace {

PyObject* g_codes = nullptr;       // aclnn.DTYPE_BY_NAME
PyObject* g_call_error = nullptr;  // aclnn.AclnnError(api, status)

// Thrown with a Python exception set; caught at the module's functions.
struct PyFail {};

template <typename F>
PyObject* guarded(F&& f)
{
    try {
        return f();
    } catch (const PyFail&) {
    } catch (const c10::OutOfMemoryError& e) {
        PyObject* torch = PyImport_ImportModule("torch");
        PyObject* type = torch != nullptr ? PyObject_GetAttrString(torch, "OutOfMemoryError") : nullptr;
        if (type != nullptr) PyErr_SetString(type, e.what_without_backtrace());
        Py_XDECREF(type);
        Py_XDECREF(torch);
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}

// Python's lock given up while the library plans and launches and torch's allocator works: a launch waits where the stream's queue is full,
// an allocation in cudaMalloc, a first call for the module to load, and other threads of the program go on meanwhile. Comes back on every
// way out, so that errors are raised with the lock held.
struct Unlocked {
    PyThreadState* state = PyEval_SaveThread();
    ~Unlocked() { PyEval_RestoreThread(state); }
    Unlocked() = default;
    Unlocked(const Unlocked&) = delete;
    Unlocked& operator=(const Unlocked&) = delete;
};

[[noreturn]] void fail_call(const char* api, aclnnStatus status)
{
    PyObject* err = PyObject_CallFunction(g_call_error, "si", api, (int)status);
    if (err != nullptr) {
        PyErr_SetObject(g_call_error, err);
        Py_DECREF(err);
    }
    throw PyFail{};
}

void check_call(const char* api, aclnnStatus status)
{
    if (status != ACLNN_SUCCESS) fail_call(api, status);
}

int64_t as_int(PyObject* o)
{
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) {
        if (!PyErr_ExceptionMatches(PyExc_TypeError)) throw PyFail{};
        PyErr_Clear();
        PyObject* n = PyNumber_Long(o);
        if (n == nullptr) throw PyFail{};
        const long long w = PyLong_AsLongLong(n);
        Py_DECREF(n);
        if (w == -1 && PyErr_Occurred()) throw PyFail{};
        return w;
    }
    return v;
}

opsnn::Dims as_dims(PyObject* o)
{
    PyObject* seq = PySequence_Fast(o, "a sequence of extents is expected");
    if (seq == nullptr) throw PyFail{};
    opsnn::Dims d;
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(seq);
    if (n > 8) {
        Py_DECREF(seq);
        PyErr_SetString(PyExc_ValueError, "a tensor descriptor has at most 8 dims");
        throw PyFail{};
    }
    try {
        for (Py_ssize_t i = 0; i < n; ++i) d.push_back(as_int(PySequence_Fast_GET_ITEM(seq, i)));
    } catch (const PyFail&) {
        Py_DECREF(seq);
        throw;
    }
    Py_DECREF(seq);
    return d;
}

opsnn::Dims as_strides(PyObject* o, const opsnn::Dims& shape)  // what is missing is 0
{
    opsnn::Dims d = as_dims(o);
    if (d.size() > shape.size()) {
        PyErr_SetString(PyExc_IndexError, "more strides than dims");
        throw PyFail{};
    }
    d.resize(shape.size());
    return d;
}

int code_of(PyObject* dtype)  // a name of aclnn.DTYPE_BY_NAME or an aclDataType value
{
    if (PyUnicode_Check(dtype)) {
        PyObject* v = PyDict_GetItemWithError(g_codes, dtype);
        if (v == nullptr) {
            if (!PyErr_Occurred()) PyErr_SetObject(PyExc_KeyError, dtype);
            throw PyFail{};
        }
        dtype = v;
    }
    return (int)as_int(dtype);
}

int code_of(at::ScalarType type)
{
    switch (type) {
        case at::kFloat: return ACL_FLOAT;
        case at::kHalf: return ACL_FLOAT16;
        case at::kBFloat16: return ACL_BF16;
        case at::kChar: return ACL_INT8;
        case at::kInt: return ACL_INT32;
        case at::kByte: return ACL_UINT8;
        case at::kLong: return ACL_INT64;
        case at::ScalarType::UInt64: return ACL_UINT64;
        case at::ScalarType::Float8_e4m3fn: return ACL_FLOAT8_E4M3FN;
        case at::ScalarType::Float8_e5m2: return ACL_FLOAT8_E5M2;
        default: break;
    }
    PyErr_Format(PyExc_KeyError, "torch.%s has no aclDataType", c10::toString(type));
    throw PyFail{};
}
int code_of(const at::Tensor& t) { return code_of(t.scalar_type()); }

const at::Tensor* tensor_of(PyObject* o, const char* what)  // nullptr for None
{
    if (o == Py_None) return nullptr;
    if (!THPVariable_Check(o)) {
        PyErr_Format(PyExc_TypeError, "%s must be a torch tensor, got %s", what, Py_TYPE(o)->tp_name);
        throw PyFail{};
    }
    return &THPVariable_Unpack(o);
}

void fill(aclTensor* d, const at::Tensor& t, int code)
{
    if (t.dim() > 8) {
        PyErr_SetString(PyExc_ValueError, "a tensor descriptor has at most 8 dims");
        throw PyFail{};
    }
    const auto sizes = t.sizes(), strides = t.strides();
    d->shape.assign(sizes.data(), sizes.data() + sizes.size());
    d->strides.assign(strides.data(), strides.data() + strides.size());
    d->storage_shape = d->shape;
    d->dtype = (aclDataType)code;
    d->data = t.data_ptr();
}

// The descriptor of an optional argument: `dtype` (None, a name or a code) names the element type of storage that torch cannot type
// itself; of 4-bit types two elements lie in each stored byte along the axis with stride 1.
const aclTensor* describe(PyObject* o, PyObject* dtype, const char* what, aclTensor* d)
{
    const at::Tensor* t = tensor_of(o, what);
    if (t == nullptr) return nullptr;
    fill(d, *t, dtype == Py_None ? code_of(*t) : code_of(dtype));
    if (PyUnicode_Check(dtype) &&
        (PyUnicode_CompareWithASCIIString(dtype, "float4_e2m1") == 0 || PyUnicode_CompareWithASCIIString(dtype, "int4") == 0)) {
        const size_t r = d->rank();
        if (r == 0) return d;
        const size_t packed = r >= 2 && d->strides[r - 1] != 1 ? r - 2 : r - 1;  // a transposed view of packed storage: the second to last
        for (size_t i = 0; i < r; ++i)
            if (i != packed) d->strides[i] *= 2;
            else d->strides[i] = 1;
        d->shape[packed] *= 2;
        d->storage_shape = d->shape;
    }
    return d;
}

void need_cuda(c10::Device device)
{
    if (device.is_cuda()) return;
    PyErr_SetString(PyExc_RuntimeError, "this library has no CPU path: the tensors must be on a CUDA device");
    throw PyFail{};
}

// A workspace block of torch's allocator on the current stream of `device`, a CUDA device (need_cuda).
struct Workspace {
    c10::DataPtr block;
    void* ptr = nullptr;
    Workspace(uint64_t bytes, c10::Device device)
    {
        if (bytes == 0) return;
        const c10::cuda::OptionalCUDAGuard guard(device);
        block = c10::cuda::CUDACachingAllocator::get()->allocate(bytes);
        ptr = block.get();
    }
};

// Phase 1's plan until phase 2 consumes it.
struct Plan {
    aclOpExecutor* ex = nullptr;
    ~Plan()
    {
        if (ex != nullptr) aclDestroyAclOpExecutor(ex);
    }
    aclOpExecutor* take()
    {
        aclOpExecutor* e = ex;
        ex = nullptr;
        return e;
    }
};

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

PyObject* wrap(const at::Tensor& out)
{
    PyObject* o = THPVariable_Wrap(out);
    if (o == nullptr) throw PyFail{};
    return o;
}

// Drops a reference on every way out.
struct Ref {
    PyObject* o;
    ~Ref() { Py_XDECREF(o); }
};

bool arity(Py_ssize_t got, Py_ssize_t want, const char* name)
{
    if (got == want) return true;
    PyErr_Format(PyExc_TypeError, "%s takes %zd arguments, got %zd", name, want, got);
    return false;
}

// npu_quant_matmul(x1, x2, scale, offset, pertoken_scale, bias, output_dtype, group, x1_dtype, x2_dtype, scale_dtype, pertoken_dtype)
PyObject* npu_quant_matmul(PyObject*, PyObject* const* a, Py_ssize_t na)
{
    if (!arity(na, 12, "npu_quant_matmul")) return nullptr;
    return guarded([&]() -> PyObject* {
        aclTensor x1, x2, sc, of, pt, bi, y;
        const at::Tensor *t1 = tensor_of(a[0], "x1"), *t2 = tensor_of(a[1], "x2");
        if (t1 == nullptr || t2 == nullptr || t1->dim() < 2 || t2->dim() < 2) {
            PyErr_SetString(PyExc_ValueError, "npu_quant_matmul: x1 and x2 must be tensors of at least two dims");
            throw PyFail{};
        }
        describe(a[0], a[8], "x1", &x1);
        describe(a[1], a[9], "x2", &x2);
        const aclTensor* scp = describe(a[2], a[10], "scale", &sc);
        const aclTensor* ofp = describe(a[3], Py_None, "offset", &of);
        const aclTensor* ptp = describe(a[4], a[11], "pertoken_scale", &pt);
        const aclTensor* bip = describe(a[5], Py_None, "bias", &bi);
        if (!THPDtype_Check(a[6])) {
            PyErr_SetString(PyExc_TypeError, "npu_quant_matmul: output_dtype must be a torch dtype");
            throw PyFail{};
        }
        const at::Tensor& batched = t1->dim() > 2 ? *t1 : *t2;
        opsnn::Dims shape;
        shape.assign(batched.sizes().data(), batched.sizes().data() + (batched.dim() - 2));
        shape.push_back(x1.dim(-2));
        shape.push_back(x2.dim(-1));
        const at::ScalarType type = reinterpret_cast<THPDtype*>(a[6])->scalar_type;
        const c10::Device device = t1->device();
        need_cuda(device);
        const int out_code = code_of(type);
        const int64_t group = as_int(a[7]);
        at::Tensor out;
        const char* api = "aclnnQuantMatmulV5GetWorkspaceSize";
        aclnnStatus status;
        {
            const Unlocked unlocked;
            out = at::Tensor(at::detail::empty_cuda(c10::IntArrayRef(shape.begin(), shape.size()), type, device, std::nullopt));
            fill(&y, out, out_code);
            uint64_t ws = 0;
            Plan plan;
            status = aclnnQuantMatmulV5GetWorkspaceSize(&x1, &x2, ptp, scp, nullptr, nullptr, ofp, nullptr, bip, false, false, group, &y, &ws, &plan.ex);
            if (status == ACLNN_SUCCESS) {
                const Workspace w(ws, device);
                api = "aclnnQuantMatmulV5";
                status = aclnnQuantMatmulV5(w.ptr, ws, plan.take(), stream());
            }
        }
        check_call(api, status);
        return wrap(out);
    });
}

// npu_weight_quant_batchmatmul(x, weight, scale, offset, bias, group_size, inner_precise, weight_dtype)
PyObject* npu_weight_quant_batchmatmul(PyObject*, PyObject* const* a, Py_ssize_t na)
{
    if (!arity(na, 8, "npu_weight_quant_batchmatmul")) return nullptr;
    return guarded([&]() -> PyObject* {
        aclTensor x, w, sc, of, bi, y;
        const at::Tensor *tx = tensor_of(a[0], "x"), *tw = tensor_of(a[1], "weight");
        if (tx == nullptr || tw == nullptr || tx->dim() < 1 || tw->dim() < 1) {
            PyErr_SetString(PyExc_ValueError, "npu_weight_quant_batchmatmul: x and weight must be tensors");
            throw PyFail{};
        }
        fill(&x, *tx, code_of(*tx));
        fill(&w, *tw, a[7] == Py_None ? code_of(*tw) : code_of(a[7]));
        const aclTensor* scp = describe(a[2], Py_None, "antiquant_scale", &sc);
        const aclTensor* ofp = describe(a[3], Py_None, "antiquant_offset", &of);
        const aclTensor* bip = describe(a[4], Py_None, "bias", &bi);
        const int64_t shape[2] = {tx->size(0), tw->size(-1) * (tw->scalar_type() == at::kInt && tw->stride(-1) == 1 ? 8 : 1)};
        const c10::Device device = tx->device();
        need_cuda(device);
        const int out_code = code_of(*tx), group = (int)as_int(a[5]), inner_precise = (int)as_int(a[6]);
        at::Tensor out;
        const char* api = "aclnnWeightQuantBatchMatmulV3GetWorkspaceSize";
        aclnnStatus status;
        {
            const Unlocked unlocked;
            out = at::Tensor(at::detail::empty_cuda(c10::IntArrayRef(shape, 2), tx->scalar_type(), device, std::nullopt));
            fill(&y, out, out_code);
            uint64_t ws = 0;
            Plan plan;
            status = aclnnWeightQuantBatchMatmulV3GetWorkspaceSize(&x, &w, scp, ofp, nullptr, nullptr, bip, group, inner_precise, &y, &ws, &plan.ex);
            if (status == ACLNN_SUCCESS) {
                const Workspace space(ws, device);
                api = "aclnnWeightQuantBatchMatmulV3";
                status = aclnnWeightQuantBatchMatmulV3(space.ptr, ws, plan.take(), stream());
            }
        }
        check_call(api, status);
        return wrap(out);
    });
}

// ---- Tensor: an aclTensor descriptor ---------------------------------------------------------------------------------------------

struct TensorObject {
    PyObject_HEAD
    PyObject* shape;   // tuple
    PyObject* keep;    // what backs the view: a torch tensor, an address, or None
    PyObject* handle;  // the aclTensor's address, or None once it has been destroyed
    PyObject* dict;    // as a class written in Python has them: attributes, weak references, subclasses, cycles collected
    PyObject* weak;
    int dtype;
};
PyTypeObject* g_tensor_type = nullptr;

PyObject* new_tensor(PyTypeObject* type, const opsnn::Dims& shape, int code, void* data, PyObject* keep, const opsnn::Dims* strides, int64_t offset, int format,
                     const opsnn::Dims& storage)
{
    aclTensor* d = aclCreateTensor(shape.begin(), shape.size(), (aclDataType)code, strides ? strides->begin() : nullptr, offset, (aclFormat)format,
                                   storage.begin(), storage.size(), data);
    if (d == nullptr) {
        PyErr_SetString(PyExc_ValueError, "aclCreateTensor rejected the arguments");
        throw PyFail{};
    }
    TensorObject* t = reinterpret_cast<TensorObject*>(type->tp_alloc(type, 0));
    if (t == nullptr) {
        aclDestroyTensor(d);
        throw PyFail{};
    }
    t->handle = PyLong_FromVoidPtr(d);
    t->shape = PyTuple_New((Py_ssize_t)shape.size());
    for (size_t i = 0; i < shape.size(); ++i) PyTuple_SET_ITEM(t->shape, (Py_ssize_t)i, PyLong_FromLongLong(shape[i]));
    Py_INCREF(keep);
    t->keep = keep;
    t->dtype = code;
    return reinterpret_cast<PyObject*>(t);
}

PyObject* tensor_new(PyTypeObject* type, PyObject* args, PyObject* kw)
{
    static const char* names[] = {"shape", "dtype", "data", "strides", "offset", "fmt", "storage_shape", nullptr};
    PyObject *shape = nullptr, *dtype = nullptr, *data = nullptr, *strides = Py_None, *storage = Py_None;
    long long offset = 0;
    int format = ACL_FORMAT_ND;
    if (!PyArg_ParseTupleAndKeywords(args, kw, "OO|OOLiO:Tensor", const_cast<char**>(names), &shape, &dtype, &data, &strides, &offset, &format, &storage))
        return nullptr;
    return guarded([&]() -> PyObject* {
        const opsnn::Dims dims = as_dims(shape);
        opsnn::Dims st;
        if (strides != Py_None) st = as_strides(strides, dims);
        Ref zero{PyLong_FromLong(0)};
        if (data == nullptr) data = zero.o;
        void* ptr = nullptr;
        if (PyLong_Check(data)) {
            ptr = PyLong_AsVoidPtr(data);
            if (ptr == nullptr && PyErr_Occurred()) throw PyFail{};
        } else if (THPVariable_Check(data)) {
            ptr = THPVariable_Unpack(data).data_ptr();
        } else if (data != Py_None) {
            Ref r{PyObject_CallMethod(data, "data_ptr", nullptr)};
            if (r.o == nullptr) throw PyFail{};
            ptr = PyLong_AsVoidPtr(r.o);
            if (ptr == nullptr && PyErr_Occurred()) throw PyFail{};
        }
        return new_tensor(type, dims, code_of(dtype), ptr, data, strides == Py_None ? nullptr : &st, offset, format,
                          storage == Py_None ? dims : as_dims(storage));
    });
}

int tensor_traverse(PyObject* o, visitproc visit, void* arg)
{
    TensorObject* t = reinterpret_cast<TensorObject*>(o);
    Py_VISIT(Py_TYPE(o));
    Py_VISIT(t->shape);
    Py_VISIT(t->keep);
    Py_VISIT(t->dict);
    return 0;
}
int tensor_clear(PyObject* o)
{
    TensorObject* t = reinterpret_cast<TensorObject*>(o);
    Py_CLEAR(t->keep);
    Py_CLEAR(t->dict);
    return 0;
}
void tensor_dealloc(PyObject* o)
{
    PyObject_GC_UnTrack(o);
    TensorObject* t = reinterpret_cast<TensorObject*>(o);
    if (t->weak != nullptr) PyObject_ClearWeakRefs(o);
    if (t->handle != nullptr && PyLong_Check(t->handle)) {
        if (void* p = PyLong_AsVoidPtr(t->handle)) aclDestroyTensor(static_cast<aclTensor*>(p));
    }
    Py_XDECREF(t->handle);
    Py_XDECREF(t->shape);
    tensor_clear(o);
    PyTypeObject* type = Py_TYPE(o);
    type->tp_free(o);
    Py_DECREF(type);
}

PyMemberDef tensor_members[] = {
    {"shape", T_OBJECT, offsetof(TensorObject, shape), 0, "view extents"},
    {"dtype", T_INT, offsetof(TensorObject, dtype), 0, "aclDataType"},
    {"handle", T_OBJECT, offsetof(TensorObject, handle), 0, "address of the aclTensor, None when destroyed"},
    {"_keep", T_OBJECT, offsetof(TensorObject, keep), 0, "what backs the view"},
    {"__dictoffset__", T_PYSSIZET, offsetof(TensorObject, dict), READONLY, nullptr},
    {"__weaklistoffset__", T_PYSSIZET, offsetof(TensorObject, weak), READONLY, nullptr},
    {nullptr, 0, 0, 0, nullptr},
};
PyGetSetDef tensor_getset[] = {{"__dict__", PyObject_GenericGetDict, PyObject_GenericSetDict, nullptr, nullptr}, {nullptr, nullptr, nullptr, nullptr, nullptr}};
PyType_Slot tensor_slots[] = {
    {Py_tp_new, reinterpret_cast<void*>(tensor_new)},
    {Py_tp_dealloc, reinterpret_cast<void*>(tensor_dealloc)},
    {Py_tp_traverse, reinterpret_cast<void*>(tensor_traverse)},
    {Py_tp_clear, reinterpret_cast<void*>(tensor_clear)},
    {Py_tp_getset, tensor_getset},
    {Py_tp_members, tensor_members},
    {Py_tp_doc, const_cast<char*>("An aclTensor descriptor. `data` is a device address (int) or a torch tensor whose storage backs the view.")},
    {0, nullptr},
};
PyType_Spec tensor_spec = {"ops_nn_b200.aclnn.Tensor", sizeof(TensorObject), 0, Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE | Py_TPFLAGS_HAVE_GC, tensor_slots};

const TensorObject* desc_of(PyObject* o, const char* what)  // nullptr for None
{
    if (o == Py_None) return nullptr;
    if (!PyObject_TypeCheck(o, g_tensor_type)) {
        PyErr_Format(PyExc_TypeError, "%s must be an aclnn.Tensor, got %s", what, Py_TYPE(o)->tp_name);
        throw PyFail{};
    }
    return reinterpret_cast<const TensorObject*>(o);
}

aclTensor* handle_of(PyObject* o, const char* what)
{
    const TensorObject* t = desc_of(o, what);
    if (t == nullptr || t->handle == nullptr || !PyLong_Check(t->handle)) return nullptr;
    return static_cast<aclTensor*>(PyLong_AsVoidPtr(t->handle));
}

// from_torch(t, dtype=None, shape=None, strides=None)
PyObject* from_torch(PyObject*, PyObject* args, PyObject* kw)
{
    static const char* names[] = {"t", "dtype", "shape", "strides", nullptr};
    PyObject *t = nullptr, *dtype = Py_None, *shape = Py_None, *strides = Py_None;
    if (!PyArg_ParseTupleAndKeywords(args, kw, "O|OOO:from_torch", const_cast<char**>(names), &t, &dtype, &shape, &strides)) return nullptr;
    if (t == Py_None) Py_RETURN_NONE;
    return guarded([&]() -> PyObject* {
        const at::Tensor& v = *tensor_of(t, "t");
        aclTensor d;
        fill(&d, v, dtype == Py_None ? code_of(v) : code_of(dtype));
        if (shape == Py_None) return new_tensor(g_tensor_type, d.shape, d.dtype, d.data, t, &d.strides, 0, ACL_FORMAT_ND, d.shape);
        const opsnn::Dims dims = as_dims(shape);
        opsnn::Dims st;
        if (strides != Py_None) st = as_strides(strides, dims);
        return new_tensor(g_tensor_type, dims, d.dtype, d.data, t, strides == Py_None ? nullptr : &st, 0, ACL_FORMAT_ND, dims);
    });
}

// Both phases of a call on descriptors: its workspace is the caller's tensor where that is large enough, else a block of the allocator on
// the device of the output's storage. Returns the workspace size that the plan asked for.
template <typename Phase1, typename Phase2>
PyObject* run_on_descriptors(const char* api1, const char* api2, PyObject* given, const TensorObject* out, Phase1&& phase1, Phase2&& phase2)
{
    const at::Tensor* t = tensor_of(given, "workspace");
    void* const given_ptr = t != nullptr ? t->data_ptr() : nullptr;
    const uint64_t given_bytes = t != nullptr ? (uint64_t)t->numel() : 0;
    const bool backed = out != nullptr && out->keep != nullptr && THPVariable_Check(out->keep);
    const c10::Device device = backed ? THPVariable_Unpack(out->keep).device() : c10::Device(c10::kCPU);
    uint64_t ws = 0;
    const char* api = api1;
    aclnnStatus status;
    bool no_workspace = false;
    {
        const Unlocked unlocked;
        Plan plan;
        status = phase1(&ws, &plan.ex);
        if (status == ACLNN_SUCCESS) {
            const bool own = t == nullptr || given_bytes < ws;
            no_workspace = own && ws != 0 && !device.is_cuda();
            if (!no_workspace) {
                const Workspace w(own ? ws : 0, device);
                api = api2;
                status = phase2(own ? w.ptr : given_ptr, own ? ws : given_bytes, plan.take(), stream());
            }
        }
    }
    if (no_workspace) {
        if (backed) need_cuda(device);
        PyErr_SetString(PyExc_AttributeError, "a workspace is needed and the output descriptor is not backed by a torch tensor");
        throw PyFail{};
    }
    check_call(api, status);
    return PyLong_FromUnsignedLongLong(ws);
}

// quant_matmul_v5(x1, x2, x1_scale, x2_scale, out, bias, transpose_x1, transpose_x2, group_size, x2_offset, workspace, y_scale, weight_nz)
PyObject* quant_matmul_v5(PyObject*, PyObject* const* a, Py_ssize_t na)
{
    if (!arity(na, 13, "quant_matmul_v5")) return nullptr;
    return guarded([&]() -> PyObject* {
        const bool nz = PyObject_IsTrue(a[12]) != 0, tr1 = PyObject_IsTrue(a[6]) != 0, tr2 = PyObject_IsTrue(a[7]) != 0;
        const aclTensor *x1 = handle_of(a[0], "x1"), *x2 = handle_of(a[1], "x2"), *s1 = handle_of(a[2], "x1_scale"), *s2 = handle_of(a[3], "x2_scale");
        const aclTensor *ys = handle_of(a[11], "y_scale"), *of = handle_of(a[9], "x2_offset"), *bi = handle_of(a[5], "bias");
        aclTensor* const out = handle_of(a[4], "out");
        const int64_t group = as_int(a[8]);
        const auto phase1 = nz ? aclnnQuantMatmulWeightNzGetWorkspaceSize : aclnnQuantMatmulV5GetWorkspaceSize;
        const auto phase2 = nz ? aclnnQuantMatmulWeightNz : aclnnQuantMatmulV5;
        return run_on_descriptors(
            nz ? "aclnnQuantMatmulWeightNzGetWorkspaceSize" : "aclnnQuantMatmulV5GetWorkspaceSize", nz ? "aclnnQuantMatmulWeightNz" : "aclnnQuantMatmulV5",
            a[10], desc_of(a[4], "out"),
            [&](uint64_t* ws, aclOpExecutor** ex) { return phase1(x1, x2, s1, s2, ys, nullptr, of, nullptr, bi, tr1, tr2, group, out, ws, ex); }, phase2);
    });
}

// weight_quant_batch_matmul(x, weight, scale, y, offset, bias, group_size, inner_precise, workspace): inner_precise None = V2, "nz" = Nz
PyObject* weight_quant_batch_matmul(PyObject*, PyObject* const* a, Py_ssize_t na)
{
    if (!arity(na, 9, "weight_quant_batch_matmul")) return nullptr;
    return guarded([&]() -> PyObject* {
        const aclTensor *x = handle_of(a[0], "x"), *w = handle_of(a[1], "weight"), *sc = handle_of(a[2], "antiquant_scale"), *y = handle_of(a[3], "y");
        const aclTensor *of = handle_of(a[4], "antiquant_offset"), *bi = handle_of(a[5], "bias");
        const TensorObject* out = desc_of(a[3], "y");
        const int group = (int)as_int(a[6]);
        if (a[7] == Py_None)
            return run_on_descriptors(
                "aclnnWeightQuantBatchMatmulV2GetWorkspaceSize", "aclnnWeightQuantBatchMatmulV2", a[8], out,
                [&](uint64_t* ws, aclOpExecutor** ex) {
                    return aclnnWeightQuantBatchMatmulV2GetWorkspaceSize(x, w, sc, of, nullptr, nullptr, bi, group, y, ws, ex);
                },
                aclnnWeightQuantBatchMatmulV2);
        if (PyUnicode_Check(a[7]) && PyUnicode_CompareWithASCIIString(a[7], "nz") == 0)
            return run_on_descriptors(
                "aclnnWeightQuantBatchMatmulNzGetWorkspaceSize", "aclnnWeightQuantBatchMatmulNz", a[8], out,
                [&](uint64_t* ws, aclOpExecutor** ex) {
                    return aclnnWeightQuantBatchMatmulNzGetWorkspaceSize(x, w, sc, of, nullptr, nullptr, bi, group, y, ws, ex);
                },
                aclnnWeightQuantBatchMatmulNz);
        const int inner_precise = (int)as_int(a[7]);
        return run_on_descriptors(
            "aclnnWeightQuantBatchMatmulV3GetWorkspaceSize", "aclnnWeightQuantBatchMatmulV3", a[8], out,
            [&](uint64_t* ws, aclOpExecutor** ex) {
                return aclnnWeightQuantBatchMatmulV3GetWorkspaceSize(x, w, sc, of, nullptr, nullptr, bi, group, inner_precise, y, ws, ex);
            },
            aclnnWeightQuantBatchMatmulV3);
    });
}

// dynamic_mx_quant(x, y_out, mxscale_out, dst_type, axis, round_mode, blocksize, scale_alg)
PyObject* dynamic_mx_quant(PyObject*, PyObject* const* a, Py_ssize_t na)
{
    if (!arity(na, 8, "dynamic_mx_quant")) return nullptr;
    return guarded([&]() -> PyObject* {
        char* mode = nullptr;
        if (a[5] != Py_None) {
            mode = PyBytes_AsString(a[5]);
            if (mode == nullptr) throw PyFail{};
        }
        const aclTensor *x = handle_of(a[0], "x"), *y = handle_of(a[1], "y_out"), *sc = handle_of(a[2], "mxscale_out");
        const int64_t axis = as_int(a[4]), block = as_int(a[6]), alg = as_int(a[7]);
        const int dst = code_of(a[3]);
        const char* api = "aclnnDynamicMxQuantGetWorkspaceSize";
        aclnnStatus status;
        {
            const Unlocked unlocked;
            uint64_t ws = 0;
            Plan plan;
            status = aclnnDynamicMxQuantGetWorkspaceSize(x, axis, mode, dst, block, alg, y, sc, &ws, &plan.ex);
            if (status == ACLNN_SUCCESS) {
                api = "aclnnDynamicMxQuant";
                status = aclnnDynamicMxQuant(nullptr, 0, plan.take(), stream());
            }
        }
        check_call(api, status);
        Py_RETURN_NONE;
    });
}

// init(dtype_codes, call_error): the package's dtype table and its exception
PyObject* init(PyObject*, PyObject* const* a, Py_ssize_t na)
{
    if (!arity(na, 2, "init")) return nullptr;
    Py_INCREF(a[0]);
    Py_INCREF(a[1]);
    Py_XDECREF(g_codes);
    Py_XDECREF(g_call_error);
    g_codes = a[0];
    g_call_error = a[1];
    Py_RETURN_NONE;
}

PyCFunction fast(PyObject* (*f)(PyObject*, PyObject* const*, Py_ssize_t)) { return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)); }

PyMethodDef methods[] = {
    {"init", fast(&init), METH_FASTCALL, nullptr},
    {"npu_quant_matmul", fast(&npu_quant_matmul), METH_FASTCALL, nullptr},
    {"npu_weight_quant_batchmatmul", fast(&npu_weight_quant_batchmatmul), METH_FASTCALL, nullptr},
    {"from_torch", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&from_torch)), METH_VARARGS | METH_KEYWORDS, nullptr},
    {"quant_matmul_v5", fast(&quant_matmul_v5), METH_FASTCALL, nullptr},
    {"weight_quant_batch_matmul", fast(&weight_quant_batch_matmul), METH_FASTCALL, nullptr},
    {"dynamic_mx_quant", fast(&dynamic_mx_quant), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_opsnn_native", "Native calls of ops_nn_b200", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__opsnn_native(void)
{
    PyObject* m = PyModule_Create(&module_def);
    if (m == nullptr) return nullptr;
    g_tensor_type = reinterpret_cast<PyTypeObject*>(PyType_FromSpec(&tensor_spec));
    if (g_tensor_type == nullptr || PyModule_AddObjectRef(m, "Tensor", reinterpret_cast<PyObject*>(g_tensor_type)) != 0) {
        Py_DECREF(m);
        return nullptr;
    }
    return m;
}
