// CPython side of the Python mirror's calls: argument checks, output and workspace allocation and the launch, in one call
// into native code.  A decode forward runs a few microseconds on the GPU; through ctypes its host side took 17 us (dtype
// queries, a device context manager, torch.empty, a dictionary of workspaces, a dozen ctypes conversions), and a half-
// precision forward 35 us with its two conversion kernels.
//
// `Storage` is the native half of QCudaStorage.  Its methods return a tensor, or None when the arguments do not fit -- the
// Python side then runs its own checks to say why -- and raise through the registered error function when the library
// reports a status.
//
// Launch overlap, unless lloom_b200_set_launch_overlap has settled the matter for all calls: a storage's first forward waits for everything before it on its stream like any kernel.  From then on
// the blocks are known to be in place (nothing writes them after the upload), and later forwards may stream them while the
// stream's previous kernel is still finishing.  A storage whose device pointer has been handed out, or that was made over a
// caller's tensor, stays with the first kind: the holder may write through it.
#include <torch/csrc/autograd/python_variable.h>
#include <torch/extension.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <map>
#include <mutex>
#include <utility>
#include <vector>

#include "../forward.h"

namespace {

using lloom::FwdIo;

PyObject *g_error = nullptr;  // callable(status, where): raises

PyObject *fail(int status, const char *where) {
    PyObject *r = PyObject_CallFunction(g_error, "is", status, where);
    if (r) {  // it should have raised
        Py_DECREF(r);
        PyErr_Format(PyExc_RuntimeError, "%s: status %d", where, status);
    }
    return nullptr;
}

// Grow-only scratch per (device, stream): launches on different streams never share a buffer.  A buffer that has been
// outgrown stays alive: a CUDA graph captured earlier may hold its address.
struct Workspaces {
    std::mutex mu;
    std::map<std::pair<int, cudaStream_t>, at::Tensor> bufs;
    std::vector<at::Tensor> retired;

    const at::Tensor &get(c10::Device dev, cudaStream_t stream, int64_t bytes) {
        std::lock_guard<std::mutex> lock(mu);
        at::Tensor &buf = bufs[{dev.index(), stream}];
        if (!buf.defined() || buf.numel() < bytes) {
            if (buf.defined()) retired.push_back(buf);
            buf = at::detail::empty_cuda({std::max<int64_t>(bytes, 1 << 20)}, at::kByte, dev, std::nullopt);
        }
        return buf;
    }
};
Workspaces &workspaces() {
    static Workspaces *w = new Workspaces;  // never destroyed: the CUDA context may be gone by then
    return *w;
}

struct Storage {
    PyObject_HEAD
    at::Tensor *data;   // packed blocks
    at::Tensor *image;  // prefill image, or null
    int64_t image_off;
    int64_t bytes;      // of the blocks, without the padding
    int dtype;
    bool settled, exposed;
};

PyTypeObject StorageType = {PyVarObject_HEAD_INIT(nullptr, 0)};  // filled in by the module's init

bool elem_type(at::ScalarType t, int &out) {
    switch (t) {
    case at::kFloat: out = LLOOM_F32; return true;
    case at::kHalf: out = LLOOM_F16; return true;
    case at::kBFloat16: out = LLOOM_BF16; return true;
    default: return false;
    }
}

int Storage_init(PyObject *o, PyObject *args, PyObject *) {
    Storage *self = reinterpret_cast<Storage *>(o);
    PyObject *t;
    int dtype;
    long long bytes;
    if (!PyArg_ParseTuple(args, "OiL", &t, &dtype, &bytes)) return -1;
    if (!THPVariable_Check(t)) {
        PyErr_SetString(PyExc_TypeError, "a tensor of packed blocks is wanted");
        return -1;
    }
    delete self->data;
    self->data = new at::Tensor(THPVariable_Unpack(t));
    self->dtype = dtype;
    self->bytes = bytes;
    self->settled = self->exposed = false;
    return 0;
}

void Storage_dealloc(PyObject *o) {
    Storage *self = reinterpret_cast<Storage *>(o);
    delete self->data;
    delete self->image;
    Py_TYPE(o)->tp_free(o);
}

PyObject *Storage_set_image(PyObject *o, PyObject *args) {
    Storage *self = reinterpret_cast<Storage *>(o);
    PyObject *t;
    long long off = 0;
    if (!PyArg_ParseTuple(args, "O|L", &t, &off)) return nullptr;
    delete self->image;
    self->image = nullptr;
    if (t != Py_None) {
        if (!THPVariable_Check(t)) {
            PyErr_SetString(PyExc_TypeError, "a tensor or None is wanted");
            return nullptr;
        }
        self->image = new at::Tensor(THPVariable_Unpack(t));
        self->image_off = off;
    }
    Py_RETURN_NONE;
}

PyObject *Storage_expose(PyObject *o, PyObject *) {
    reinterpret_cast<Storage *>(o)->exposed = true;
    Py_RETURN_NONE;
}

// Whether this storage's next forward may start before its stream predecessor has finished
bool overlaps(const Storage *self) {
    const int mode = lloom::launch_overlap();
    return mode > 0 || (mode < 0 && self->settled && !self->exposed);
}

PyObject *Storage_exposed(PyObject *o, PyObject *) { return PyBool_FromLong(reinterpret_cast<Storage *>(o)->exposed); }
PyObject *Storage_overlaps(PyObject *o, PyObject *) { return PyBool_FromLong(overlaps(reinterpret_cast<Storage *>(o))); }

bool shape2(PyObject *t, int64_t &n, int64_t &k) {
    if (!PyTuple_Check(t) || PyTuple_GET_SIZE(t) != 2) return false;
    n = PyLong_AsLongLong(PyTuple_GET_ITEM(t, 0));
    k = PyLong_AsLongLong(PyTuple_GET_ITEM(t, 1));
    return !PyErr_Occurred() && n > 0 && k > 0;
}

// An activation tensor of this storage's device, [.., k], contiguous, of a type the kernels read
bool acts_ok(const Storage *self, const at::Tensor &x, int64_t k, int &x_type) {
    return x.defined() && x.device() == self->data->device() && x.layout() == at::kStrided && elem_type(x.scalar_type(), x_type) &&
           x.dim() >= 2 && x.size(-1) == k && x.numel() > 0 && x.is_contiguous();
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

PyObject *none_or_error() {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
}

// forward(x, (n, k)[, out, column, store]) -> [.., n] of x's type, or f32 into columns of `out` [m, ld]
PyObject *Storage_forward(PyObject *o, PyObject *const *args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    Storage *self = reinterpret_cast<Storage *>(o);
    int64_t n, k;
    int store = LLOOM_STORE_PLAIN, x_type;
    if (nargs < 2 || !THPVariable_Check(args[0]) || !shape2(args[1], n, k)) return none_or_error();
    at::Tensor x = THPVariable_Unpack(args[0]);
    if (!acts_ok(self, x, k, x_type)) Py_RETURN_NONE;
    int64_t column = 0;
    at::Tensor y;
    if (nargs == 5) {
        column = PyLong_AsLongLong(args[3]);
        store = (int)PyLong_AsLong(args[4]);
        if (PyErr_Occurred()) return nullptr;
        if (args[2] != Py_None) {
            if (!THPVariable_Check(args[2])) Py_RETURN_NONE;
            y = THPVariable_Unpack(args[2]);
        }
    }
    const c10::Device dev = self->data->device();
    c10::cuda::CUDAGuard guard(dev);
    const int64_t m = x.numel() / k;
    FwdIo io;
    io.overlap = overlaps(self);
    if (x_type != LLOOM_F32 && !aligned16(x.const_data_ptr())) x = x.clone();
    io.x_type = x_type;
    int64_t ldy = n;
    char *yp;
    const bool fresh = !y.defined();
    if (!fresh) {
        ldy = y.dim() >= 2 ? y.stride(-2) : y.numel();
        yp = static_cast<char *>(y.data_ptr()) + 4 * column;
    } else {
        c10::SmallVector<int64_t, 5> sizes(x.sizes().begin(), x.sizes().end());
        sizes.back() = n;
        const bool plain = store == LLOOM_STORE_PLAIN;
        y = at::detail::empty_cuda(sizes, plain ? x.scalar_type() : at::kFloat, dev, std::nullopt);
        io.y_type = plain ? x_type : LLOOM_F32;
        yp = static_cast<char *>(y.data_ptr());
    }
    const bool image = self->image && m > 8 && store == LLOOM_STORE_PLAIN;
    const int64_t need = image ? lloom_b200_workspace_bytes_with_image(self->dtype, m, n, k)
                               : lloom_b200_workspace_bytes(self->dtype, m, n, k);
    if (need <= 0) Py_RETURN_NONE;
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    const at::Tensor &ws = workspaces().get(dev, stream, need);
    const int rc = lloom::qmatmul_forward(self->dtype, self->data->const_data_ptr(),
                                          image ? static_cast<char *>(self->image->data_ptr()) + self->image_off : nullptr,
                                          x.const_data_ptr(), yp, m, n, k, ldy, store, ws.data_ptr(), ws.numel(), stream, io);
    if (rc != LLOOM_OK) return fail(rc, "qmatmul_fwd");
    self->settled = true;
    if (fresh && y.scalar_type() != x.scalar_type()) y = y.to(x.scalar_type());  // a store block's outputs are f32
    return THPVariable_Wrap(y);
    END_HANDLE_TH_ERRORS
}

// embedding(ids, (rows, hidden)) -> f32 ids.shape + [hidden]
PyObject *Storage_embedding(PyObject *o, PyObject *const *args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    Storage *self = reinterpret_cast<Storage *>(o);
    int64_t rows, hidden;
    if (nargs != 2 || !THPVariable_Check(args[0]) || !shape2(args[1], rows, hidden)) return none_or_error();
    const int64_t be = lloom_b200_block_elems(self->dtype), bb = lloom_b200_block_bytes(self->dtype);
    if (hidden % be != 0 || self->bytes != rows * (hidden / be) * bb) Py_RETURN_NONE;
    const c10::Device dev = self->data->device();
    c10::cuda::CUDAGuard guard(dev);
    at::Tensor ids = THPVariable_Unpack(args[0]);
    c10::SmallVector<int64_t, 5> sizes(ids.sizes().begin(), ids.sizes().end());
    sizes.push_back(hidden);
    if (ids.device() != dev || (ids.scalar_type() != at::kLong && ids.scalar_type() != at::kInt)) ids = ids.to(dev, at::kLong);
    ids = ids.contiguous();
    at::Tensor out = at::detail::empty_cuda(sizes, at::kFloat, dev, std::nullopt);
    if (ids.numel() > 0) {
        const int rc = lloom::get_rows(self->dtype, self->data->const_data_ptr(), rows, hidden, ids.const_data_ptr(),
                                       ids.scalar_type() == at::kLong, ids.numel(), out.data_ptr<float>(),
                                       c10::cuda::getCurrentCUDAStream(dev.index()).stream(), lloom::launch_overlap() != 0);
        if (rc != LLOOM_OK) return fail(rc, "get_rows");
    }
    return THPVariable_Wrap(out);
    END_HANDLE_TH_ERRORS
}

// experts(x, ids, n_experts, n, k) -> f32 [batch, topk, n]
PyObject *Storage_experts(PyObject *o, PyObject *const *args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    Storage *self = reinterpret_cast<Storage *>(o);
    if (nargs != 5 || !THPVariable_Check(args[0]) || !THPVariable_Check(args[1])) Py_RETURN_NONE;
    const int64_t n_experts = PyLong_AsLongLong(args[2]), n = PyLong_AsLongLong(args[3]), k = PyLong_AsLongLong(args[4]);
    if (PyErr_Occurred()) return nullptr;
    at::Tensor x = THPVariable_Unpack(args[0]), ids = THPVariable_Unpack(args[1]);
    const c10::Device dev = self->data->device();
    if (x.dim() != 3 || ids.dim() != 2 || x.device() != dev || ids.device() != dev || x.size(2) != k || x.size(0) != ids.size(0) ||
        (x.size(1) != 1 && x.size(1) != ids.size(1)) || x.numel() == 0 || ids.numel() == 0)
        Py_RETURN_NONE;
    c10::cuda::CUDAGuard guard(dev);
    if (x.scalar_type() != at::kFloat) x = x.to(at::kFloat);
    x = x.contiguous();
    if (ids.scalar_type() != at::kLong && ids.scalar_type() != at::kInt) ids = ids.to(at::kLong);
    ids = ids.contiguous();
    at::Tensor out = at::detail::empty_cuda({x.size(0), ids.size(1), n}, at::kFloat, dev, std::nullopt);
    const int64_t need = lloom_b200_workspace_bytes(self->dtype, 1, n, k);
    if (need <= 0) Py_RETURN_NONE;
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    const at::Tensor &ws = workspaces().get(dev, stream, need);
    FwdIo io;
    io.overlap = overlaps(self);
    const int rc = lloom::indexed_moe_forward(self->dtype, self->data->const_data_ptr(), n_experts, n, k, x.const_data_ptr<float>(),
                                              x.size(0), x.size(1), ids.const_data_ptr(), ids.scalar_type() == at::kLong, ids.size(1),
                                              out.data_ptr<float>(), ws.data_ptr(), ws.numel(), stream, io);
    if (rc != LLOOM_OK) return fail(rc, "indexed_moe_forward");
    self->settled = true;
    return THPVariable_Wrap(out);
    END_HANDLE_TH_ERRORS
}


// group(storages, (n, ..), k, x, stores or None, outs or None) -> list of f32 [.., n_g]
PyObject *module_group(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    if (nargs != 6 || !PyList_Check(args[0]) || !PyList_Check(args[1]) || !THPVariable_Check(args[3])) Py_RETURN_NONE;
    const Py_ssize_t G = PyList_GET_SIZE(args[0]);
    if (G < 1 || G > LLOOM_B200_MAX_GROUP || PyList_GET_SIZE(args[1]) != G) Py_RETURN_NONE;
    const int64_t k = PyLong_AsLongLong(args[2]);
    if (PyErr_Occurred()) return nullptr;
    const at::Tensor &x = THPVariable_Unpack(args[3]);
    PyObject *stores = args[4] == Py_None ? nullptr : args[4], *outs = args[5] == Py_None ? nullptr : args[5];
    if ((stores && (!PyList_Check(stores) || PyList_GET_SIZE(stores) != G)) || (outs && (!PyList_Check(outs) || PyList_GET_SIZE(outs) != G)))
        Py_RETURN_NONE;
    Storage *st[LLOOM_B200_MAX_GROUP];
    const void *w[LLOOM_B200_MAX_GROUP];
    float *y[LLOOM_B200_MAX_GROUP];
    int64_t n[LLOOM_B200_MAX_GROUP], ld[LLOOM_B200_MAX_GROUP], n_max = 0;
    int store[LLOOM_B200_MAX_GROUP];
    FwdIo io;
    io.overlap = true;
    for (Py_ssize_t g = 0; g < G; ++g) {
        PyObject *s = PyList_GET_ITEM(args[0], g);
        if (Py_TYPE(s) != &StorageType) Py_RETURN_NONE;
        st[g] = reinterpret_cast<Storage *>(s);
        if (st[g]->dtype != st[0]->dtype || st[g]->data->device() != st[0]->data->device()) Py_RETURN_NONE;
        w[g] = st[g]->data->const_data_ptr();
        n[g] = PyLong_AsLongLong(PyList_GET_ITEM(args[1], g));
        store[g] = stores ? (int)PyLong_AsLong(PyList_GET_ITEM(stores, g)) : LLOOM_STORE_PLAIN;
        if (PyErr_Occurred()) return nullptr;
        n_max = std::max(n_max, n[g]);
        io.overlap = io.overlap && overlaps(st[g]);
    }
    int x_type;
    if (!acts_ok(st[0], x, k, x_type) || x_type != LLOOM_F32) Py_RETURN_NONE;
    const c10::Device dev = st[0]->data->device();
    c10::cuda::CUDAGuard guard(dev);
    const int64_t m = x.numel() / k;
    const int64_t need = lloom_b200_workspace_bytes(st[0]->dtype, m, n_max, k);
    if (need <= 0) Py_RETURN_NONE;
    THPObjectPtr list(PyList_New(G));
    if (!list) return nullptr;
    for (Py_ssize_t g = 0; g < G; ++g) {
        PyObject *item;
        if (outs) {
            item = PyList_GET_ITEM(outs, g);
            if (!THPVariable_Check(item)) Py_RETURN_NONE;
            Py_INCREF(item);
            const at::Tensor &t = THPVariable_Unpack(item);
            y[g] = static_cast<float *>(t.data_ptr());
            ld[g] = t.dim() >= 2 ? t.stride(-2) : t.numel();
        } else {
            c10::SmallVector<int64_t, 5> sizes(x.sizes().begin(), x.sizes().end());
            sizes.back() = n[g];
            at::Tensor t = at::detail::empty_cuda(sizes, at::kFloat, dev, std::nullopt);
            y[g] = static_cast<float *>(t.data_ptr());
            ld[g] = n[g];
            item = THPVariable_Wrap(std::move(t));
            if (!item) return nullptr;
        }
        PyList_SET_ITEM(list.get(), g, item);
    }
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    const at::Tensor &ws = workspaces().get(dev, stream, need);
    const int rc = lloom::qmatmul_forward_group(st[0]->dtype, (int)G, w, x.const_data_ptr(), y, n, ld, store, m, k, ws.data_ptr(),
                                                ws.numel(), stream, io);
    if (rc != LLOOM_OK) return fail(rc, "qmatmul_fwd_group");
    for (Py_ssize_t g = 0; g < G; ++g) st[g]->settled = true;
    return list.release();
    END_HANDLE_TH_ERRORS
}

// workspace(device index, stream, bytes) -> uint8 tensor of at least that size, kept for later calls
PyObject *module_workspace(PyObject *, PyObject *args) {
    HANDLE_TH_ERRORS
    int index;
    unsigned long long stream;
    long long bytes;
    if (!PyArg_ParseTuple(args, "iKL", &index, &stream, &bytes)) return nullptr;
    const c10::Device dev(c10::kCUDA, (c10::DeviceIndex)index);
    c10::cuda::CUDAGuard guard(dev);
    return THPVariable_Wrap(workspaces().get(dev, reinterpret_cast<cudaStream_t>(stream), bytes));
    END_HANDLE_TH_ERRORS
}

PyObject *module_set_error(PyObject *, PyObject *fn) {
    Py_INCREF(fn);
    Py_XDECREF(g_error);
    g_error = fn;
    Py_RETURN_NONE;
}

#define FAST(fn) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(fn))
PyMethodDef storage_methods[] = {{"forward", FAST(Storage_forward), METH_FASTCALL, nullptr},
                                 {"embedding", FAST(Storage_embedding), METH_FASTCALL, nullptr},
                                 {"experts", FAST(Storage_experts), METH_FASTCALL, nullptr},
                                 {"set_image", Storage_set_image, METH_VARARGS, nullptr},
                                 {"expose", Storage_expose, METH_NOARGS, nullptr},
                                 {"exposed", Storage_exposed, METH_NOARGS, nullptr},
                                 {"overlaps", Storage_overlaps, METH_NOARGS, nullptr},
                                 {nullptr, nullptr, 0, nullptr}};

PyMethodDef module_methods[] = {{"group", FAST(module_group), METH_FASTCALL, nullptr},
                                {"workspace", module_workspace, METH_VARARGS, nullptr},
                                {"set_error", module_set_error, METH_O, nullptr},
                                {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, module_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
    StorageType.tp_name = "lloom_b200._native.Storage";
    StorageType.tp_basicsize = sizeof(Storage);
    StorageType.tp_flags = Py_TPFLAGS_DEFAULT;
    StorageType.tp_new = PyType_GenericNew;
    StorageType.tp_init = Storage_init;
    StorageType.tp_dealloc = Storage_dealloc;
    StorageType.tp_methods = storage_methods;
    if (PyType_Ready(&StorageType) < 0) return nullptr;
    PyObject *m = PyModule_Create(&module_def);
    if (!m) return nullptr;
    Py_INCREF(&StorageType);
    if (PyModule_AddObject(m, "Storage", reinterpret_cast<PyObject *>(&StorageType)) < 0) return nullptr;
    return m;
}
