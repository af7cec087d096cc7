// The way from a DeviceSession method to the C ABI: reads the tensors of a call
// (kind, layout, dtype, address, element count) and calls the library, all in native
// code.  The same through ctypes and tensor methods costs about 9 us per
// collective and 0.28 us per tensor of a group (788 us for 8 ranks x 199
// tensors, more than half of the GPU's time on them); here it is below 1 us
// and about 10 ns per tensor.  The library call runs without the GIL, as under ctypes.
//
// Every function returns the C ABI's code (0: done); what is wrong with the
// arguments raises ValueError / TypeError.
#include <Python.h>

#include <torch/csrc/autograd/python_variable.h>

#include <vector>

#include "capi_cuda.h"

namespace
{
// `group`: tensors of several dtypes, which the caller splits
constexpr long kMixedDtypes = -1000;

int dtype_code(c10::ScalarType t)
{
    switch (t) {
    case c10::ScalarType::Char:
        return 0;
    case c10::ScalarType::Short:
        return 1;
    case c10::ScalarType::Int:
        return 2;
    case c10::ScalarType::Long:
        return 3;
    case c10::ScalarType::Byte:
        return 4;
    case c10::ScalarType::UInt16:
        return 5;
    case c10::ScalarType::UInt32:
        return 6;
    case c10::ScalarType::UInt64:
        return 7;
    case c10::ScalarType::BFloat16:
        return 8;
    case c10::ScalarType::Half:
        return 9;
    case c10::ScalarType::Float:
        return 10;
    case c10::ScalarType::Double:
        return 11;
    default:
        return -1;
    }
}

struct Raised {
};  // a Python exception is set

int supported_dtype(const at::Tensor &t)
{
    const int code = dtype_code(t.scalar_type());
    if (code < 0) {
        PyErr_Format(PyExc_TypeError, "unsupported dtype %s", c10::toString(t.scalar_type()));
        throw Raised{};
    }
    return code;
}

const at::Tensor &tensor_of(PyObject *o, const char *call)
{
    if (!THPVariable_Check(o)) {
        PyErr_Format(PyExc_TypeError, "%s: tensor expected, got %s", call, Py_TYPE(o)->tp_name);
        throw Raised{};
    }
    return THPVariable_Unpack(o);
}

void *checked_ptr(const at::Tensor &t, const char *call)
{
    if (!t.is_cuda()) {
        PyErr_Format(PyExc_ValueError, "%s: CUDA tensor expected", call);
        throw Raised{};
    }
    if (!t.is_contiguous()) {
        PyErr_Format(PyExc_ValueError, "%s: contiguous tensor expected", call);
        throw Raised{};
    }
    return t.data_ptr();
}

// What a collective needs of its per-rank tensors: one tensor, or in a loopback
// session a list with one per rank (None: this rank has none).
struct PerRank {
    static constexpr int kMost = 16;
    void *ptr[kMost];
    unsigned long long count = 0;  // of rank 0's tensor
    int dt = -1;

    PerRank(PyObject *x, int vranks, const char *what, const char *call)
    {
        if (vranks <= 1) {
            take(x, 0, call);
            return;
        }
        if (!(PyList_Check(x) || PyTuple_Check(x)) || PySequence_Fast_GET_SIZE(x) != vranks ||
            vranks > kMost) {
            PyErr_Format(PyExc_ValueError, "loopback session: %s must be a list of %d tensors", what,
                         vranks);
            throw Raised{};
        }
        for (int v = 0; v < vranks; ++v) { take(PySequence_Fast_GET_ITEM(x, v), v, call); }
    }

  private:
    void take(PyObject *o, int v, const char *call)
    {
        if (o == Py_None && v > 0) {
            ptr[v] = nullptr;
            return;
        }
        const at::Tensor &t = tensor_of(o, call);
        ptr[v] = checked_ptr(t, call);
        if (v == 0) {
            count = static_cast<unsigned long long>(t.numel());
            dt = supported_dtype(t);
        }
    }
};

// Same for destinations, where None may stand for any rank's and for all of them.
void dest_ptrs(PyObject *x, int vranks, const char *call, void **ptr)
{
    if (vranks <= 1) {
        ptr[0] = x == Py_None ? nullptr : checked_ptr(tensor_of(x, call), call);
        return;
    }
    if (!(PyList_Check(x) || PyTuple_Check(x)) || PySequence_Fast_GET_SIZE(x) != vranks ||
        vranks > PerRank::kMost) {
        PyErr_Format(PyExc_ValueError, "loopback session: out must be a list of %d tensors", vranks);
        throw Raised{};
    }
    for (int v = 0; v < vranks; ++v) {
        PyObject *o = PySequence_Fast_GET_ITEM(x, v);
        ptr[v] = o == Py_None ? nullptr : checked_ptr(tensor_of(o, call), call);
    }
}

struct Args {
    PyObject *const *a;
    Py_ssize_t n;
    void expect(Py_ssize_t want) const
    {
        if (n != want) {
            PyErr_Format(PyExc_TypeError, "%zd arguments expected, got %zd", want, n);
            throw Raised{};
        }
    }
    long integer(int i) const
    {
        const long v = PyLong_AsLong(a[i]);
        if (v == -1 && PyErr_Occurred()) { throw Raised{}; }
        return v;
    }
    void *pointer(int i) const
    {
        void *p = PyLong_AsVoidPtr(a[i]);
        if (p == nullptr && PyErr_Occurred()) { throw Raised{}; }
        return p;
    }
    double real(int i) const
    {
        if (a[i] == Py_None) { return 1.0; }
        const double v = PyFloat_AsDouble(a[i]);
        if (v == -1.0 && PyErr_Occurred()) { throw Raised{}; }
        return v;
    }
};

template <typename F>
PyObject *guarded(F f)
{
    try {
        return PyLong_FromLong(f());
    } catch (const Raised &) {
        return nullptr;
    } catch (const std::exception &e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

#define WITHOUT_GIL(rc, call)                                                  \
    do {                                                                       \
        Py_BEGIN_ALLOW_THREADS rc = (call);                                    \
        Py_END_ALLOW_THREADS                                                   \
    } while (0)

// (handle, vranks, tensor, out | None, op, scale | None, algo, stream)
PyObject *all_reduce(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    return guarded([&]() -> long {
        const Args g{a, n};
        g.expect(8);
        void *h = g.pointer(0), *stream = g.pointer(7);
        const int vranks = static_cast<int>(g.integer(1));
        PerRank in(a[2], vranks, "tensor", "all_reduce");
        void *out_ptr[PerRank::kMost];
        void **out = in.ptr;
        if (a[3] != Py_None) {
            dest_ptrs(a[3], vranks, "all_reduce", out_ptr);
            out = out_ptr;
        }
        const int op = static_cast<int>(g.integer(4)), algo = static_cast<int>(g.integer(6));
        const double scale = g.real(5);
        int rc;
        WITHOUT_GIL(rc, stdmlc_dw_all_reduce(h, in.ptr, out, in.count, in.dt, op, scale, algo, stream));
        return rc;
    });
}

// (handle, vranks, tensor, out, op, root, scale | None, stream); out may be None for a rank
PyObject *reduce(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    return guarded([&]() -> long {
        const Args g{a, n};
        g.expect(8);
        void *h = g.pointer(0), *stream = g.pointer(7);
        const int vranks = static_cast<int>(g.integer(1));
        PerRank in(a[2], vranks, "tensor", "reduce");
        void *out[PerRank::kMost];
        dest_ptrs(a[3], vranks, "reduce", out);
        const int op = static_cast<int>(g.integer(4)), root = static_cast<int>(g.integer(5));
        const double scale = g.real(6);
        int rc;
        WITHOUT_GIL(rc, stdmlc_dw_reduce(h, in.ptr, out, in.count, in.dt, op, root, scale, stream));
        return rc;
    });
}

// (handle, vranks, world, tensor, out, stream)
PyObject *all_gather(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    return guarded([&]() -> long {
        const Args g{a, n};
        g.expect(6);
        void *h = g.pointer(0), *stream = g.pointer(5);
        const int vranks = static_cast<int>(g.integer(1));
        const unsigned long long world = static_cast<unsigned long long>(g.integer(2));
        PerRank in(a[3], vranks, "tensor", "all_gather");
        PerRank out(a[4], vranks, "out", "all_gather");
        if (out.count != in.count * world) {
            PyErr_SetString(PyExc_ValueError,
                            "all_gather: out must hold world * tensor.numel() elements");
            throw Raised{};
        }
        int rc;
        WITHOUT_GIL(rc, stdmlc_dw_all_gather(h, in.ptr, out.ptr, in.count, in.dt, stream));
        return rc;
    });
}

// (handle, vranks, tensor, out | None, root, stream)
PyObject *broadcast(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    return guarded([&]() -> long {
        const Args g{a, n};
        g.expect(6);
        void *h = g.pointer(0), *stream = g.pointer(5);
        const int vranks = static_cast<int>(g.integer(1));
        PerRank in(a[2], vranks, "tensor", "broadcast");
        void *out_ptr[PerRank::kMost];
        void **out = in.ptr;
        if (a[3] != Py_None) {
            dest_ptrs(a[3], vranks, "broadcast", out_ptr);
            out = out_ptr;
        }
        const int root = static_cast<int>(g.integer(4));
        int rc;
        WITHOUT_GIL(rc, stdmlc_dw_broadcast(h, in.ptr, out, in.count, in.dt, root, stream));
        return rc;
    });
}

// Addresses of one rank's tensors; of rank 0's operands also the counts and the
// dtype.  `dt` null: the dtype does not matter (destinations).  False: rank 0's
// tensors have several dtypes.
bool take_list(PyObject *seq, size_t n, int *dt, unsigned long long *counts, void **ptr)
{
    constexpr const char *kCall = "group_all_reduce";
    for (size_t i = 0; i < n; ++i) {
        const at::Tensor &t = tensor_of(PySequence_Fast_GET_ITEM(seq, i), kCall);
        if (dt != nullptr) {
            const int code = supported_dtype(t);
            if (*dt < 0) { *dt = code; }
            if (code != *dt) {
                if (counts != nullptr) { return false; }
                PyErr_SetString(PyExc_ValueError, "group_all_reduce: one dtype per call");
                throw Raised{};
            }
        }
        if (counts != nullptr) { counts[i] = static_cast<unsigned long long>(t.numel()); }
        ptr[i] = checked_ptr(t, kCall);
    }
    return true;
}

// Addresses of every rank's tensors, [rank][tensor].
bool take_group(PyObject *x, int vranks, const char *what, size_t *n, int *dt,
                std::vector<unsigned long long> *counts, std::vector<void *> &ptr)
{
    if (vranks > 1 && (!(PyList_Check(x) || PyTuple_Check(x)) ||
                       PySequence_Fast_GET_SIZE(x) != vranks)) {
        PyErr_Format(PyExc_ValueError, "loopback session: %s must be a list of %d tensors", what,
                     vranks);
        throw Raised{};
    }
    for (int v = 0; v < vranks || v == 0; ++v) {
        PyObject *item = vranks > 1 ? PySequence_Fast_GET_ITEM(x, v) : x;
        if (!(PyList_Check(item) || PyTuple_Check(item))) {
            PyErr_SetString(PyExc_ValueError, "group_all_reduce: lists of tensors expected");
            throw Raised{};
        }
        const size_t len = static_cast<size_t>(PySequence_Fast_GET_SIZE(item));
        if (counts != nullptr && v == 0) {
            *n = len;
            counts->resize(len);
        }
        if (len != *n) {
            PyErr_SetString(PyExc_ValueError,
                            "group_all_reduce: every rank needs the same number of tensors");
            throw Raised{};
        }
        ptr.resize(ptr.size() + len);
        if (!take_list(item, len, dt, (counts != nullptr && v == 0) ? counts->data() : nullptr,
                       ptr.data() + ptr.size() - len)) {
            return false;
        }
    }
    return true;
}

// (handle, vranks, tensors, outs | None, wire dtype code | -1, op, scale | None, algo, stream)
PyObject *group_all_reduce(PyObject *, PyObject *const *a, Py_ssize_t nargs)
{
    return guarded([&]() -> long {
        const Args g{a, nargs};
        g.expect(9);
        void *h = g.pointer(0), *stream = g.pointer(8);
        const int vranks = static_cast<int>(g.integer(1));
        // kept between calls of a thread: a step's gradients come in the same numbers
        static thread_local std::vector<void *> in, out;
        static thread_local std::vector<unsigned long long> counts;
        in.clear();
        out.clear();
        size_t n = 0;
        int dt = -1;
        if (!take_group(a[2], vranks, "tensors", &n, &dt, &counts, in)) { return kMixedDtypes; }
        if (n == 0) { return 0; }
        if (a[3] != Py_None) {
            take_group(a[3], vranks, "outs", &n, nullptr, nullptr, out);
        }
        int wire = static_cast<int>(g.integer(4)), user = -1;
        if (wire < 0 || wire == dt) {
            wire = dt;
        } else {
            user = dt;
        }
        const int op = static_cast<int>(g.integer(5)), algo = static_cast<int>(g.integer(7));
        const double scale = g.real(6);
        void *const *outs = a[3] != Py_None ? out.data() : in.data();
        int rc;
        WITHOUT_GIL(rc, stdmlc_dw_group_all_reduce(h, n, in.data(), outs, counts.data(), wire, op,
                                                   user, scale, algo, stream));
        return rc;
    });
}

PyMethodDef kMethods[] = {
    {"all_reduce", reinterpret_cast<PyCFunction>(all_reduce), METH_FASTCALL, nullptr},
    {"reduce", reinterpret_cast<PyCFunction>(reduce), METH_FASTCALL, nullptr},
    {"all_gather", reinterpret_cast<PyCFunction>(all_gather), METH_FASTCALL, nullptr},
    {"broadcast", reinterpret_cast<PyCFunction>(broadcast), METH_FASTCALL, nullptr},
    {"group_all_reduce", reinterpret_cast<PyCFunction>(group_all_reduce), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_fastcall",
                       "Collectives on CUDA tensors: argument checks and the library call.", -1,
                       kMethods, nullptr, nullptr, nullptr, nullptr};
}  // namespace

PyMODINIT_FUNC PyInit__fastcall()
{
    PyObject *m = PyModule_Create(&kModule);
    if (m != nullptr) { PyModule_AddIntConstant(m, "MIXED_DTYPES", kMixedDtypes); }
    return m;
}
