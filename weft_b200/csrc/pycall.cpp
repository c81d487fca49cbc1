// The call path of a CompiledKernel as native code (extension module weft_b200._pycall).
//
// CompiledKernel.__call__ checks each argument against the kernel's ABI record and calls a C symbol through ctypes; in
// Python that is 5 to 8 microseconds per call, more than most decode kernels run.  A Plan holds the same record as plain
// arrays and does the same checks on the Buffers of a call.  It decides nothing on its own: whenever an argument is not a
// Buffer that passes every check (or a keyword was given, or the kernel is closed) it answers None and the Python path
// runs, which raises the error that belongs to the mistake -- so the rules and their messages stand in one place.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <structmember.h>

#include <cstdint>
#include <cstring>

namespace {

constexpr int MAX_ARGS = 8, MAX_RANK = 4, MAX_EXTENTS = 6, MAX_DIMS = 6;

struct Param {
    PyObject *encoding;               // interned str
    int rank;
    int symbol[MAX_RANK];             // index of the extent, or -1: the literal below
    long long literal[MAX_RANK];
    long long record_elements, storage_bytes;
    uint64_t alignment;
    int alias;                        // group number: ranges of different groups must not overlap
    bool writable;
};

struct Plan {
    PyObject_HEAD
    vectorcallfunc call;
    PyTypeObject *buffer_type;
    Py_ssize_t at_address, at_nbytes, at_readonly, at_shape, at_encoding;    // slots of a Buffer
    int args, extents, dims;
    Param params[MAX_ARGS];
    int dim[MAX_DIMS];                // extent that goes into each trailing size_t of the symbol
    uintptr_t symbol;
    bool open;
};

PyObject *slot(PyObject *o, Py_ssize_t offset) { return *reinterpret_cast<PyObject **>(reinterpret_cast<char *>(o) + offset); }

// Offset of a __slots__ member of `type`, or -1.
Py_ssize_t slot_offset(PyObject *type, const char *name) {
    PyObject *d = PyObject_GetAttrString(type, name);
    Py_ssize_t at = -1;
    if (d && Py_IS_TYPE(d, &PyMemberDescr_Type)) {
        const PyMemberDef *m = reinterpret_cast<PyMemberDescrObject *>(d)->d_member;
        if (m->type == T_OBJECT_EX) at = m->offset;
    }
    Py_XDECREF(d);
    PyErr_Clear();
    return at;
}

int call_symbol(uintptr_t f, const uint64_t *a, int n) {
    using U = uint64_t;
    switch (n) {     // every argument of these symbols is a pointer or a size_t
    case 3: return reinterpret_cast<int (*)(U, U, U)>(f)(a[0], a[1], a[2]);
    case 4: return reinterpret_cast<int (*)(U, U, U, U)>(f)(a[0], a[1], a[2], a[3]);
    case 5: return reinterpret_cast<int (*)(U, U, U, U, U)>(f)(a[0], a[1], a[2], a[3], a[4]);
    case 6: return reinterpret_cast<int (*)(U, U, U, U, U, U)>(f)(a[0], a[1], a[2], a[3], a[4], a[5]);
    case 7: return reinterpret_cast<int (*)(U, U, U, U, U, U, U)>(f)(a[0], a[1], a[2], a[3], a[4], a[5], a[6]);
    case 8: return reinterpret_cast<int (*)(U, U, U, U, U, U, U, U)>(f)(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7]);
    case 9: return reinterpret_cast<int (*)(U, U, U, U, U, U, U, U, U)>(f)(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8]);
    default: return reinterpret_cast<int (*)(U, U, U, U, U, U, U, U, U, U)>(f)(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9]);
    }
}

// Checks the arguments and fills the C argument list; false: the Python path has to look at this call.
bool bind(const Plan *p, PyObject *const *args, uint64_t *out) {
    long long extent[MAX_EXTENTS];
    uint64_t lo[MAX_ARGS], hi[MAX_ARGS];
    for (int i = 0; i < p->extents; ++i) extent[i] = -1;
    for (int i = 0; i < p->args; ++i) {
        const Param &q = p->params[i];
        PyObject *b = args[i];
        if (!Py_IS_TYPE(b, p->buffer_type)) return false;
        PyObject *address = slot(b, p->at_address), *nbytes = slot(b, p->at_nbytes), *readonly = slot(b, p->at_readonly), *shape = slot(b, p->at_shape),
                 *encoding = slot(b, p->at_encoding);
        if (!address || !nbytes || !readonly || !shape || !encoding || !PyLong_CheckExact(address) || !PyLong_CheckExact(nbytes) || !PyTuple_CheckExact(shape)) return false;
        if (encoding != q.encoding && (!PyUnicode_CheckExact(encoding) || PyUnicode_Compare(encoding, q.encoding) != 0)) return false;
        if (PyTuple_GET_SIZE(shape) != q.rank) return false;
        long long elements = 1, last = 0;
        for (int r = 0; r < q.rank; ++r) {
            PyObject *e = PyTuple_GET_ITEM(shape, r);
            if (!PyLong_CheckExact(e)) return false;
            last = PyLong_AsLongLong(e);
            if (last < 0) { PyErr_Clear(); return false; }
            if (q.symbol[r] < 0) {
                if (last != q.literal[r]) return false;
            } else if (extent[q.symbol[r]] < 0) {
                extent[q.symbol[r]] = last;
            } else if (last != extent[q.symbol[r]]) {
                return false;
            }
            if (__builtin_mul_overflow(elements, last, &elements)) return false;
        }
        if (q.rank && last % q.record_elements) return false;
        long long span;
        if (__builtin_mul_overflow(elements / q.record_elements, q.storage_bytes, &span)) return false;
        const uint64_t at = PyLong_AsUnsignedLongLong(address);
        const long long bytes = PyLong_AsLongLong(nbytes);
        if (PyErr_Occurred()) { PyErr_Clear(); return false; }
        if (span > bytes || (span && at % q.alignment)) return false;
        if (q.writable && readonly != Py_False) return false;
        lo[i] = at;
        hi[i] = at + (uint64_t)span;
        if (span)
            for (int j = 0; j < i; ++j)
                if (p->params[j].alias != q.alias && hi[j] > lo[j] && lo[i] < hi[j] && lo[j] < hi[i]) return false;
        out[i] = at;
    }
    for (int d = 0; d < p->dims; ++d) {
        const long long v = extent[p->dim[d]];
        if (v < 0) return false;
        out[p->args + d] = (uint64_t)v;
    }
    return true;
}

// plan(*buffers) -> None: not taken; else the symbol's return value
PyObject *plan_call(PyObject *self, PyObject *const *args, size_t nargsf, PyObject *kwnames) {
    Plan *p = reinterpret_cast<Plan *>(self);
    uint64_t list[MAX_ARGS + MAX_DIMS];
    if (!p->open || kwnames || PyVectorcall_NARGS(nargsf) != p->args || !bind(p, args, list)) Py_RETURN_NONE;
    const uintptr_t symbol = p->symbol;
    const int count = p->args + p->dims;
    int result;
    Py_BEGIN_ALLOW_THREADS
    result = call_symbol(symbol, list, count);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(result);
}

PyObject *plan_close(PyObject *self, PyObject *) {
    reinterpret_cast<Plan *>(self)->open = false;
    Py_RETURN_NONE;
}

void plan_free(PyObject *self) {
    Plan *p = reinterpret_cast<Plan *>(self);
    PyTypeObject *type = Py_TYPE(self);
    for (int i = 0; i < p->args; ++i) Py_XDECREF(p->params[i].encoding);
    Py_XDECREF(reinterpret_cast<PyObject *>(p->buffer_type));
    type->tp_free(self);
    Py_DECREF(type);
}

// Plan(Buffer, symbol address, [(encoding, (extent index or ~literal, ...), record elements, storage bytes, alignment, alias
// group, writable), ...], (extent index of each C dimension, ...), number of extents)
PyObject *plan_new(PyTypeObject *type, PyObject *args, PyObject *) {
    PyObject *buffer, *params, *dims;
    unsigned long long symbol;
    int extents;
    if (!PyArg_ParseTuple(args, "O!KO!O!i", &PyType_Type, &buffer, &symbol, &PyList_Type, &params, &PyTuple_Type, &dims, &extents)) return nullptr;
    Plan *p = reinterpret_cast<Plan *>(type->tp_alloc(type, 0));
    if (!p) return nullptr;
    p->call = plan_call;
    p->buffer_type = reinterpret_cast<PyTypeObject *>(Py_NewRef(buffer));
    p->symbol = (uintptr_t)symbol;
    p->extents = extents;
    p->at_address = slot_offset(buffer, "address");
    p->at_nbytes = slot_offset(buffer, "nbytes");
    p->at_readonly = slot_offset(buffer, "readonly");
    p->at_shape = slot_offset(buffer, "shape");
    p->at_encoding = slot_offset(buffer, "encoding");
    const Py_ssize_t count = PyList_GET_SIZE(params) + PyTuple_GET_SIZE(dims);
    bool ok = p->at_address >= 0 && p->at_nbytes >= 0 && p->at_readonly >= 0 && p->at_shape >= 0 && p->at_encoding >= 0 && extents >= 0 && extents <= MAX_EXTENTS &&
              PyList_GET_SIZE(params) <= MAX_ARGS && PyTuple_GET_SIZE(dims) <= MAX_DIMS && count >= 3 && count <= 10;
    for (Py_ssize_t i = 0; ok && i < PyList_GET_SIZE(params); ++i) {
        Param &q = p->params[i];
        PyObject *encoding, *shape;
        int writable;
        if (!PyArg_ParseTuple(PyList_GET_ITEM(params, i), "UO!LLKip", &encoding, &PyTuple_Type, &shape, &q.record_elements, &q.storage_bytes, &q.alignment, &q.alias, &writable)) {
            Py_DECREF(p);
            return nullptr;
        }
        ok = PyTuple_GET_SIZE(shape) <= MAX_RANK && q.record_elements > 0 && q.alignment > 0;
        q.writable = writable != 0;
        q.rank = (int)PyTuple_GET_SIZE(shape);
        for (int r = 0; ok && r < q.rank; ++r) {
            const long long v = PyLong_AsLongLong(PyTuple_GET_ITEM(shape, r));
            q.symbol[r] = v >= 0 ? (int)v : -1;
            q.literal[r] = v >= 0 ? 0 : ~v;
            ok = !PyErr_Occurred() && (v < 0 || v < extents);
        }
        q.encoding = Py_NewRef(encoding);
        PyUnicode_InternInPlace(&q.encoding);
        p->args = (int)i + 1;
    }
    for (Py_ssize_t d = 0; ok && d < PyTuple_GET_SIZE(dims); ++d) {
        const long v = PyLong_AsLong(PyTuple_GET_ITEM(dims, d));
        ok = !PyErr_Occurred() && v >= 0 && v < extents;
        p->dim[d] = (int)v;
        p->dims = (int)d + 1;
    }
    if (!ok) {
        Py_DECREF(p);
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "this kernel's record does not fit the native call path");
        return nullptr;
    }
    p->open = true;
    return reinterpret_cast<PyObject *>(p);
}

PyMethodDef plan_methods[] = {{"close", plan_close, METH_NOARGS, "From now on every call is left to the Python path."}, {nullptr, nullptr, 0, nullptr}};
PyMemberDef plan_members[] = {{"__vectorcalloffset__", T_PYSSIZET, offsetof(Plan, call), READONLY, nullptr}, {nullptr, 0, 0, 0, nullptr}};
PyType_Slot plan_slots[] = {{Py_tp_new, reinterpret_cast<void *>(plan_new)}, {Py_tp_dealloc, reinterpret_cast<void *>(plan_free)},
                            {Py_tp_call, reinterpret_cast<void *>(PyVectorcall_Call)}, {Py_tp_methods, plan_methods}, {Py_tp_members, plan_members}, {0, nullptr}};
PyType_Spec plan_spec = {"weft_b200._pycall.Plan", sizeof(Plan), 0, Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL, plan_slots};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_pycall", nullptr, -1, nullptr, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__pycall(void) {
    PyObject *m = PyModule_Create(&module), *type = PyType_FromSpec(&plan_spec);
    if (!m || !type || PyModule_AddObject(m, "Plan", type) < 0) return nullptr;
    return m;
}
