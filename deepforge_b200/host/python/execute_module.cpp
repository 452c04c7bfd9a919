// CPython entry to df_execute / df_execute_on: the UID -> pointer dict is read straight into two arrays. The ctypes form
// of the same call builds two ctypes arrays and converts every argument in Python, 2.5 us of the 5.4 us that one small
// execute() took; this takes 0.2.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include "deepforge_b200.h"

#include <memory>
#include <new>

namespace {

// An address or a UID as ctypes takes it: an int of any sign, cut to 64 bits.
bool integer(PyObject* object, std::uint64_t& value) {
    if (!PyLong_Check(object)) {
        PyErr_Format(PyExc_TypeError, "an integer is required (got type %s)", Py_TYPE(object)->tp_name);
        return false;
    }
    value = PyLong_AsUnsignedLongLongMask(object);
    return !(value == static_cast<std::uint64_t>(-1) && PyErr_Occurred());
}

bool pointer(PyObject* object, void*& value) {   // None counts as null
    std::uint64_t bits = 0;
    if (object != Py_None && !integer(object, bits)) return false;
    value = reinterpret_cast<void*>(bits);
    return true;
}

// execute(executable, pack, workspace, stream, on_stream) -> Status code
PyObject* execute(PyObject*, PyObject* const* arguments, Py_ssize_t count) {
    if (count != 5) {
        PyErr_SetString(PyExc_TypeError, "execute takes (executable, pack, workspace, stream, on_stream)");
        return nullptr;
    }
    void *executable, *workspace, *stream;
    if (!pointer(arguments[0], executable) || !pointer(arguments[2], workspace) || !pointer(arguments[3], stream)) return nullptr;
    PyObject* pack = arguments[1];
    if (!PyDict_Check(pack)) {
        PyErr_SetString(PyExc_TypeError, "the pack must be a dict");
        return nullptr;
    }
    constexpr Py_ssize_t kFew = 32;
    std::int64_t few_uids[kFew];
    void* few_pointers[kFew];
    std::int64_t* uids = few_uids;
    void** pointers = few_pointers;
    std::unique_ptr<std::int64_t[]> many_uids;
    std::unique_ptr<void*[]> many_pointers;
    const Py_ssize_t size = PyDict_GET_SIZE(pack);
    if (size > kFew) {
        many_uids.reset(new (std::nothrow) std::int64_t[size]);
        many_pointers.reset(new (std::nothrow) void*[size]);
        if (!many_uids || !many_pointers) return PyErr_NoMemory();
        uids = many_uids.get();
        pointers = many_pointers.get();
    }
    Py_ssize_t position = 0, filled = 0;
    PyObject *key, *value;
    while (filled < size && PyDict_Next(pack, &position, &key, &value)) {
        std::uint64_t uid;
        if (!integer(key, uid) || !pointer(value, pointers[filled])) return nullptr;
        uids[filled++] = static_cast<std::int64_t>(uid);
    }
    const int on_stream = PyObject_IsTrue(arguments[4]);
    if (on_stream < 0) return nullptr;
    int code;
    Py_BEGIN_ALLOW_THREADS
    code = on_stream ? df_execute_on(static_cast<df_executable*>(executable), stream, uids, pointers, static_cast<size_t>(filled), workspace)
                     : df_execute(static_cast<df_executable*>(executable), nullptr, uids, pointers, static_cast<size_t>(filled), workspace);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(code);
}

PyMethodDef methods[] = {
    {"execute", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(execute)), METH_FASTCALL, "df_execute / df_execute_on on a UID -> pointer dict"},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_execute", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__execute() { return PyModule_Create(&module); }
