// Python side of the tree selects and backups: takes the device pointers and shapes out of the caller's mapping of arrays and
// calls the launchers of libmctsnc_b200.so, whose addresses Python hands over once (`bind`).
//
// A launch has up to 23 arguments.  Gathering them in Python and passing them through ctypes took 12 us of host time, more
// than the kernels of a small wave run (100 trees x 19 edges: 11 us select, 3 us backup); here it takes 1 to 2 us.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include "../../include/duct_b200.h"
#include "../../include/puct_b200.h"

namespace {

// the launchers' types are those of the public headers: a launcher whose arguments change does not compile here
struct {
    decltype(&puct_select_winner_recalc_launch) puct_select;
    decltype(&puct_select_virtual_loss_launch) puct_select_vl;
    decltype(&puct_backup_launch) puct_backup;
    decltype(&puct_v2_select_launch) puct_v2_select;
    decltype(&puct_v2_backup_launch) puct_v2_backup;
    decltype(&duct_select_launch) duct_select;
    decltype(&duct_backup_launch) duct_backup;
} fn;

enum Key { EDGE_CHILD, EDGE_PRIOR, EDGE_W, EDGE_N, EDGE_INFLIGHT, NODE_INFLIGHT, NODE_EXPAND_INFLIGHT, NODE_EXPANDED, NODE_COUNT,
           OUT_SELECTED, OUT_PATH, OUT_LEN, CHILD, NODE_PRIOR, NODE_W, NODE_N, NODE_TERMINAL, TREES, WARPS, N_KEYS };
const char *const KEY_NAMES[N_KEYS] = {"edge_child", "edge_prior", "edge_w", "edge_n", "edge_inflight", "node_inflight", "node_expand_inflight",
                                       "node_expanded", "node_count", "out_selected", "out_path", "out_len", "child", "node_prior", "node_w",
                                       "node_n", "node_terminal", "trees", "warps"};
PyObject *key_objects[N_KEYS];
PyObject *str_data_ptr, *str_shape, *str_interface, *str_data;

// new reference to d[key]
PyObject *item(PyObject *d, int key) {
    if (PyDict_CheckExact(d)) {
        PyObject *v = PyDict_GetItemWithError(d, key_objects[key]);
        if (!v) {
            if (!PyErr_Occurred()) PyErr_SetObject(PyExc_KeyError, key_objects[key]);
            return nullptr;
        }
        Py_INCREF(v);
        return v;
    }
    return PyObject_GetItem(d, key_objects[key]);
}

// device address of an array: torch tensors (data_ptr), anything with __cuda_array_interface__, None = null
bool address(PyObject *a, void **out) {
    if (a == Py_None) {
        *out = nullptr;
        return true;
    }
    PyObject *p = PyObject_CallMethodNoArgs(a, str_data_ptr);
    if (!p) {
        if (!PyErr_ExceptionMatches(PyExc_AttributeError)) return false;
        PyErr_Clear();
        PyObject *interface = PyObject_GetAttr(a, str_interface);
        if (!interface) {
            if (PyErr_ExceptionMatches(PyExc_AttributeError)) PyErr_Format(PyExc_TypeError, "not a device array: %R", (PyObject *)Py_TYPE(a));
            return false;
        }
        PyObject *data = PyObject_GetItem(interface, str_data);
        Py_DECREF(interface);
        if (!data) return false;
        p = PySequence_GetItem(data, 0);
        Py_DECREF(data);
        if (!p) return false;
    }
    *out = PyLong_AsVoidPtr(p);
    Py_DECREF(p);
    return !(*out == nullptr && PyErr_Occurred());
}

bool address_of(PyObject *d, int key, void **out) {
    PyObject *a = item(d, key);
    if (!a) return false;
    const bool ok = address(a, out);
    Py_DECREF(a);
    return ok;
}

bool integer_of(PyObject *d, int key, int *out) {
    PyObject *v = item(d, key);
    if (!v) return false;
    PyObject *n = PyNumber_Long(v);
    Py_DECREF(v);
    if (!n) return false;
    const long x = PyLong_AsLong(n);
    Py_DECREF(n);
    if (x == -1 && PyErr_Occurred()) return false;
    *out = (int)x;
    return true;
}

// shape[index] of d[key] for each of `count` indexes
bool extents_of(PyObject *d, int key, const int *index, int count, int *out) {
    PyObject *a = item(d, key);
    if (!a) return false;
    PyObject *shape = PyObject_GetAttr(a, str_shape);
    Py_DECREF(a);
    if (!shape) return false;
    bool ok = true;
    for (int i = 0; i < count && ok; i++) {
        PyObject *n = PySequence_GetItem(shape, index[i]);
        ok = n != nullptr;
        if (!ok) break;
        const long x = PyLong_AsLong(n);
        Py_DECREF(n);
        if (x == -1 && PyErr_Occurred()) ok = false;
        out[i] = (int)x;
    }
    Py_DECREF(shape);
    return ok;
}

struct Shape {
    int trees, nodes, edges, warps, depth;
};

bool shape_of(PyObject *d, int key, int node_axis, int edge_axis, Shape *s) {
    const int axes[2] = {node_axis, edge_axis}, last = 2;
    int ext[2];
    if (!integer_of(d, TREES, &s->trees) || !extents_of(d, key, axes, 2, ext) || !integer_of(d, WARPS, &s->warps) ||
        !extents_of(d, OUT_PATH, &last, 1, &s->depth))
        return false;
    s->nodes = ext[0];
    s->edges = ext[1];
    return true;
}

// pointers of d's arrays, in the order of `keys`
template <int N>
bool addresses(PyObject *d, const int (&keys)[N], void **out) {
    for (int i = 0; i < N; i++)
        if (!address_of(d, keys[i], &out[i])) return false;
    return true;
}

bool count_is(Py_ssize_t got, Py_ssize_t want) {
    if (got == want) return true;
    PyErr_Format(PyExc_TypeError, "%zd arguments, expected %zd", got, want);
    return false;
}

// the arguments of a launch: as many as there should be, and launchers to hand them to
bool ready(Py_ssize_t got, Py_ssize_t want) {
    if (!fn.duct_backup) PyErr_SetString(PyExc_RuntimeError, "no launchers: bind() has not been called");
    return fn.duct_backup && count_is(got, want);
}

// the launch itself: other Python threads may run meanwhile (it waits where the device's queue is full)
template <typename Launch>
PyObject *launched(Launch launch) {
    int code;
    Py_BEGIN_ALLOW_THREADS
    code = launch();
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(code);
}

float real(PyObject *o) { return (float)PyFloat_AsDouble(o); }
int whole(PyObject *o) { return (int)PyLong_AsLong(o); }

// puct_select(d, cpuct, c_pw, alpha_pw, soft_winner, virtual_loss, stream) -> error code
PyObject *puct_select(PyObject *, PyObject *const *a, Py_ssize_t n) {
    if (!ready(n, 7)) return nullptr;
    const float cpuct = real(a[1]), c_pw = real(a[2]), alpha = real(a[3]);
    const int soft = whole(a[4]), vl = whole(a[5]);
    void *stream = PyLong_AsVoidPtr(a[6]), *p[11];
    Shape s;
    static const int keys[11] = {EDGE_CHILD, EDGE_PRIOR, EDGE_W, EDGE_N, EDGE_INFLIGHT, NODE_EXPAND_INFLIGHT, NODE_EXPANDED, NODE_COUNT,
                                 OUT_SELECTED, OUT_PATH, OUT_LEN};
    if (PyErr_Occurred() || !shape_of(a[0], EDGE_CHILD, 1, 2, &s) || !addresses(a[0], keys, p)) return nullptr;
    return launched([&] {
        if (vl == 1)
            return fn.puct_select(cpuct, c_pw, alpha, soft, (int *)p[0], (float *)p[1], (float *)p[2], (int *)p[3], (int *)p[4], (int *)p[5],
                                  (int *)p[6], (int *)p[7], (int *)p[8], (int *)p[9], (int *)p[10], s.trees, s.nodes, s.edges, s.warps,
                                  s.depth, stream);
        return fn.puct_select_vl(cpuct, c_pw, alpha, soft, vl, (int *)p[0], (float *)p[1], (float *)p[2], (int *)p[3], (int *)p[4],
                                 (int *)p[5], (int *)p[6], (int *)p[7], (int *)p[8], (int *)p[9], (int *)p[10], s.trees, s.nodes, s.edges,
                                 s.warps, s.depth, stream);
    });
}

// puct_backup(d, values, virtual_loss, stream) -> error code
PyObject *puct_backup(PyObject *, PyObject *const *a, Py_ssize_t n) {
    if (!ready(n, 4)) return nullptr;
    const int vl = whole(a[2]);
    void *stream = PyLong_AsVoidPtr(a[3]), *values, *p[8];
    Shape s;
    static const int keys[8] = {EDGE_W, EDGE_N, EDGE_INFLIGHT, NODE_EXPAND_INFLIGHT, NODE_COUNT, OUT_SELECTED, OUT_PATH, OUT_LEN};
    if (PyErr_Occurred() || !address(a[1], &values) || !shape_of(a[0], EDGE_CHILD, 1, 2, &s) || !addresses(a[0], keys, p)) return nullptr;
    return launched([&] { return fn.puct_backup(vl, (float *)p[0], (int *)p[1], (int *)p[2], (int *)p[3], (int *)p[4], (int *)p[5], (int *)p[6],
                                          (int *)p[7], (float *)values, s.trees, s.nodes, s.edges, s.warps, s.depth, stream); });
}

// puct_v2_select(d, variant, cpuct, c_pw, alpha_pw, stream) -> error code
PyObject *puct_v2_select(PyObject *, PyObject *const *a, Py_ssize_t n) {
    if (!ready(n, 6)) return nullptr;
    const int variant = whole(a[1]);
    const float cpuct = real(a[2]), c_pw = real(a[3]), alpha = real(a[4]);
    void *stream = PyLong_AsVoidPtr(a[5]), *p[11];
    Shape s;
    static const int keys[11] = {EDGE_CHILD, EDGE_PRIOR, EDGE_W, EDGE_N, NODE_INFLIGHT, NODE_EXPAND_INFLIGHT, NODE_EXPANDED, NODE_COUNT,
                                 OUT_SELECTED, OUT_PATH, OUT_LEN};
    if (PyErr_Occurred() || !shape_of(a[0], EDGE_CHILD, 1, 2, &s) || !addresses(a[0], keys, p)) return nullptr;
    return launched([&] { return fn.puct_v2_select(variant, cpuct, c_pw, alpha, (int *)p[0], (float *)p[1], (float *)p[2], (int *)p[3], (int *)p[4],
                                             (int *)p[5], (int *)p[6], (int *)p[7], (int *)p[8], (int *)p[9], (int *)p[10], s.trees, s.nodes,
                                             s.edges, s.warps, s.depth, stream); });
}

// puct_v2_backup(d, values, virtual_loss, stream) -> error code
PyObject *puct_v2_backup(PyObject *, PyObject *const *a, Py_ssize_t n) {
    if (!ready(n, 4)) return nullptr;
    const int vl = whole(a[2]);
    void *stream = PyLong_AsVoidPtr(a[3]), *values, *p[9];
    Shape s;
    static const int keys[9] = {EDGE_CHILD, EDGE_W, EDGE_N, NODE_INFLIGHT, NODE_EXPAND_INFLIGHT, NODE_COUNT, OUT_SELECTED, OUT_PATH, OUT_LEN};
    if (PyErr_Occurred() || !address(a[1], &values) || !shape_of(a[0], EDGE_CHILD, 1, 2, &s) || !addresses(a[0], keys, p)) return nullptr;
    return launched([&] { return fn.puct_v2_backup(vl, (int *)p[0], (float *)p[1], (int *)p[2], (int *)p[3], (int *)p[4], (int *)p[5], (int *)p[6],
                                             (int *)p[7], (int *)p[8], (float *)values, s.trees, s.nodes, s.edges, s.warps, s.depth, stream); });
}

// duct_select(d, cpuct, virtual_loss, stream) -> error code
PyObject *duct_select(PyObject *, PyObject *const *a, Py_ssize_t n) {
    if (!ready(n, 4)) return nullptr;
    const float cpuct = real(a[1]);
    const int vl = whole(a[2]);
    void *stream = PyLong_AsVoidPtr(a[3]), *p[10];
    Shape s;
    static const int keys[10] = {CHILD, NODE_PRIOR, NODE_W, NODE_N, NODE_INFLIGHT, NODE_TERMINAL, NODE_COUNT, OUT_SELECTED, OUT_PATH, OUT_LEN};
    if (PyErr_Occurred() || !shape_of(a[0], NODE_PRIOR, 1, 3, &s) || !addresses(a[0], keys, p)) return nullptr;
    return launched([&] { return fn.duct_select(cpuct, vl, (int *)p[0], (float *)p[1], (float *)p[2], (int *)p[3], (int *)p[4], (int *)p[5],
                                          (int *)p[6], (int *)p[7], (int *)p[8], (int *)p[9], s.trees, s.nodes, s.edges, s.warps, s.depth,
                                          stream); });
}

// duct_backup(d, values, new_child, virtual_loss, stream) -> error code
PyObject *duct_backup(PyObject *, PyObject *const *a, Py_ssize_t n) {
    if (!ready(n, 5)) return nullptr;
    const int vl = whole(a[3]);
    void *stream = PyLong_AsVoidPtr(a[4]), *values, *new_child, *p[7];
    Shape s;
    static const int keys[7] = {CHILD, NODE_W, NODE_N, NODE_INFLIGHT, OUT_SELECTED, OUT_PATH, OUT_LEN};
    if (PyErr_Occurred() || !address(a[1], &values) || !address(a[2], &new_child) || !shape_of(a[0], NODE_PRIOR, 1, 3, &s) ||
        !addresses(a[0], keys, p))
        return nullptr;
    return launched([&] { return fn.duct_backup(vl, (int *)p[0], (float *)p[1], (int *)p[2], (int *)p[3], (int *)p[4], (int *)p[5], (int *)p[6],
                                          (float *)values, (int *)new_child, s.trees, s.nodes, s.edges, s.warps, s.depth, stream); });
}

// bind(addresses of the seven launchers, in the order of `fn`)
PyObject *bind(PyObject *, PyObject *const *a, Py_ssize_t n) {
    if (!count_is(n, 7)) return nullptr;
    void *p[7];
    for (int i = 0; i < 7; i++) {
        p[i] = PyLong_AsVoidPtr(a[i]);
        if (PyErr_Occurred()) return nullptr;
        if (!p[i]) {
            PyErr_Format(PyExc_ValueError, "bind: launcher %d has no address", i);
            return nullptr;
        }
    }
    fn.puct_select = (decltype(fn.puct_select))p[0];
    fn.puct_select_vl = (decltype(fn.puct_select_vl))p[1];
    fn.puct_backup = (decltype(fn.puct_backup))p[2];
    fn.puct_v2_select = (decltype(fn.puct_v2_select))p[3];
    fn.puct_v2_backup = (decltype(fn.puct_v2_backup))p[4];
    fn.duct_select = (decltype(fn.duct_select))p[5];
    fn.duct_backup = (decltype(fn.duct_backup))p[6];
    Py_RETURN_NONE;
}

#define METHOD(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {METHOD(bind), METHOD(puct_select), METHOD(puct_backup), METHOD(puct_v2_select), METHOD(puct_v2_backup),
                         METHOD(duct_select), METHOD(duct_backup), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_wave", "Launches of the tree selects and backups.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__wave(void) {
    for (int i = 0; i < N_KEYS; i++)
        if (!(key_objects[i] = PyUnicode_InternFromString(KEY_NAMES[i]))) return nullptr;
    str_data_ptr = PyUnicode_InternFromString("data_ptr");
    str_shape = PyUnicode_InternFromString("shape");
    str_interface = PyUnicode_InternFromString("__cuda_array_interface__");
    str_data = PyUnicode_InternFromString("data");
    if (!str_data_ptr || !str_shape || !str_interface || !str_data) return nullptr;
    return PyModule_Create(&module);
}
