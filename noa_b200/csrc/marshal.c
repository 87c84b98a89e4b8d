/* The Python API's argument marshalling (noa_b200/fourier_project.py), natively: one call takes the tensors,
 * shapes, transforms and options of a central-slice call as Python objects, fills the C ABI's structures on
 * the stack and calls the entry point without the interpreter lock. Built through ctypes structures, the
 * same took longer than a small call runs on the GPU (an extraction of 64
 * slices of 64^2 from a 64^3 volume: 17.4 us a call, now 6.7 us; rasterizing them 23.3 us, now 18.5 us).
 *
 * What the fast path does not know (inline transforms, matrices to pack) goes through the Python helper
 * that the ctypes path uses, so that both accept and refuse the same arguments. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>
#include <string.h>

#include "noa_b200/fourier_project.h"

static PyObject *g_error, *g_dtypes, *g_interps, *g_transform_helper, *g_ews_helper, *g_float32, *g_tensor; /* from init() */
static PyObject *s_data_ptr, *s_dtype, *s_shape, *s_stride, *s_is_contiguous, *s_fftfreq_sinc, *s_fftfreq_blackman;

static int fail(long code, const char* message) {
    PyObject* e = PyObject_CallFunction(g_error, "ls", code, message);
    if (e) {
        PyErr_SetObject(g_error, e);
        Py_DECREF(e);
    }
    return -1;
}

/* int(x), its low 64 bits as ctypes' integers take it, and float(x). */
static int to_int64(PyObject* x, int64_t* out) {
    if (PyLong_CheckExact(x)) {
        *out = (int64_t) PyLong_AsUnsignedLongLongMask(x);
    } else {
        PyObject* n = PyNumber_Long(x);
        if (!n)
            return -1;
        *out = (int64_t) PyLong_AsUnsignedLongLongMask(n);
        Py_DECREF(n);
    }
    return *out == -1 && PyErr_Occurred() ? -1 : 0;
}

static int to_double(PyObject* x, double* out) {
    if (PyFloat_CheckExact(x)) {
        *out = PyFloat_AS_DOUBLE(x);
        return 0;
    }
    PyObject* f = PyNumber_Float(x);
    if (!f)
        return -1;
    *out = PyFloat_AS_DOUBLE(f);
    Py_DECREF(f);
    return 0;
}

/* `count` integers of a sequence. EXACT: of that length; SHAPE: a shorter one is padded with zeros, which the
 * library refuses; HEAD: the first of a longer one. */
enum Length { EXACT, SHAPE, HEAD };
static int to_int64s(PyObject* seq, int64_t* out, Py_ssize_t count, enum Length length) {
    PyObject* t = PySequence_Fast(seq, "a sequence of integers is expected");
    if (!t)
        return -1;
    int st = 0;
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(t);
    if (n > count ? length != HEAD : n < count ? length != SHAPE : 0) {
        PyErr_Format(PyExc_IndexError, "%zd integers are expected, got %zd", count, n);
        st = -1;
    }
    for (Py_ssize_t i = 0; st == 0 && i < count; ++i) {
        out[i] = 0;
        if (i < n)
            st = to_int64(PySequence_Fast_GET_ITEM(t, i), &out[i]);
    }
    Py_DECREF(t);
    return st;
}

/* Four integers of anything that is read by index: a tuple or a list (the first of a longer one), else by its
 * own subscripts. */
static int to_target_shape(PyObject* x, int64_t out[4]) {
    if (PyTuple_Check(x) || PyList_CheckExact(x))
        return to_int64s(x, out, 4, HEAD);
    for (long i = 0; i < 4; ++i) {
        PyObject* key = PyLong_FromLong(i);
        PyObject* v = key ? PyObject_GetItem(x, key) : NULL;
        Py_XDECREF(key);
        if (!v)
            return -1;
        const int st = to_int64(v, &out[i]);
        Py_DECREF(v);
        if (st != 0)
            return -1;
    }
    return 0;
}

/* A tensor, a number (constant input) or None. 1: present, 0: None, -1: error. */
static int to_array(PyObject* t, nb_array* a) {
    memset(a, 0, sizeof(*a));
    if (t == Py_None)
        return 0;
    if (PyFloat_Check(t) || PyLong_Check(t) || PyComplex_Check(t)) {
        a->is_value = 1;
        a->dtype = PyComplex_Check(t) ? NB_DTYPE_C32 : NB_DTYPE_F32;
        const Py_complex v = PyComplex_AsCComplex(t);
        if (v.real == -1.0 && PyErr_Occurred())
            return -1;
        a->value[0] = v.real;
        a->value[1] = v.imag;
        return 1;
    }
    PyObject* shape = PyObject_GetAttr(t, s_shape);
    if (!shape)
        return -1;
    if (PyObject_Size(shape) != 4) {
        PyObject* text = PyErr_Occurred() ? NULL : PyUnicode_FromFormat("expected a 4-D (BDHW) tensor, got shape %S", shape);
        if (text) {
            fail(NB_ERROR_INVALID, PyUnicode_AsUTF8(text));
            Py_DECREF(text);
        }
        Py_DECREF(shape);
        return -1;
    }
    int st = to_int64s(shape, a->shape, 4, EXACT);
    Py_DECREF(shape);
    if (st != 0)
        return -1;
    PyObject* ptr = PyObject_CallMethodNoArgs(t, s_data_ptr);
    if (!ptr)
        return -1;
    a->data = PyLong_AsVoidPtr(ptr);
    Py_DECREF(ptr);
    if (!a->data && PyErr_Occurred())
        return -1;
    PyObject* dtype = PyObject_GetAttr(t, s_dtype);
    if (!dtype)
        return -1;
    PyObject* code = PyDict_GetItemWithError(g_dtypes, dtype);
    if (!code) {
        if (!PyErr_Occurred())
            PyErr_SetObject(PyExc_KeyError, dtype);
        Py_DECREF(dtype);
        return -1;
    }
    a->dtype = (int32_t) PyLong_AsLong(code);
    Py_DECREF(dtype);
    PyObject* stride = PyObject_CallMethodNoArgs(t, s_stride);
    if (!stride)
        return -1;
    st = to_int64s(stride, a->strides, 4, EXACT);
    Py_DECREF(stride);
    return st == 0 ? 1 : -1;
}

/* A contiguous (n, 12) or (n, 4) float32 tensor; everything else through the helper, which may make tensors
 * that live in `keep`. */
static int to_transform(PyObject* x, int rotation, PyObject* keep, nb_transform* t) {
    memset(t, 0, sizeof(*t));
    if (x == Py_None && !rotation)
        return 0; /* NB_XFORM_NONE */
    if (Py_TYPE(x) == (PyTypeObject*) g_tensor) {
        PyObject* dtype = PyObject_GetAttr(x, s_dtype);
        PyObject* shape = dtype ? PyObject_GetAttr(x, s_shape) : NULL;
        PyObject* whole = shape ? PyObject_CallMethodNoArgs(x, s_is_contiguous) : NULL;
        int64_t n[2] = {0, 0};
        int st = whole ? 0 : -1, plain = 0;
        if (st == 0 && dtype == g_float32 && whole == Py_True && PyObject_Size(shape) == 2) {
            st = to_int64s(shape, n, 2, EXACT);
            plain = st == 0 && (n[1] == 12 || n[1] == 4);
        }
        Py_XDECREF(dtype);
        Py_XDECREF(shape);
        Py_XDECREF(whole);
        if (st != 0)
            return -1;
        if (plain) {
            PyObject* ptr = PyObject_CallMethodNoArgs(x, s_data_ptr);
            if (!ptr)
                return -1;
            t->data = PyLong_AsVoidPtr(ptr);
            Py_DECREF(ptr);
            t->kind = n[1] == 12 ? NB_XFORM_MAT33_F32 : NB_XFORM_QUAT_F32;
            t->count = n[0];
            return !t->data && PyErr_Occurred() ? -1 : 0;
        }
    }
    PyObject* made = PyObject_CallFunctionObjArgs(g_transform_helper, x, rotation ? Py_True : Py_False, keep, NULL);
    if (!made)
        return -1;
    Py_buffer view;
    int st = PyObject_GetBuffer(made, &view, PyBUF_SIMPLE);
    if (st == 0) {
        if (view.len == (Py_ssize_t) sizeof(*t))
            memcpy(t, view.buf, sizeof(*t));
        else
            st = fail(NB_ERROR_INVALID, "unexpected transform structure");
        PyBuffer_Release(&view);
    }
    Py_DECREF(made);
    return st;
}

static int to_window(PyObject* w, double* sinc, double* blackman) {
    *sinc = *blackman = -1.0;
    const int given = w == Py_None ? 0 : PyObject_IsTrue(w);
    if (given <= 0)
        return given;
    PyObject* v = PyObject_GetAttr(w, s_fftfreq_sinc);
    if (!v)
        return -1;
    int st = to_double(v, sinc);
    Py_DECREF(v);
    if (st != 0 || !(v = PyObject_GetAttr(w, s_fftfreq_blackman)))
        return -1;
    st = to_double(v, blackman);
    Py_DECREF(v);
    return st;
}

/* One number, or a pair of them as a tuple; anything else (an array, a tensor) through the helper. */
static int to_ews_radius(PyObject* ews, double out[2]) {
    if (PyFloat_CheckExact(ews) || PyLong_CheckExact(ews)) {
        const int st = to_double(ews, &out[0]);
        out[1] = out[0];
        return st;
    }
    PyObject* pair;
    if (PyTuple_CheckExact(ews)) {
        pair = Py_NewRef(ews);
    } else {
        pair = PyObject_CallOneArg(g_ews_helper, ews);
        if (!pair)
            return -1;
    }
    int st = PyTuple_Check(pair) && PyTuple_GET_SIZE(pair) >= 2 ? 0 : -1;
    if (st != 0)
        PyErr_SetString(PyExc_IndexError, "ews_radius: two numbers are expected");
    for (int i = 0; st == 0 && i < 2; ++i)
        st = to_double(PyTuple_GET_ITEM(pair, i), &out[i]);
    Py_DECREF(pair);
    return st;
}

/* (interp, fftfreq_cutoff, target_shape, ews_radius, windowed_sinc, w_windowed_sinc, add_to_output,
 * correct_weights) */
static int to_options(PyObject* o, nb_options* out) {
    memset(out, 0, sizeof(*out));
    if (!PyTuple_Check(o) || PyTuple_GET_SIZE(o) != 8) {
        PyErr_SetString(PyExc_TypeError, "options: a tuple of 8 values");
        return -1;
    }
    PyObject* interp = PyTuple_GET_ITEM(o, 0);
    if (PyUnicode_Check(interp)) {
        PyObject* code = PyDict_GetItemWithError(g_interps, interp);
        if (!code) {
            if (!PyErr_Occurred())
                PyErr_SetObject(PyExc_KeyError, interp);
            return -1;
        }
        interp = code;
    }
    int64_t method;
    if (to_int64(interp, &method) != 0)
        return -1;
    out->interp = (int32_t) method;
    if (to_double(PyTuple_GET_ITEM(o, 1), &out->fftfreq_cutoff) != 0)
        return -1;
    PyObject* target = PyTuple_GET_ITEM(o, 2);
    if (target != Py_None && to_target_shape(target, out->target_shape) != 0)
        return -1;
    if (to_ews_radius(PyTuple_GET_ITEM(o, 3), out->ews_radius) != 0)
        return -1;
    if (to_window(PyTuple_GET_ITEM(o, 4), &out->fftfreq_sinc, &out->fftfreq_blackman) != 0 ||
        to_window(PyTuple_GET_ITEM(o, 5), &out->w_fftfreq_sinc, &out->w_fftfreq_blackman) != 0)
        return -1;
    const int add = PyObject_IsTrue(PyTuple_GET_ITEM(o, 6)), correct = PyObject_IsTrue(PyTuple_GET_ITEM(o, 7));
    if (add < 0 || correct < 0)
        return -1;
    out->add_to_output = add;
    out->correct_weights = correct;
    return 0;
}

typedef int (*entry2)(int32_t, const nb_array*, const nb_array*, const int64_t*, const nb_array*, const nb_array*,
                      const int64_t*, const nb_transform*, const nb_transform*, const nb_options*, void*);
typedef int (*entry4)(int32_t, const nb_array*, const nb_array*, const int64_t*, const nb_array*, const nb_array*,
                      const int64_t*, const nb_transform*, const nb_transform*, const nb_transform*,
                      const nb_transform*, const nb_options*, void*);

/* call(entry, remap, input, input_weight, input_shape, output, output_weight, output_shape, options, stream,
 *      scaling, rotation[, scaling, rotation]) -> status */
static PyObject* call(PyObject* self, PyObject* const* args, Py_ssize_t n) {
    (void) self;
    if (n != 12 && n != 14) {
        PyErr_SetString(PyExc_TypeError, "call: 12 or 14 arguments");
        return NULL;
    }
    void* entry = PyLong_AsVoidPtr(args[0]);
    const long remap = PyLong_AsLong(args[1]);
    if (PyErr_Occurred())
        return NULL;
    nb_array arrays[4];
    const nb_array* present[4];
    int64_t shapes[2][4];
    static const int at[4] = {2, 3, 5, 6};
    for (int i = 0; i < 4; ++i) {
        const int st = to_array(args[at[i]], &arrays[i]);
        if (st < 0)
            return NULL;
        present[i] = st ? &arrays[i] : NULL;
    }
    if (to_int64s(args[4], shapes[0], 4, SHAPE) != 0 || to_int64s(args[7], shapes[1], 4, SHAPE) != 0)
        return NULL;
    nb_options options;
    if (to_options(args[8], &options) != 0)
        return NULL;
    int64_t stream = 0;
    if (args[9] != Py_None && !PyLong_Check(args[9])) {
        PyErr_SetString(PyExc_TypeError, "stream: an integer handle is expected");
        return NULL;
    }
    if (args[9] != Py_None && to_int64(args[9], &stream) != 0)
        return NULL;
    PyObject* keep = PyList_New(0);
    if (!keep)
        return NULL;
    nb_transform xf[4];
    for (int i = 0; i < (int) n - 10; ++i) {
        if (to_transform(args[10 + i], i & 1, keep, &xf[i]) != 0) {
            Py_DECREF(keep);
            return NULL;
        }
    }
    int code;
    Py_BEGIN_ALLOW_THREADS
    if (n == 12)
        code = ((entry2) entry)((int32_t) remap, present[0], present[1], shapes[0], present[2], present[3], shapes[1],
                                &xf[0], &xf[1], &options, (void*) (uintptr_t) stream);
    else
        code = ((entry4) entry)((int32_t) remap, present[0], present[1], shapes[0], present[2], present[3], shapes[1],
                                &xf[0], &xf[1], &xf[2], &xf[3], &options, (void*) (uintptr_t) stream);
    Py_END_ALLOW_THREADS
    Py_DECREF(keep);
    return PyLong_FromLong(code);
}

/* init(error class, {dtype: code}, {interp: code}, transform helper, ews_radius helper, torch.float32,
 *      torch.Tensor) */
static PyObject* init(PyObject* self, PyObject* args) {
    (void) self;
    PyObject *error, *dtypes, *interps, *helper, *ews, *float32, *tensor;
    if (!PyArg_ParseTuple(args, "OO!O!OOOO", &error, &PyDict_Type, &dtypes, &PyDict_Type, &interps, &helper, &ews,
                          &float32, &tensor))
        return NULL;
    PyObject** to[7] = {&g_error, &g_dtypes, &g_interps, &g_transform_helper, &g_ews_helper, &g_float32, &g_tensor};
    PyObject* from[7] = {error, dtypes, interps, helper, ews, float32, tensor};
    for (int i = 0; i < 7; ++i) {
        Py_INCREF(from[i]);
        Py_XSETREF(*to[i], from[i]);
    }
    Py_RETURN_NONE;
}

static PyMethodDef methods[] = {{"call", (PyCFunction) (void (*)(void)) call, METH_FASTCALL, NULL},
                                {"init", init, METH_VARARGS, NULL},
                                {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_marshal", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__marshal(void) {
    s_data_ptr = PyUnicode_InternFromString("data_ptr");
    s_dtype = PyUnicode_InternFromString("dtype");
    s_shape = PyUnicode_InternFromString("shape");
    s_stride = PyUnicode_InternFromString("stride");
    s_is_contiguous = PyUnicode_InternFromString("is_contiguous");
    s_fftfreq_sinc = PyUnicode_InternFromString("fftfreq_sinc");
    s_fftfreq_blackman = PyUnicode_InternFromString("fftfreq_blackman");
    return PyModule_Create(&module);
}
