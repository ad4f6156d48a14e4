// bsg_pycall.cpp -- the Python binding's per-call work in native code: the
// addresses of arrays and tensors, the segment table of a batch, a swaption
// book's structs, and the calls themselves.
//
// abi.py declares the whole ABI with ctypes; these are the calls whose
// arguments cost more there than the call: 4,096 book segments took 1.04 ms to
// copy into a ctypes array (the GPU prices such a pool in 0.19 ms), a served
// request 12 us, a small swaption book 45 us.  The functions are the library
// that abi.load() opened (bind() takes their addresses), and the GIL is
// released while one runs.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstdint>
#include <cstring>
#include <new>
#include <vector>

#include "bsg.h"

namespace {

decltype(&bsg_price_soa) f_price_soa;
decltype(&bsg_price_soa_f64) f_price_soa_f64;
decltype(&bsg_price_batch) f_price_batch;
decltype(&bsg_price_books_plain) f_books_plain;
decltype(&bsg_server_submit) f_submit;
decltype(&bsg_server_wait) f_wait;
decltype(&bsg_price_swaptions) f_swaptions;

PyObject* g_ndarray;          // numpy.ndarray
PyObject* g_ascontiguous;     // numpy.ascontiguousarray
PyObject* g_float64;          // numpy.float64
PyObject* g_name_data_ptr;    // interned attribute names
PyObject* g_sw_names[11];

// The address of a numpy array, a tensor-like with data_ptr(), an int or
// None; false with an exception set for anything else.
bool address(PyObject* x, uintptr_t* out) {
    if (x == Py_None) {
        *out = 0;
        return true;
    }
    if (PyLong_Check(x)) {
        *out = (uintptr_t)PyLong_AsUnsignedLongLongMask(x);
        return !PyErr_Occurred();
    }
    const int arr = PyObject_IsInstance(x, g_ndarray);
    if (arr < 0) return false;
    if (arr) {
        Py_buffer b;
        if (PyObject_GetBuffer(x, &b, PyBUF_STRIDES) == 0) {
            *out = (uintptr_t)b.buf;
            PyBuffer_Release(&b);
            return true;
        }
        PyErr_Clear();  // a type the buffer protocol has no format for
        PyObject* c = PyObject_GetAttrString(x, "ctypes");
        PyObject* d = c ? PyObject_GetAttrString(c, "data") : nullptr;
        Py_XDECREF(c);
        if (!d) return false;
        *out = (uintptr_t)PyLong_AsUnsignedLongLongMask(d);
        Py_DECREF(d);
        return !PyErr_Occurred();
    }
    PyObject* m = PyObject_GetAttr(x, g_name_data_ptr);
    if (!m) {
        if (!PyErr_ExceptionMatches(PyExc_AttributeError)) return false;
        PyErr_Clear();
        PyErr_Format(PyExc_TypeError, "cannot take the address of %R", (PyObject*)Py_TYPE(x));
        return false;
    }
    PyObject* v = PyObject_CallNoArgs(m);
    Py_DECREF(m);
    PyObject* i = v ? PyNumber_Long(v) : nullptr;
    Py_XDECREF(v);
    if (!i) return false;
    *out = (uintptr_t)PyLong_AsUnsignedLongLongMask(i);
    Py_DECREF(i);
    return !PyErr_Occurred();
}

// A C-contiguous array of type `fmt` and length >= n; its buffer stays held.
bool host_array(PyObject* x, char fmt, size_t n, Py_buffer* b) {
    const int arr = PyObject_IsInstance(x, g_ndarray);
    if (arr < 0) return false;
    if (arr && PyObject_GetBuffer(x, b, PyBUF_C_CONTIGUOUS | PyBUF_FORMAT) == 0) {
        const char* f = b->format;
        if (f && f[0] == '=') ++f;  // so where the array is not aligned; the calls copy it
        if (f && f[0] == fmt && f[1] == 0 && b->itemsize == 4 && b->ndim >= 1 && b->shape[0] >= 0 &&
            (size_t)b->shape[0] >= n)
            return true;
        PyBuffer_Release(b);
    }
    PyErr_Clear();
    PyErr_SetString(PyExc_TypeError,
                    "host arrays must be C-contiguous float32 (otype int32) of length >= n");
    return false;
}

// A whole number modulo 2^64, as ctypes takes one: an int or what has
// __index__ (numpy's integers); no float and no text.
bool whole(PyObject* x, uint64_t* out) {
#if PY_VERSION_HEX >= 0x030C0000
    if (PyLong_CheckExact(x) && PyUnstable_Long_IsCompact((PyLongObject*)x)) {
        *out = (uint64_t)PyUnstable_Long_CompactValue((PyLongObject*)x);
        return true;
    }
#endif
    *out = PyLong_AsUnsignedLongLongMask(x);  // through __index__
    return !PyErr_Occurred();
}

bool as_int(PyObject* x, uint64_t* out) {  // int(x), for a segment's two entries
    if (PyLong_Check(x)) return whole(x, out);
    PyObject* i = PyNumber_Long(x);
    const bool ok = i && whole(i, out);
    Py_XDECREF(i);
    return ok;
}

bool six_and_one(PyObject* const* a, uintptr_t* p) {  // six inputs and the prices
    for (int i = 0; i < 7; ++i)
        if (!address(a[i], &p[i])) return false;
    return true;
}

bool arg_count(Py_ssize_t got, Py_ssize_t want) {
    if (got == want) return true;
    PyErr_Format(PyExc_TypeError, "%zd arguments expected, got %zd", want, got);
    return false;
}

PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!arg_count(n, 7)) return nullptr;
    void* f[7];
    for (int i = 0; i < 7; ++i) {
        f[i] = PyLong_AsVoidPtr(a[i]);
        if (PyErr_Occurred()) return nullptr;
    }
    std::memcpy(&f_price_soa, &f[0], sizeof(void*));
    std::memcpy(&f_price_soa_f64, &f[1], sizeof(void*));
    std::memcpy(&f_price_batch, &f[2], sizeof(void*));
    std::memcpy(&f_books_plain, &f[3], sizeof(void*));
    std::memcpy(&f_submit, &f[4], sizeof(void*));
    std::memcpy(&f_wait, &f[5], sizeof(void*));
    std::memcpy(&f_swaptions, &f[6], sizeof(void*));
    Py_RETURN_NONE;
}

// price_soa(ctx, s, k, r, v, t, otype, prices, n, num_runs, flags, f64)
PyObject* price_soa(PyObject*, PyObject* const* a, Py_ssize_t na) {
    if (!arg_count(na, 12)) return nullptr;
    uintptr_t ctx, p[7];
    uint64_t n, runs, flags;
    if (!address(a[0], &ctx) || !whole(a[8], &n) || !whole(a[9], &runs) || !whole(a[10], &flags)) return nullptr;
    const bool f64 = a[11] == Py_True;
    Py_buffer held[7];
    int m = 0;
    if (!f64 && !(flags & BSG_DEVICE_PTRS)) {
        for (; m < 7; ++m) {
            if (!host_array(a[1 + m], m == 5 ? 'i' : 'f', n, &held[m])) {
                while (m > 0) PyBuffer_Release(&held[--m]);
                return nullptr;
            }
            p[m] = (uintptr_t)held[m].buf;
        }
    } else if (!six_and_one(a + 1, p)) {
        return nullptr;
    }
    int st;
    Py_BEGIN_ALLOW_THREADS
    if (f64)
        st = f_price_soa_f64((bsg_ctx*)ctx, (const double*)p[0], (const double*)p[1], (const double*)p[2],
                             (const double*)p[3], (const double*)p[4], (const int32_t*)p[5], (double*)p[6],
                             (size_t)n, (int)runs, (unsigned)flags);
    else
        st = f_price_soa((bsg_ctx*)ctx, (const float*)p[0], (const float*)p[1], (const float*)p[2],
                         (const float*)p[3], (const float*)p[4], (const int32_t*)p[5], (float*)p[6], (size_t)n,
                         (int)runs, (unsigned)flags);
    Py_END_ALLOW_THREADS
    while (m > 0) PyBuffer_Release(&held[--m]);
    return PyLong_FromLong(st);
}

template <typename T>
bool resized(std::vector<T>* v, Py_ssize_t n) {
    try {
        v->resize((size_t)n);
        return true;
    } catch (const std::bad_alloc&) {
        PyErr_NoMemory();
        return false;
    }
}

bool read_segments(PyObject* list, std::vector<bsg_segment>* out) {
    PyObject* seq = PySequence_Fast(list, "segments must be a sequence of (offset, length) pairs");
    if (!seq) return false;
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(seq);
    bool ok = resized(out, n);
    for (Py_ssize_t i = 0; i < n && ok; ++i) {
        PyObject* item = PySequence_Fast_GET_ITEM(seq, i);
        uint64_t o = 0, l = 0;
        if (PyTuple_CheckExact(item) && PyTuple_GET_SIZE(item) == 2 && PyLong_CheckExact(PyTuple_GET_ITEM(item, 0)) &&
            PyLong_CheckExact(PyTuple_GET_ITEM(item, 1))) {
            ok = whole(PyTuple_GET_ITEM(item, 0), &o) && whole(PyTuple_GET_ITEM(item, 1), &l);
        } else {
            // reading this one may run Python code, which may change the caller's
            // list or the pair: go on with tuples of what is in them now
            PyObject* now = PySequence_Tuple(seq);
            Py_DECREF(seq);
            seq = now;
            PyObject* pair = seq ? PySequence_Tuple(PyTuple_GET_ITEM(seq, i)) : nullptr;
            if (pair && PyTuple_GET_SIZE(pair) != 2) {
                PyErr_SetString(PyExc_ValueError, "a segment is an (offset, length) pair");
                ok = false;
            } else {
                ok = pair && as_int(PyTuple_GET_ITEM(pair, 0), &o) && as_int(PyTuple_GET_ITEM(pair, 1), &l);
            }
            Py_XDECREF(pair);
        }
        (*out)[(size_t)i] = bsg_segment{o, l};
    }
    Py_XDECREF(seq);
    return ok;
}

// price_batch(ctx, pool, prices, pool_len, segments, num_runs, flags, plain)
PyObject* price_batch(PyObject*, PyObject* const* a, Py_ssize_t na) {
    if (!arg_count(na, 8)) return nullptr;
    uintptr_t ctx, p[7];
    uint64_t pool_len, runs, flags;
    if (!address(a[0], &ctx) || !whole(a[3], &pool_len) || !whole(a[5], &runs) || !whole(a[6], &flags))
        return nullptr;
    PyObject* pool = PySequence_Tuple(a[1]);
    if (!pool) return nullptr;
    bool ok = PyTuple_GET_SIZE(pool) == 6;
    if (!ok) PyErr_SetString(PyExc_TypeError, "the pool is six arrays");
    for (int i = 0; i < 6 && ok; ++i) ok = address(PyTuple_GET_ITEM(pool, i), &p[i]);
    Py_DECREF(pool);
    std::vector<bsg_segment> segs;
    if (!ok || !address(a[2], &p[6]) || !read_segments(a[4], &segs)) return nullptr;
    bsg_segment none{0, 0};
    const bsg_segment* sp = segs.empty() ? &none : segs.data();
    const auto fn = a[7] == Py_True ? f_books_plain : f_price_batch;
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = fn((bsg_ctx*)ctx, (const float*)p[0], (const float*)p[1], (const float*)p[2], (const float*)p[3],
            (const float*)p[4], (const int32_t*)p[5], (float*)p[6], (size_t)pool_len, sp, segs.size(), (int)runs,
            (unsigned)flags);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(st);
}

// server_submit(server, s, k, r, v, t, otype, prices, n) -> (status, id)
PyObject* server_submit(PyObject*, PyObject* const* a, Py_ssize_t na) {
    if (!arg_count(na, 9)) return nullptr;
    uintptr_t srv, p[7];
    uint64_t n, id = 0;
    if (!address(a[0], &srv) || !six_and_one(a + 1, p) || !whole(a[8], &n)) return nullptr;
    const bsg_request req{(const float*)p[0], (const float*)p[1], (const float*)p[2], (const float*)p[3],
                          (const float*)p[4], (const int32_t*)p[5], (float*)p[6], (size_t)n};
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = f_submit((bsg_server*)srv, &req, &id);
    Py_END_ALLOW_THREADS
    return Py_BuildValue("iK", st, (unsigned long long)id);
}

// server_wait(server, id, timeout_s) -> (status, latency_s)
PyObject* server_wait(PyObject*, PyObject* const* a, Py_ssize_t na) {
    if (!arg_count(na, 3)) return nullptr;
    uintptr_t srv;
    uint64_t id;
    const double limit = PyFloat_AsDouble(a[2]);
    if ((limit == -1.0 && PyErr_Occurred()) || !address(a[0], &srv) || !whole(a[1], &id)) return nullptr;
    double lat = Py_NAN;
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = f_wait((bsg_server*)srv, id, limit, &lat);
    Py_END_ALLOW_THREADS
    return Py_BuildValue("id", st, lat);
}

// np.ascontiguousarray(x, dtype=np.float64), and its data
PyObject* doubles(PyObject* x, const double** data) {
    PyObject* y = PyObject_CallFunctionObjArgs(g_ascontiguous, x, g_float64, nullptr);
    Py_buffer b;
    if (!y || PyObject_GetBuffer(y, &b, PyBUF_C_CONTIGUOUS) != 0) {
        Py_XDECREF(y);
        return nullptr;
    }
    *data = (const double*)b.buf;
    PyBuffer_Release(&b);
    return y;
}

// price_swaptions(ctx, swaptions, trials, prices, errors): a tuple of swaptions,
// prices and errors of its length
PyObject* price_swaptions(PyObject*, PyObject* const* a, Py_ssize_t na) {
    if (!arg_count(na, 5)) return nullptr;
    uintptr_t ctx, price, err;
    uint64_t trials;
    if (!address(a[0], &ctx) || !whole(a[2], &trials) || !address(a[3], &price) || !address(a[4], &err))
        return nullptr;
    PyObject* const seq = a[1];
    if (!PyTuple_Check(seq)) {
        PyErr_SetString(PyExc_TypeError, "swaptions must be a tuple");
        return nullptr;
    }
    const Py_ssize_t n = PyTuple_GET_SIZE(seq);
    std::vector<bsg_swaption> sw;
    std::vector<PyObject*> keep;  // two arrays a swaption, NULL where not there yet
    bool ok = resized(&sw, n > 0 ? n : 1) && resized(&keep, 2 * n);
    for (Py_ssize_t i = 0; i < n && ok; ++i) {
        PyObject* w = PyTuple_GET_ITEM(seq, i);
        bsg_swaption* s = &sw[(size_t)i];
        double* const d[6] = {&s->strike, &s->compounding, &s->maturity, &s->tenor, &s->payment_interval, &s->years};
        for (int j = 0; j < 11 && ok; ++j) {
            PyObject* v = PyObject_GetAttr(w, g_sw_names[j]);
            if (!v) {
                ok = false;
            } else if (j < 6) {
                *d[j] = PyFloat_AsDouble(v);
                ok = !PyErr_Occurred();
            } else if (j < 8) {
                uint64_t x = 0;
                ok = whole(v, &x);
                (j == 6 ? s->n_steps : s->n_factors) = (int)x;
            } else if (j < 10) {
                keep[(size_t)(2 * i + j - 8)] = doubles(v, j == 8 ? &s->yield : &s->factors);
                ok = keep[(size_t)(2 * i + j - 8)] != nullptr;
            } else {
                ok = whole(v, &s->seed);
            }
            Py_XDECREF(v);
        }
    }
    int st = 0;
    if (ok) {
        Py_BEGIN_ALLOW_THREADS
        st = f_swaptions((bsg_ctx*)ctx, sw.data(), (size_t)n, trials, (double*)price, (double*)err);
        Py_END_ALLOW_THREADS
    }
    for (PyObject* y : keep) Py_XDECREF(y);
    return ok ? PyLong_FromLong(st) : nullptr;
}

#define FAST(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FAST(bind), FAST(price_soa), FAST(price_batch), FAST(server_submit),
                         FAST(server_wait), FAST(price_swaptions),
                         {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_pycall", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__pycall() {
    static const char* const names[11] = {"strike", "compounding", "maturity", "tenor", "payment_interval", "years",
                                          "n_steps", "n_factors", "yield_curve", "factors", "seed"};
    PyObject* np = PyImport_ImportModule("numpy");
    if (!np) return nullptr;
    g_ndarray = PyObject_GetAttrString(np, "ndarray");
    g_ascontiguous = PyObject_GetAttrString(np, "ascontiguousarray");
    g_float64 = PyObject_GetAttrString(np, "float64");
    Py_DECREF(np);
    g_name_data_ptr = PyUnicode_InternFromString("data_ptr");
    for (int i = 0; i < 11; ++i) g_sw_names[i] = PyUnicode_InternFromString(names[i]);
    if (!g_ndarray || !g_ascontiguous || !g_float64 || !g_name_data_ptr || PyErr_Occurred()) return nullptr;
    return PyModule_Create(&module);
}
