/* Python module _ftb200_step: a decode step from the caller's two dicts to the library in one native call.
 *
 * DynamicDecodeLayer.forward() (decode_layer.py) fills the library's argument block from some twenty dict entries and tensor
 * addresses; in Python that is 4.3 us of a step whose kernel takes 5 (one greedy row of 32000 columns).  This module does the same for
 * the common form of a call - the whole batch, on the stream the layer's memory was allocated on, logits of the type the slice
 * was made for - and answers None for every other one, which the Python code then serves.  Every address and scalar is
 * read from the caller's objects in every call; nothing of theirs is kept.  What is kept of the layer is a copy of the argument
 * block that its Python code filled, which nothing but this module reads or writes, and the constants of its set-up; the layer
 * drops the slice when it is set up again or allocates memory.  The criteria's block, whose counter all steps of a layer share, is
 * the layer's own, and the slice holds on to it. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <stdint.h>

#include "ftb200.h"

int ftb200_last_launch_count(void);

typedef struct {
    ftb200_sampling_params  params;      /* with the layer's own buffers filled in */
    ftb200_stop_params*     stop;        /* null until a call has needed one */
    PyObject *              stop_object, /* the ctypes structure that `stop` lies in */
                           *dtype, *current_stream, *device_index;
    unsigned long long      home; /* stream the layer's memory was allocated on */
    int                     type, batch, temp, pen, min_length; /* (type: FTB200_F32 .. FTB200_BF16, what dtype stands for) */
    long long               launches;
} Slice;

static const char kCapsule[] = "ftb200.slice";
static PyObject * s_logits, *s_step, *s_ite, *s_local, *s_max_input, *s_end_id, *s_input_lengths, *s_bias, *s_bad, *s_stop, *s_limit,
    *s_output_ids, *s_finished, *s_seq, *s_cum, *s_log_probs, *s_data_ptr, *s_dtype, *s_shape, *s_dim;

/* Entry of a dict, null where it is absent or None (borrowed). */
static PyObject* entry(PyObject* d, PyObject* key)
{
    PyObject* v = PyDict_GetItemWithError(d, key);
    return v == Py_None ? NULL : v;
}

static int call_integer(PyObject* o, PyObject* method, unsigned long long* out)
{
    PyObject* r = PyObject_VectorcallMethod(method, &o, 1 | PY_VECTORCALL_ARGUMENTS_OFFSET, NULL);
    if (r == NULL) {
        return 0;
    }
    *out = PyLong_AsUnsignedLongLong(r);
    Py_DECREF(r);
    return !(*out == (unsigned long long)-1 && PyErr_Occurred());
}

/* Address of an entry's data, null where the entry is absent; 0 on an error (set). */
static int address(PyObject* d, PyObject* key, void** out)
{
    PyObject*          t = entry(d, key);
    unsigned long long a = 0;
    if (t == NULL) {
        *out = NULL;
        return !PyErr_Occurred();
    }
    if (!call_integer(t, s_data_ptr, &a)) {
        return 0;
    }
    *out = (void*)(uintptr_t)a;
    return 1;
}

/* An int entry; `absent` where there is none.  0: not an int (the Python code converts it). */
static int integer(PyObject* d, PyObject* key, long absent, long* out)
{
    PyObject* v = entry(d, key);
    if (v == NULL) {
        *out = absent;
        return !PyErr_Occurred();
    }
    if (!PyLong_CheckExact(v)) {
        return 0;
    }
    *out = PyLong_AsLong(v);
    if (*out == -1 && PyErr_Occurred()) {
        PyErr_Clear();
        return 0;
    }
    return *out >= INT32_MIN && *out <= INT32_MAX;
}

/* Words of a list [2, L] (shared by the rows) or [rows, 2, L]: L, and whether it is shared. */
static int word_list(PyObject* t, int* len, int* shared)
{
    PyObject* shape = PyObject_GetAttr(t, s_shape);
    int       ok    = 0;
    if (shape == NULL) {
        return 0;
    }
    if (PyTuple_Check(shape) && (PyTuple_GET_SIZE(shape) == 2 || PyTuple_GET_SIZE(shape) == 3)) {
        const Py_ssize_t n = PyTuple_GET_SIZE(shape);
        *len               = (int)PyLong_AsLong(PyTuple_GET_ITEM(shape, n - 1));
        *shared            = n == 2 || PyLong_AsLong(PyTuple_GET_ITEM(shape, 0)) == 1;
        ok                 = !PyErr_Occurred();
    }
    Py_DECREF(shape);
    return ok;
}

/* True / False: the step is done (should_stop); an int: the library's status; None: not a call of the common form, nothing done. */
static PyObject* step(PyObject* self, PyObject* const* args, Py_ssize_t nargs)
{
    (void)self;
    if (nargs != 4) {
        PyErr_SetString(PyExc_TypeError, "step(slice, outputs, inputs, deadline_ms)");
        return NULL;
    }
    Slice* S = (Slice*)PyCapsule_GetPointer(args[0], kCapsule);
    if (S == NULL) {
        return NULL;
    }
    PyObject *out = args[1], *in = args[2];
    const int deadline = (int)PyLong_AsLong(args[3]);
    if (PyErr_Occurred()) {
        return NULL;
    }
    if (!PyDict_CheckExact(out) || !PyDict_CheckExact(in)) {
        Py_RETURN_NONE;
    }
    PyObject* logits = entry(in, s_logits);
    if (logits == NULL) {
        goto python;
    }
    {
        const Py_ssize_t rows  = PyObject_Size(logits);
        PyObject*        dtype = PyObject_GetAttr(logits, s_dtype);
        const int        same  = dtype == S->dtype && rows == S->batch;
        Py_XDECREF(dtype);
        unsigned long long dim = 0;
        if (!same || !call_integer(logits, s_dim, &dim) || dim != 2) {
            goto python;
        }
    }
    long pos, ite, local, mil;
    if (!integer(in, s_step, -1, &pos) || !integer(in, s_ite, 0, &ite) || !integer(in, s_local, S->batch, &local)
        || !integer(in, s_max_input, -1, &mil) || pos < 0 || mil < 0 || ite != 0 || local != S->batch) {
        goto python;
    }
    unsigned long long stream = 0;
    {
        PyObject* r = PyObject_CallOneArg(S->current_stream, S->device_index);
        if (r == NULL) {
            goto python;
        }
        stream = PyLong_AsUnsignedLongLong(r);
        Py_DECREF(r);
        if (PyErr_Occurred() || stream != S->home) {
            goto python;
        }
    }
    void *x, *end, *il, *bias, *bad, *stop, *limit, *ids, *fin, *seq, *cum, *lp;
    if (!address(in, s_logits, &x) || !address(in, s_end_id, &end) || !address(in, s_input_lengths, &il) || !address(in, s_bias, &bias)
        || !address(in, s_bad, &bad) || !address(in, s_stop, &stop) || !address(in, s_limit, &limit)
        || !address(out, s_output_ids, &ids) || !address(out, s_finished, &fin) || !address(out, s_seq, &seq)
        || !address(out, s_cum, &cum) || !address(out, s_log_probs, &lp)) {
        goto python;
    }
    /* (an empty tensor has no address: the Python code tells it from an absent one) */
    PyObject *bad_t = entry(in, s_bad), *stop_t = entry(in, s_stop), *limit_t = entry(in, s_limit);
    int       bad_len = 0, bad_shared = 0, stop_len = 0, unused;
    if (end == NULL || ids == NULL || fin == NULL || ((stop_t != NULL || limit_t != NULL) && S->stop == NULL)
        || (bad_t != NULL && (bad == NULL || !word_list(bad_t, &bad_len, &bad_shared)))
        || (stop_t != NULL && (stop == NULL || !word_list(stop_t, &stop_len, &unused))) || (limit_t != NULL && limit == NULL)) {
        goto python;
    }

    ftb200_sampling_params* P = &S->params;
    P->dtype                  = S->type;
    P->step                   = (int)pos;
    P->max_input_length       = (int)mil;
    P->logits                 = x;
    P->embedding_bias         = bias;
    P->end_ids                = (const int*)end;
    P->input_lengths          = (const int*)il;
    P->output_ids             = (int*)ids;
    P->bad_words              = (const int*)bad;
    P->bad_words_len          = bad_len;
    P->bad_words_shared       = bad_shared;
    /* host-side gating of the penalty kernels (BaseSamplingLayer.cc:302-349) */
    P->apply_temperature = bias != NULL || S->temp;
    P->apply_repetition  = pos > 1 && S->pen;
    P->apply_min_length  = S->min_length > pos - mil;
    P->sequence_length   = (int*)seq;
    P->finished          = (uint8_t*)fin;
    P->cum_log_probs     = (float*)cum;
    /* [request_output_len, batch] sliced at (step - max_input_length) (DynamicDecodeLayer.cc:427-435) */
    P->output_log_probs = lp == NULL ? NULL : (float*)lp + (pos - mil) * (long)S->batch;
    P->stream           = (void*)(uintptr_t)stream;
    int rc, should_stop = 0;
    if (stop_t == NULL && limit_t == NULL) {
        Py_BEGIN_ALLOW_THREADS;
        rc = ftb200_decode_step_sampling(P);
        Py_END_ALLOW_THREADS;
    }
    else {
        S->stop->stop_words            = (const int*)stop;
        S->stop->stop_words_len        = stop_len;
        S->stop->sequence_limit_length = (const uint32_t*)limit;
        Py_BEGIN_ALLOW_THREADS;
        rc = ftb200_decode_step(P, S->stop, deadline, &should_stop);
        Py_END_ALLOW_THREADS;
    }
    S->launches += ftb200_last_launch_count();
    if (rc != 0) {
        return PyLong_FromLong(rc);
    }
    return PyBool_FromLong(should_stop);
python:
    PyErr_Clear(); /* (the Python code meets the same object and says what is wrong with it) */
    Py_RETURN_NONE;
}

static void drop(PyObject* capsule)
{
    Slice* S = (Slice*)PyCapsule_GetPointer(capsule, kCapsule);
    if (S != NULL) {
        Py_XDECREF(S->stop_object);
        Py_XDECREF(S->dtype);
        Py_XDECREF(S->current_stream);
        Py_XDECREF(S->device_index);
        PyMem_Free(S);
    }
}

static PyObject* make(PyObject* self, PyObject* args)
{
    (void)self;
    unsigned long long params, stop, home;
    PyObject *         stop_object, *dtype, *current_stream, *device_index;
    int                type, batch, temp, pen, min_length;
    if (!PyArg_ParseTuple(args, "KKOOiOOKippi", &params, &stop, &stop_object, &dtype, &type, &current_stream, &device_index, &home,
                          &batch, &temp, &pen, &min_length)) {
        return NULL;
    }
    Slice* S = (Slice*)PyMem_Calloc(1, sizeof(Slice));
    if (S == NULL) {
        return PyErr_NoMemory();
    }
    S->params         = *(const ftb200_sampling_params*)(uintptr_t)params;
    S->stop           = (ftb200_stop_params*)(uintptr_t)stop;
    S->stop_object    = Py_NewRef(stop_object);
    S->dtype          = Py_NewRef(dtype);
    S->current_stream = Py_NewRef(current_stream);
    S->device_index   = Py_NewRef(device_index);
    S->home           = home;
    S->type = type, S->batch = batch, S->temp = temp, S->pen = pen, S->min_length = min_length;
    PyObject* c = PyCapsule_New(S, kCapsule, drop);
    if (c == NULL) {
        PyMem_Free(S);
    }
    return c;
}

static PyObject* launches(PyObject* self, PyObject* capsule)
{
    (void)self;
    Slice* S = (Slice*)PyCapsule_GetPointer(capsule, kCapsule);
    return S == NULL ? NULL : PyLong_FromLongLong(S->launches);
}

static PyMethodDef methods[] = {
    {"step", (PyCFunction)(void (*)(void))step, METH_FASTCALL, "step(slice, outputs, inputs, deadline_ms) -> bool | int | None"},
    {"make", make, METH_VARARGS,
     "make(params, stop, stop_object, dtype, type, current_stream, device_index, home, batch, temperature, penalty, min_length) -> "
     "slice; params and stop are addresses, params is copied"},
    {"launches", launches, METH_O, "kernels that a slice's steps have launched"},
    {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_ftb200_step", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__ftb200_step(void)
{
    const struct {
        PyObject**  at;
        const char* name;
    } names[] = {{&s_logits, "logits"}, {&s_step, "step"}, {&s_ite, "ite"}, {&s_local, "local_batch_size"},
                 {&s_max_input, "max_input_length"}, {&s_end_id, "end_id"}, {&s_input_lengths, "input_lengths"},
                 {&s_bias, "embedding_bias"}, {&s_bad, "bad_words_list"}, {&s_stop, "stop_words_list"},
                 {&s_limit, "sequence_limit_length"}, {&s_output_ids, "output_ids"}, {&s_finished, "finished"},
                 {&s_seq, "sequence_length"}, {&s_cum, "cum_log_probs"}, {&s_log_probs, "output_log_probs"},
                 {&s_data_ptr, "data_ptr"}, {&s_dtype, "dtype"}, {&s_shape, "shape"}, {&s_dim, "dim"}};
    for (size_t i = 0; i < sizeof(names) / sizeof(names[0]); ++i) {
        *names[i].at = PyUnicode_InternFromString(names[i].name);
        if (*names[i].at == NULL) {
            return NULL;
        }
    }
    return PyModule_Create(&module);
}
