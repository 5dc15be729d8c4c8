/* Calls of the C ABI's per-token entries without ctypes: a launch of the smallest linears takes about 5 us on the
 * host, and converting a dozen arguments through ctypes 1.2 us of it; here it takes 0.2. One builtin per entry, in
 * the entry's own argument order: integers (addresses included) or None for a null pointer. The interpreter lock is
 * released around the call, as ctypes does. Returns the entry's return code. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <cuda_runtime_api.h>
#include "../../include/ampstein_b200.h"

static int get_p(PyObject* o, void** out)
{
    if (o == Py_None) { *out = NULL; return 1; }
    *out = PyLong_AsVoidPtr(o);
    return !(*out == NULL && PyErr_Occurred());
}

static int get_i(PyObject* o, int* out)
{
    const long v = PyLong_AsLong(o);
    if (v == -1 && PyErr_Occurred()) return 0;
    if (v < -2147483648L || v > 2147483647L) { PyErr_SetString(PyExc_OverflowError, "argument does not fit in an int"); return 0; }
    *out = (int) v;
    return 1;
}

static int get_l(PyObject* o, long* out)
{
    *out = PyLong_AsLong(o);
    return !(*out == -1 && PyErr_Occurred());
}

static int get_f(PyObject* o, float* out)
{
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) return 0;
    *out = (float) v;
    return 1;
}

static int count(const char* name, Py_ssize_t have, Py_ssize_t want)
{
    if (have == want) return 1;
    PyErr_Format(PyExc_TypeError, "%s takes %zd arguments, got %zd", name, want, have);
    return 0;
}

#define ENTRY(name) static PyObject* py_##name(PyObject* self, PyObject* const* a, Py_ssize_t n)
#define CALL(expr) do { int rc; Py_BEGIN_ALLOW_THREADS rc = (expr); Py_END_ALLOW_THREADS return PyLong_FromLong(rc); } while (0)

#define GEMM(name) \
ENTRY(name) \
{ \
    void *A, *B, *C, *suh, *had, *svh, *st; int v[6]; \
    if (!count(#name, n, 13) || !get_p(a[0], &A) || !get_p(a[1], &B) || !get_p(a[2], &C) || !get_p(a[3], &suh) || !get_p(a[4], &had) || \
        !get_p(a[5], &svh) || !get_p(a[12], &st)) return NULL; \
    for (int i = 0; i < 6; ++i) if (!get_i(a[6 + i], &v[i])) return NULL; \
    CALL(name(A, B, C, suh, had, svh, v[0], v[1], v[2], v[3], v[4], v[5], (cudaStream_t) st)); \
}
GEMM(amp_exl3_gemm)
GEMM(amp_exl3_gemm_bf16)

#define MGEMM(name) \
ENTRY(name) \
{ \
    void* p[6]; int v[7]; void *cp, *ns, *src, *st; int nsrc; \
    if (!count(#name, n, 18)) return NULL; \
    for (int i = 0; i < 6; ++i) if (!get_p(a[i], &p[i])) return NULL; \
    for (int i = 0; i < 7; ++i) if (!get_i(a[6 + i], &v[i])) return NULL; \
    if (!get_p(a[13], &cp) || !get_p(a[14], &ns) || !get_p(a[15], &src) || !get_i(a[16], &nsrc) || !get_p(a[17], &st)) return NULL; \
    CALL(name(p[0], p[1], p[2], p[3], p[4], p[5], v[0], v[1], v[2], v[3], v[4], v[5], v[6], cp, ns, src, nsrc, (cudaStream_t) st)); \
}
MGEMM(amp_exl3_mgemm)
MGEMM(amp_exl3_mgemm_bf16)

ENTRY(amp_exl3_moe_coop)
{
    void *args, *st;
    if (!count("amp_exl3_moe_coop", n, 2) || !get_p(a[0], &args) || !get_p(a[1], &st)) return NULL;
    CALL(amp_exl3_moe_coop((const amp_moe_coop_args*) args, (cudaStream_t) st));
}

ENTRY(amp_exl3_moe_sorted)
{
    void *args, *st;
    if (!count("amp_exl3_moe_sorted", n, 2) || !get_p(a[0], &args) || !get_p(a[1], &st)) return NULL;
    CALL(amp_exl3_moe_sorted((const amp_moe_sorted_args*) args, (cudaStream_t) st));
}

ENTRY(amp_b200_rms_norm_res)
{
    void *x, *res, *w, *y, *out, *st; long rows; int dim; float eps;
    if (!count("amp_b200_rms_norm_res", n, 9) || !get_p(a[0], &x) || !get_p(a[1], &res) || !get_p(a[2], &w) || !get_p(a[3], &y) ||
        !get_p(a[4], &out) || !get_l(a[5], &rows) || !get_i(a[6], &dim) || !get_f(a[7], &eps) || !get_p(a[8], &st)) return NULL;
    CALL(amp_b200_rms_norm_res(x, res, w, y, out, rows, dim, eps, (cudaStream_t) st));
}

ENTRY(amp_b200_silu_mul)
{
    void *g, *u, *out, *st; long cnt;
    if (!count("amp_b200_silu_mul", n, 5) || !get_p(a[0], &g) || !get_p(a[1], &u) || !get_p(a[2], &out) || !get_l(a[3], &cnt) || !get_p(a[4], &st)) return NULL;
    CALL(amp_b200_silu_mul(g, u, out, cnt, (cudaStream_t) st));
}

#define M(name) { #name, (PyCFunction) (void (*)(void)) py_##name, METH_FASTCALL, NULL }
static PyMethodDef methods[] = { M(amp_exl3_gemm), M(amp_exl3_gemm_bf16), M(amp_exl3_mgemm), M(amp_exl3_mgemm_bf16), M(amp_exl3_moe_coop),
                                 M(amp_exl3_moe_sorted), M(amp_b200_rms_norm_res), M(amp_b200_silu_mul), { NULL, NULL, 0, NULL } };
static struct PyModuleDef module = { PyModuleDef_HEAD_INIT, "_fast", NULL, -1, methods, NULL, NULL, NULL, NULL };
PyMODINIT_FUNC PyInit__fast(void) { return PyModule_Create(&module); }
