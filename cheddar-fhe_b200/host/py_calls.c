/*
 * CPython entry points for the calls a program makes per operation: they take
 * the Python objects (torch tensors, index lists, constants) straight to the C
 * ABI of libcheddar_b200.so. A call on a small ciphertext runs on the GPU for
 * two microseconds, so what the interpreter spends on argument conversion is
 * what bounds it: ctypes took 4.6 us to wrap one index array and 0.8 us per
 * tensor list (2.7 GHz Xeon), the conversions below 0.2 and 0.2 per tensor.
 *
 * Every function returns the entry point's code; the caller raises. The
 * interpreter lock is released around the entry point.
 */
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include "../../include/cheddar_b200.h"

static PyObject *s_data_ptr, *s_dim, *s_size, *s_stride;
static PyObject *as_int32, *as_uint32; /* converters for arguments that are no ready-made 32-bit array */
static PyObject *zero;

/* ---- argument conversion: 0 on success, -1 with a Python error set ---- */
static int get_ptr(PyObject *t, void **out) {
  PyObject *v = PyObject_CallMethodNoArgs(t, s_data_ptr);
  if (!v) return -1;
  *out = PyLong_AsVoidPtr(v);
  Py_DECREF(v);
  return *out == NULL && PyErr_Occurred() ? -1 : 0;
}

/* an operand that an operation can do without: None is passed on as NULL */
static int get_optional(PyObject *t, void **out) {
  *out = NULL;
  return t == Py_None ? 0 : get_ptr(t, out);
}

#define SMALL_LIST 64
typedef struct {
  void *small[SMALL_LIST];
  void **p;
  Py_ssize_t n;
} ptr_list;

static void free_ptrs(ptr_list *l) {
  if (l->p != l->small) PyMem_Free(l->p);
}

static int get_ptrs(PyObject *seq, int (*get)(PyObject *, void **), ptr_list *l) {
  l->p = l->small;
  l->n = 0;
  PyObject *f = PySequence_Fast(seq, "a list of tensors is expected");
  if (!f) return -1;
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(f);
  if (n > SMALL_LIST && !(l->p = (void **)PyMem_Malloc(n * sizeof(void *)))) {
    l->p = l->small;
    Py_DECREF(f);
    PyErr_NoMemory();
    return -1;
  }
  for (Py_ssize_t i = 0; i < n; i++)
    if (get(PySequence_Fast_GET_ITEM(f, i), l->p + i)) {
      free_ptrs(l);
      l->p = l->small;
      Py_DECREF(f);
      return -1;
    }
  l->n = n;
  Py_DECREF(f);
  return 0;
}

/* operands of `count` destinations: a shorter list ends in NULLs */
static int get_operands(PyObject *seq, Py_ssize_t count, ptr_list *l) {
  if (get_ptrs(seq, get_optional, l)) return -1;
  if (l->n > count) {
    PyErr_SetString(PyExc_IndexError, "more operands than destinations");
    free_ptrs(l);
    return -1;
  }
  if (count > SMALL_LIST && l->n < count) {
    void **longer = (void **)PyMem_Malloc(count * sizeof(void *));
    if (!longer) {
      free_ptrs(l);
      PyErr_NoMemory();
      return -1;
    }
    for (Py_ssize_t i = 0; i < l->n; i++) longer[i] = l->p[i];
    free_ptrs(l);
    l->p = longer;
  }
  while (l->n < count) l->p[l->n++] = NULL;
  return 0;
}

/* 32-bit integers: a contiguous array of that type is used where it lies,
 * anything else goes through numpy. */
typedef struct {
  Py_buffer b;
  int held;
  void *p;
  int n;
} int_list;

static void free_ints(int_list *l) {
  if (l->held) PyBuffer_Release(&l->b);
  l->held = 0;
}

static int take_buffer(PyObject *o, char fmt, int_list *l) {
  if (PyObject_GetBuffer(o, &l->b, PyBUF_FORMAT | PyBUF_C_CONTIGUOUS)) {
    PyErr_Clear();
    return 0;
  }
  const char *f = l->b.format ? l->b.format : "B";
  if (*f == '<' || *f == '=' || *f == '@') f++;
  if (l->b.itemsize != 4 || f[1] || (*f != fmt && *f != (fmt == 'i' ? 'l' : 'L'))) {
    PyBuffer_Release(&l->b);
    return 0;
  }
  l->held = 1;
  l->p = l->b.buf;
  l->n = l->b.ndim ? (int)l->b.shape[0] : 1; /* the rows of a 2-D array, as len() counts */
  return 1;
}

static int get_ints(PyObject *o, char fmt, int_list *l) {
  l->held = 0;
  l->p = NULL;
  l->n = 0;
  if (take_buffer(o, fmt, l)) return 0;
  PyObject *a = PyObject_CallOneArg(fmt == 'i' ? as_int32 : as_uint32, o);
  if (!a) return -1;
  const int ok = take_buffer(a, fmt, l);
  Py_DECREF(a); /* the buffer keeps the array alive */
  if (!ok) {
    PyErr_SetString(PyExc_TypeError, "a list of integers is expected");
    return -1;
  }
  return 0;
}

/* constants that an operation can do without */
static int get_constants(PyObject *o, int_list *l) {
  if (o != Py_None) return get_ints(o, 'I', l);
  l->held = 0;
  l->p = NULL;
  l->n = 0;
  return 0;
}

/* an integer (no number with a fraction, even if it is 0) */
static int get_ll(PyObject *o, long long *out) {
  *out = PyLong_AsLongLong(o);
  return *out == -1 && PyErr_Occurred() ? -1 : 0;
}

/* what int() makes of it, modulo 2^64: flags, Galois elements, limb counts */
static int get_converted(PyObject *o, long long *out) {
  PyObject *i = PyNumber_Long(o);
  if (!i) return -1;
  *out = (long long)PyLong_AsUnsignedLongLongMask(i);
  Py_DECREF(i);
  return *out == -1 && PyErr_Occurred() ? -1 : 0;
}

/* number of polynomials and words between them of a [limbs, N] or [polys, limbs, N] tensor */
static int get_shape(PyObject *t, long long *polys, long long *stride) {
  long long dim;
  PyObject *v = PyObject_CallMethodNoArgs(t, s_dim);
  if (!v || get_ll(v, &dim)) {
    Py_XDECREF(v);
    return -1;
  }
  Py_DECREF(v);
  *polys = 1;
  *stride = 0;
  if (dim == 2) return 0;
  v = PyObject_CallMethodOneArg(t, s_size, zero);
  if (!v || get_ll(v, polys)) {
    Py_XDECREF(v);
    return -1;
  }
  Py_DECREF(v);
  if (dim != 3) return 0;
  v = PyObject_CallMethodOneArg(t, s_stride, zero);
  if (!v || get_ll(v, stride)) {
    Py_XDECREF(v);
    return -1;
  }
  Py_DECREF(v);
  return 0;
}

#define HANDLE(o) ((cfhe_context *)PyLong_AsVoidPtr(o))
#define NEED(count)                                                     \
  if (n != (count)) {                                                   \
    PyErr_SetString(PyExc_TypeError, "wrong number of arguments");      \
    return NULL;                                                        \
  }
#define ENTER(call)        \
  Py_BEGIN_ALLOW_THREADS;  \
  rc = (call);             \
  Py_END_ALLOW_THREADS
typedef uint32_t u32;

/* ---- transforms: (handle, dst, src, gidx, mont_conv) ---- */
static PyObject *py_ntt(PyObject *self, PyObject *const *a, Py_ssize_t n) {
  NEED(5)
  void *d, *s;
  long long polys, ss, dp, ds, mont;
  int_list g;
  int rc;
  if (get_ptr(a[1], &d) || get_ptr(a[2], &s) || get_shape(a[2], &polys, &ss) || get_shape(a[1], &dp, &ds) ||
      get_converted(a[4], &mont) || get_ints(a[3], 'i', &g))
    return NULL;
  ENTER(cfhe_ntt(HANDLE(a[0]), d, s, g.p, g.n, (int)polys, ds, ss, mont != 0));
  free_ints(&g);
  return PyLong_FromLong(rc);
}

/* (handle, dst, src, gidx, consts, mont_keep, centred) */
static PyObject *py_intt(PyObject *self, PyObject *const *a, Py_ssize_t n) {
  NEED(7)
  void *d, *s;
  long long polys, ss, dp, ds, keep, centred;
  int_list g, k;
  int rc;
  if (get_ptr(a[1], &d) || get_ptr(a[2], &s) || get_shape(a[2], &polys, &ss) || get_shape(a[1], &dp, &ds) ||
      get_converted(a[5], &keep) || get_converted(a[6], &centred) || get_ints(a[3], 'i', &g))
    return NULL;
  if (get_constants(a[4], &k)) {
    free_ints(&g);
    return NULL;
  }
  ENTER(cfhe_intt(HANDLE(a[0]), d, s, g.p, g.n, (int)polys, ds, ss, k.p, keep != 0, centred != 0));
  free_ints(&g);
  free_ints(&k);
  return PyLong_FromLong(rc);
}

/* ---- element-wise: (handle, op, dst, a, b, gidx) ---- */
static PyObject *py_binary(PyObject *self, PyObject *const *a, Py_ssize_t n) {
  NEED(6)
  void *d, *x, *y;
  long long op;
  int_list g;
  int rc;
  if (get_ll(a[1], &op) || get_ptr(a[2], &d) || get_ptr(a[3], &x) || get_optional(a[4], &y) || get_ints(a[5], 'i', &g))
    return NULL;
  ENTER(cfhe_binary(HANDLE(a[0]), (int)op, d, x, y, g.p, g.n));
  free_ints(&g);
  return PyLong_FromLong(rc);
}

/* (handle, op, dst, a, b, consts, gidx) */
static PyObject *py_const_op(PyObject *self, PyObject *const *a, Py_ssize_t n) {
  NEED(7)
  void *d, *x, *y;
  long long op;
  int_list g, k;
  int rc;
  if (get_ll(a[1], &op) || get_ptr(a[2], &d) || get_ptr(a[3], &x) || get_optional(a[4], &y) || get_ints(a[6], 'i', &g))
    return NULL;
  if (get_ints(a[5], 'I', &k)) {
    free_ints(&g);
    return NULL;
  }
  ENTER(cfhe_const_op(HANDLE(a[0]), (int)op, d, x, y, k.p, g.p, g.n));
  free_ints(&g);
  free_ints(&k);
  return PyLong_FromLong(rc);
}

/* (handle, with_const, op, dsts, a_list, b_list, consts, gidx) */
static PyObject *py_elementwise_multi(PyObject *self, PyObject *const *a, Py_ssize_t n) {
  NEED(8)
  long long wc, op;
  ptr_list d, x, y;
  int_list g, k;
  int rc;
  PyObject *ret = NULL;
  if (get_converted(a[1], &wc) || get_converted(a[2], &op) || get_ptrs(a[3], get_optional, &d)) return NULL;
  if (get_operands(a[4], d.n, &x)) goto free_d;
  if (a[5] == Py_None)
    y.p = NULL;
  else if (get_operands(a[5], d.n, &y))
    goto free_x;
  if (get_constants(a[6], &k)) goto free_y;
  if (get_ints(a[7], 'i', &g)) goto free_k;
  ENTER(cfhe_elementwise_multi(HANDLE(a[0]), wc != 0, (int)op, (int)d.n, (u32 *const *)d.p,
                               (const u32 *const *)x.p, (const u32 *const *)y.p, k.p, g.p, g.n));
  ret = PyLong_FromLong(rc);
  free_ints(&g);
free_k:
  free_ints(&k);
free_y:
  free_ptrs(&y);
free_x:
  free_ptrs(&x);
free_d:
  free_ptrs(&d);
  return ret;
}

/* (handle, d0, d1, d2, b1, a1, b2, a2, gidx) */
static PyObject *py_tensor(PyObject *self, PyObject *const *a, Py_ssize_t n) {
  NEED(9)
  void *p[7];
  int_list g;
  int rc;
  for (int i = 0; i < 7; i++)
    if (get_ptr(a[1 + i], p + i)) return NULL;
  if (get_ints(a[8], 'i', &g)) return NULL;
  ENTER(cfhe_tensor(HANDLE(a[0]), p[0], p[1], p[2], p[3], p[4], p[5], p[6], g.p, g.n));
  free_ints(&g);
  return PyLong_FromLong(rc);
}

/* (handle, dst, src, add, galois, gidx) */
static PyObject *py_permute(PyObject *self, PyObject *const *a, Py_ssize_t n) {
  NEED(6)
  void *d, *s, *add;
  long long galois;
  int_list g;
  int rc;
  if (get_ptr(a[1], &d) || get_ptr(a[2], &s) || get_optional(a[3], &add) || get_converted(a[4], &galois) ||
      get_ints(a[5], 'i', &g))
    return NULL;
  ENTER(cfhe_permute(HANDLE(a[0]), d, s, add, (u32)galois, g.p, g.n));
  free_ints(&g);
  return PyLong_FromLong(rc);
}

/* ---- mod-switch: (handle, level, kind, dst, src) ---- */
static PyObject *py_moddown(PyObject *self, PyObject *const *a, Py_ssize_t n) {
  NEED(5)
  void *d, *s;
  long long level, kind, polys, ss, dp, ds;
  int rc;
  if (get_ll(a[1], &level) || get_ll(a[2], &kind) || get_ptr(a[3], &d) || get_ptr(a[4], &s) ||
      get_shape(a[4], &polys, &ss) || get_shape(a[3], &dp, &ds))
    return NULL;
  ENTER(cfhe_moddown(HANDLE(a[0]), (int)level, (int)kind, d, s, (int)polys, ds, ss));
  return PyLong_FromLong(rc);
}

/* the two digit lists of a key; the library reads beta(level) entries of each */
#define KEYS(kb, ka)                                              \
  ptr_list kb##_l, ka##_l;                                        \
  const int beta = cfhe_beta(HANDLE(a[0]), (int)level);           \
  if (beta < 0) return PyLong_FromLong(beta);                     \
  if (get_ptrs(kb, get_ptr, &kb##_l)) return NULL;                \
  if (get_ptrs(ka, get_ptr, &ka##_l)) {                           \
    free_ptrs(&kb##_l);                                           \
    return NULL;                                                  \
  }                                                               \
  if (kb##_l.n < beta || ka##_l.n < beta) {                       \
    free_ptrs(&kb##_l);                                           \
    free_ptrs(&ka##_l);                                           \
    PyErr_SetString(PyExc_ValueError, "a key holds fewer digits than the level needs"); \
    return NULL;                                                  \
  }
#define FREE_KEYS(kb, ka) \
  free_ptrs(&kb##_l);     \
  free_ptrs(&ka##_l)
#define KEY_ARGS(kb, ka) (const u32 *const *)kb##_l.p, (const u32 *const *)ka##_l.p

/* (handle, level, out_b, out_a, d, bx, evk_b, evk_a, key_main) */
static PyObject *py_keyswitch(PyObject *self, PyObject *const *a, Py_ssize_t n) {
  NEED(9)
  void *p[4];
  long long level, key_main;
  int rc;
  for (int i = 0; i < 3; i++)
    if (get_ptr(a[2 + i], p + i)) return NULL;
  if (get_optional(a[5], p + 3) || get_ll(a[1], &level) || get_converted(a[8], &key_main)) return NULL;
  PyObject *kb = a[6], *ka = a[7];
  KEYS(kb, ka)
  ENTER(cfhe_keyswitch(HANDLE(a[0]), (int)level, p[0], p[1], p[2], p[3], KEY_ARGS(kb, ka), (int)key_main));
  FREE_KEYS(kb, ka);
  return PyLong_FromLong(rc);
}

/* (handle, level, out_b, out_a, b1, a1, b2, a2, evk_b, evk_a, key_main, rescale) */
static PyObject *py_hmult(PyObject *self, PyObject *const *a, Py_ssize_t n) {
  NEED(12)
  void *p[6];
  long long level, key_main, rescale;
  int rc;
  for (int i = 0; i < 6; i++)
    if (get_ptr(a[2 + i], p + i)) return NULL;
  if (get_ll(a[1], &level) || get_converted(a[10], &key_main) || get_converted(a[11], &rescale)) return NULL;
  PyObject *kb = a[8], *ka = a[9];
  KEYS(kb, ka)
  ENTER(cfhe_hmult(HANDLE(a[0]), (int)level, p[0], p[1], p[2], p[3], p[4], p[5], KEY_ARGS(kb, ka), (int)key_main,
                   rescale != 0));
  FREE_KEYS(kb, ka);
  return PyLong_FromLong(rc);
}

/* keys or plaintexts of a transform's steps: a list of lists of tensors, one flat
 * table, `digits` entries of each list. part >= 0: every key is a pair of lists,
 * take that one, and a key that is None has NULL entries. */
static int get_key_table(PyObject *keys, Py_ssize_t digits, int part, ptr_list *l) {
  l->p = l->small;
  l->n = 0;
  PyObject *f = PySequence_Fast(keys, "a list of keys is expected");
  if (!f) return -1;
  Py_ssize_t cap = SMALL_LIST;
  for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(f); i++) {
    PyObject *k = PySequence_Fast_GET_ITEM(f, i), *own = NULL, *d = NULL;
    const Py_ssize_t cnt = digits;
    if (k != Py_None || part < 0) {
      if (part >= 0) k = own = PySequence_GetItem(k, part);
      if (!k || !(d = PySequence_Fast(k, "a list of tensors is expected"))) goto fail;
      if (PySequence_Fast_GET_SIZE(d) < digits) {
        PyErr_SetString(PyExc_ValueError, "a key holds fewer digits than the level needs");
        goto fail;
      }
    }
    if (l->n + cnt > cap) {
      while (l->n + cnt > cap) cap *= 2;
      void **grown = (void **)PyMem_Malloc(cap * sizeof(void *));
      if (!grown) {
        PyErr_NoMemory();
        goto fail;
      }
      for (Py_ssize_t j = 0; j < l->n; j++) grown[j] = l->p[j];
      free_ptrs(l);
      l->p = grown;
    }
    for (Py_ssize_t j = 0; j < cnt; j++) {
      if (!d)
        l->p[l->n + j] = NULL;
      else if (get_optional(PySequence_Fast_GET_ITEM(d, j), l->p + l->n + j))
        goto fail;
    }
    l->n += cnt;
    Py_XDECREF(d);
    Py_XDECREF(own);
    continue;
  fail:
    Py_XDECREF(d);
    Py_XDECREF(own);
    free_ptrs(l);
    Py_DECREF(f);
    return -1;
  }
  Py_DECREF(f);
  return 0;
}

/* Keys of n_rot rotations, none of them None: a list per rotation, of which the
 * first `digits` tensors count, or all digits of all rotations in fewer lists.
 * The library reads n_rot * digits entries, so no fewer may come out. */
static int get_rotation_keys(PyObject *keys, Py_ssize_t n_rot, Py_ssize_t digits, ptr_list *l) {
  PyObject *f = PySequence_Fast(keys, "a list of keys is expected");
  if (!f) return -1;
  PyObject *all = PyList_New(0);
  int per_rotation = PySequence_Fast_GET_SIZE(f) >= n_rot, rc = all ? 0 : -1;
  for (Py_ssize_t i = 0; !rc && i < PySequence_Fast_GET_SIZE(f); i++) {
    PyObject *d = PySequence_Fast(PySequence_Fast_GET_ITEM(f, i), "a list of tensors is expected");
    if (!d) {
      rc = -1;
      break;
    }
    if (i < n_rot && PySequence_Fast_GET_SIZE(d) < digits) per_rotation = 0;
    rc = PyList_Append(all, d);
    Py_DECREF(d);
  }
  Py_DECREF(f);
  l->p = l->small;
  l->n = 0;
  const Py_ssize_t want = n_rot * digits;
  if (!rc && want > SMALL_LIST && !(l->p = (void **)PyMem_Malloc(want * sizeof(void *)))) {
    l->p = l->small;
    PyErr_NoMemory();
    rc = -1;
  }
  for (Py_ssize_t i = 0; !rc && i < PyList_GET_SIZE(all); i++) {
    PyObject *d = PyList_GET_ITEM(all, i);
    for (Py_ssize_t j = 0; !rc && j < PySequence_Fast_GET_SIZE(d); j++) {
      void *p;
      rc = get_ptr(PySequence_Fast_GET_ITEM(d, j), &p);
      if (!rc && l->n < want && (!per_rotation || j < digits)) l->p[l->n++] = p;
    }
  }
  if (!rc && l->n < want) {
    PyErr_SetString(PyExc_ValueError, "fewer keys or digits than the rotations need");
    rc = -1;
  }
  Py_XDECREF(all);
  if (rc) free_ptrs(l);
  return rc;
}

/* (handle, level, out, bx, ax, rots, evk_b, evk_a, key_main) */
static PyObject *py_hoisted_rotations(PyObject *self, PyObject *const *a, Py_ssize_t n) {
  NEED(9)
  void *p[3];
  long long level, key_main;
  int rc;
  for (int i = 0; i < 3; i++)
    if (get_ptr(a[2 + i], p + i)) return NULL;
  if (get_ll(a[1], &level) || get_converted(a[8], &key_main)) return NULL;
  const int beta = cfhe_beta(HANDLE(a[0]), (int)level);
  if (beta < 0) return PyLong_FromLong(beta);
  int_list r;
  ptr_list kb, ka;
  PyObject *ret = NULL;
  if (get_ints(a[5], 'i', &r)) return NULL;
  if (get_rotation_keys(a[6], r.n, beta, &kb)) goto free_r;
  if (get_rotation_keys(a[7], r.n, beta, &ka)) goto free_kb;
  ENTER(cfhe_hoisted_rotations(HANDLE(a[0]), (int)level, p[0], p[1], p[2], r.n, r.p, (const u32 *const *)kb.p,
                               (const u32 *const *)ka.p, (int)key_main));
  ret = PyLong_FromLong(rc);
  free_ptrs(&ka);
free_kb:
  free_ptrs(&kb);
free_r:
  free_ints(&r);
  return ret;
}

/* (handle, level, out_b, out_a, in_b, in_a, baby_rots, baby_keys, giant_rots, giant_keys, pts, key_main, rescale) */
static PyObject *py_linear_transform(PyObject *self, PyObject *const *a, Py_ssize_t n) {
  NEED(13)
  void *p[4];
  long long level, key_main, rescale;
  int rc;
  for (int i = 0; i < 4; i++)
    if (get_ptr(a[2 + i], p + i)) return NULL;
  if (get_ll(a[1], &level) || get_converted(a[11], &key_main) || get_converted(a[12], &rescale)) return NULL;
  const int beta = cfhe_beta(HANDLE(a[0]), (int)level);
  if (beta < 0) return PyLong_FromLong(beta);
  int_list br, gr;
  ptr_list t[5]; /* baby b, baby a, giant b, giant a, plaintexts */
  int got = 0;
  PyObject *ret = NULL;
  if (get_ints(a[6], 'i', &br)) return NULL;
  if (get_ints(a[8], 'i', &gr)) {
    free_ints(&br);
    return NULL;
  }
  for (; got < 4; got++)
    if (get_key_table(a[got < 2 ? 7 : 9], beta, got & 1, t + got)) goto done;
  if (get_key_table(a[10], br.n, -1, t + got)) goto done;
  got++;
  if (t[4].n < (Py_ssize_t)br.n * gr.n || t[0].n < (Py_ssize_t)br.n * beta || t[2].n < (Py_ssize_t)gr.n * beta) {
    PyErr_SetString(PyExc_ValueError, "fewer keys or plaintexts than baby and giant steps");
    goto done;
  }
  ENTER(cfhe_linear_transform(HANDLE(a[0]), (int)level, rescale != 0, p[0], p[1], p[2], p[3], br.n, br.p,
                              (const u32 *const *)t[0].p, (const u32 *const *)t[1].p, gr.n, gr.p,
                              (const u32 *const *)t[2].p, (const u32 *const *)t[3].p, (const u32 *const *)t[4].p,
                              (int)key_main));
  ret = PyLong_FromLong(rc);
done:
  while (got > 0) free_ptrs(t + --got);
  free_ints(&br);
  free_ints(&gr);
  return ret;
}

/* (handle, ys, xs, packed, gidx) */
static PyObject *py_ctpt_gemm(PyObject *self, PyObject *const *a, Py_ssize_t n) {
  NEED(5)
  ptr_list y, x;
  void *w;
  int_list g;
  int rc;
  PyObject *ret = NULL;
  if (get_ptr(a[3], &w) || get_ptrs(a[1], get_ptr, &y)) return NULL;
  if (get_ptrs(a[2], get_ptr, &x)) goto free_y;
  if (get_ints(a[4], 'i', &g)) goto free_x;
  ENTER(cfhe_ctpt_gemm(HANDLE(a[0]), (u32 *const *)y.p, (const u32 *const *)x.p, w, (int)x.n, (int)y.n, g.p, g.n));
  ret = PyLong_FromLong(rc);
  free_ints(&g);
free_x:
  free_ptrs(&x);
free_y:
  free_ptrs(&y);
  return ret;
}

/* ---- client side: (handle, dst, gidx, seed, stream) ---- */
static PyObject *py_sample_uniform(PyObject *self, PyObject *const *a, Py_ssize_t n) {
  NEED(5)
  void *d;
  int_list g;
  int rc;
  const unsigned long long seed = PyLong_AsUnsignedLongLongMask(a[3]);
  if (PyErr_Occurred()) return NULL;
  const unsigned long stream = PyLong_AsUnsignedLongMask(a[4]);
  if (PyErr_Occurred() || get_ptr(a[1], &d) || get_ints(a[2], 'i', &g)) return NULL;
  ENTER(cfhe_sample_uniform(HANDLE(a[0]), d, g.p, g.n, seed, (unsigned)stream));
  free_ints(&g);
  return PyLong_FromLong(rc);
}

/* (handle, dst, gidx, sigma, seed, stream) */
static PyObject *py_sample_error(PyObject *self, PyObject *const *a, Py_ssize_t n) {
  NEED(6)
  void *d;
  int_list g;
  int rc;
  const double sigma = PyFloat_AsDouble(a[3]);
  if (sigma == -1.0 && PyErr_Occurred()) return NULL;
  const unsigned long long seed = PyLong_AsUnsignedLongLongMask(a[4]);
  if (PyErr_Occurred()) return NULL;
  const unsigned long stream = PyLong_AsUnsignedLongMask(a[5]);
  if (PyErr_Occurred() || get_ptr(a[1], &d) || get_ints(a[2], 'i', &g)) return NULL;
  ENTER(cfhe_sample_error(HANDLE(a[0]), d, g.p, g.n, sigma, seed, (unsigned)stream));
  free_ints(&g);
  return PyLong_FromLong(rc);
}

/* (handle, b, a, s, e, m, gidx) */
static PyObject *py_encrypt(PyObject *self, PyObject *const *a, Py_ssize_t n) {
  NEED(7)
  void *p[5];
  int_list g;
  int rc;
  for (int i = 0; i < 4; i++)
    if (get_ptr(a[1 + i], p + i)) return NULL;
  if (get_optional(a[5], p + 4) || get_ints(a[6], 'i', &g)) return NULL;
  ENTER(cfhe_encrypt(HANDLE(a[0]), p[0], p[1], p[2], p[3], p[4], g.p, g.n));
  free_ints(&g);
  return PyLong_FromLong(rc);
}

/* (handle, dst, coeffs, gidx); coeffs: a contiguous array of N doubles */
static PyObject *py_encode_coeffs(PyObject *self, PyObject *const *a, Py_ssize_t n) {
  NEED(4)
  void *d;
  Py_buffer c;
  int_list g;
  int rc;
  if (get_ptr(a[1], &d) || PyObject_GetBuffer(a[2], &c, PyBUF_FORMAT | PyBUF_C_CONTIGUOUS)) return NULL;
  if (!c.format || c.format[0] != 'd' || c.len != (Py_ssize_t)cfhe_degree(HANDLE(a[0])) * 8) {
    PyBuffer_Release(&c);
    PyErr_SetString(PyExc_ValueError, "N doubles are expected");
    return NULL;
  }
  if (get_ints(a[3], 'i', &g)) {
    PyBuffer_Release(&c);
    return NULL;
  }
  ENTER(cfhe_encode_coeffs(HANDLE(a[0]), d, c.buf, g.p, g.n));
  PyBuffer_Release(&c);
  free_ints(&g);
  return PyLong_FromLong(rc);
}

/* (as_int32, as_uint32): converters to contiguous 32-bit arrays */
static PyObject *py_set_converters(PyObject *self, PyObject *const *a, Py_ssize_t n) {
  NEED(2)
  Py_XDECREF(as_int32);
  Py_XDECREF(as_uint32);
  as_int32 = Py_NewRef(a[0]);
  as_uint32 = Py_NewRef(a[1]);
  Py_RETURN_NONE;
}

#define M(name) {#name, (PyCFunction)(void (*)(void))py_##name, METH_FASTCALL, NULL}
static PyMethodDef methods[] = {M(ntt),           M(intt),      M(binary),        M(const_op),
                                M(elementwise_multi), M(tensor), M(permute),      M(moddown),
                                M(keyswitch),     M(hmult),     M(hoisted_rotations), M(linear_transform),
                                M(ctpt_gemm),     M(sample_uniform), M(sample_error), M(encrypt),
                                M(encode_coeffs),
                                M(set_converters), {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "cheddar_b200_calls", NULL, -1, methods,
                                    NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit_cheddar_b200_calls(void) {
  s_data_ptr = PyUnicode_InternFromString("data_ptr");
  s_dim = PyUnicode_InternFromString("dim");
  s_size = PyUnicode_InternFromString("size");
  s_stride = PyUnicode_InternFromString("stride");
  zero = PyLong_FromLong(0);
  if (!s_data_ptr || !s_dim || !s_size || !s_stride || !zero) return NULL;
  return PyModule_Create(&module);
}
