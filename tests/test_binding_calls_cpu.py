"""Argument handling of the Python binding's calls (host/py_calls.c), without a
GPU: the module is compiled against a stand-in for the library that records what
an entry point is given. What the binding cannot pass on safely has to be an
exception, with the entry point not called."""
import ctypes as C
import importlib.util
import os
import subprocess
import sysconfig

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BETA = 2  # digits a key holds at the stand-in's only level

STAND_IN = r"""
#include <string.h>
#include "cheddar_b200.h"
#define T const uint32_t *const *
CFHE_API int calls = 0, n_ints = 0, ints[64], polys = 0;
CFHE_API const void *table[5][128];
CFHE_API long long strides[2];
static int rec(const int *g, int n) {
  n_ints = n;
  for (int i = 0; i < n && i < 64; i++) ints[i] = g[i];
  calls++;
  return 0;
}
static void keep(int t, const void *p, int n) { if (p && n > 0) memcpy(table[t], p, n * sizeof(void *)); }
int cfhe_beta(const cfhe_context *h, int level) { return level == 1 ? 2 : -1; }
int cfhe_degree(const cfhe_context *h) { return 65536; }
int cfhe_ntt(cfhe_context *h, uint32_t *d, const uint32_t *s, const int *g, int n, int np, long long ds, long long ss,
             int m) { polys = np; strides[0] = ds; strides[1] = ss; return rec(g, n); }
int cfhe_intt(cfhe_context *h, uint32_t *d, const uint32_t *s, const int *g, int n, int np, long long ds, long long ss,
              const uint32_t *k, int mk, int ce) { return rec(g, n); }
int cfhe_binary(cfhe_context *h, int op, uint32_t *d, const uint32_t *a, const uint32_t *b, const int *g, int n) {
  return rec(g, n); }
int cfhe_const_op(cfhe_context *h, int op, uint32_t *d, const uint32_t *a, const uint32_t *b, const uint32_t *k,
                  const int *g, int n) { return rec((const int *)k, n); }
int cfhe_elementwise_multi(cfhe_context *h, int wc, int op, int np, uint32_t *const *d, T a, T b, const uint32_t *k,
                           const int *g, int n) {
  polys = np; keep(0, d, np); keep(1, a, np); memset(table[2], 0, sizeof(table[2])); keep(2, b, np); return rec(g, n); }
int cfhe_tensor(cfhe_context *h, uint32_t *a, uint32_t *b, uint32_t *c, const uint32_t *d, const uint32_t *e,
                const uint32_t *f, const uint32_t *i, const int *g, int n) { return rec(g, n); }
int cfhe_permute(cfhe_context *h, uint32_t *d, const uint32_t *s, const uint32_t *a, uint32_t ge, const int *g, int n) {
  return rec((const int *)&ge, 1); }
int cfhe_moddown(cfhe_context *h, int l, int k, uint32_t *d, const uint32_t *s, int np, long long ds, long long ss) {
  return rec(&l, 1); }
int cfhe_keyswitch(cfhe_context *h, int l, uint32_t *ob, uint32_t *oa, const uint32_t *d, const uint32_t *bx, T kb, T ka,
                   int km) { keep(0, kb, 2); keep(1, ka, 2); return rec(&l, 1); }
int cfhe_hmult(cfhe_context *h, int l, uint32_t *ob, uint32_t *oa, const uint32_t *b1, const uint32_t *a1,
               const uint32_t *b2, const uint32_t *a2, T kb, T ka, int km, int r) {
  keep(0, kb, 2); keep(1, ka, 2); return rec(&l, 1); }
int cfhe_hoisted_rotations(cfhe_context *h, int l, uint32_t *o, const uint32_t *bx, const uint32_t *ax, int nr,
                           const int *r, T kb, T ka, int km) { keep(0, kb, 2 * nr); keep(1, ka, 2 * nr); return rec(r, nr); }
int cfhe_linear_transform(cfhe_context *h, int l, int re, uint32_t *ob, uint32_t *oa, const uint32_t *ib,
                          const uint32_t *ia, int nb, const int *br, T bkb, T bka, int ng, const int *gr, T gkb, T gka,
                          T pt, int km) {
  keep(0, bkb, 2 * nb); keep(1, bka, 2 * nb); keep(2, gkb, 2 * ng); keep(3, gka, 2 * ng); keep(4, pt, nb * ng);
  return rec(br, nb); }
int cfhe_ctpt_gemm(cfhe_context *h, uint32_t *const *y, T x, const void *w, int ni, int no, const int *g, int n) {
  keep(0, y, no); keep(1, x, ni); return rec(g, n); }
int cfhe_sample_uniform(cfhe_context *h, uint32_t *d, const int *g, int n, unsigned long long s, unsigned st) {
  strides[0] = (long long)s; strides[1] = st; return rec(g, n); }
int cfhe_sample_error(cfhe_context *h, uint32_t *d, const int *g, int n, double si, unsigned long long s, unsigned st) {
  return rec(g, n); }
int cfhe_encrypt(cfhe_context *h, uint32_t *b, const uint32_t *a, const uint32_t *s, const uint32_t *e,
                 const uint32_t *m, const int *g, int n) { return rec(g, n); }
int cfhe_encode_coeffs(cfhe_context *h, uint32_t *d, const double *c, const int *g, int n) { return rec(g, n); }
"""


class Tensor:
    """What the binding asks of a device tensor."""

    def __init__(self, addr, shape=(1, 65536), stride0=0):
        self.addr, self.shape, self.stride0 = addr, shape, stride0

    def data_ptr(self):
        return self.addr

    def dim(self):
        return len(self.shape)

    def size(self, i):
        return self.shape[i]

    def stride(self, i):
        return self.stride0


class Binding:
    def __init__(self, folder):
        src = os.path.join(folder, "stand_in.c")
        with open(src, "w") as f:
            f.write(STAND_IN)
        path = os.path.join(folder, "cheddar_b200_calls.so")
        subprocess.check_call(["gcc", "-O1", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "include"),
                               "-I" + sysconfig.get_paths()["include"], src,
                               os.path.join(ROOT, "cheddar-fhe_b200", "host", "py_calls.c"), "-o", path])
        spec = importlib.util.spec_from_file_location("cheddar_b200_calls", path)
        self.k = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(self.k)
        self.k.set_converters(lambda a: np.ascontiguousarray(a, dtype=np.int32),
                              lambda a: np.ascontiguousarray(a, dtype=np.uint32))
        self.lib = C.CDLL(path)

    def value(self, name):
        return C.c_int.in_dll(self.lib, name).value

    def table(self, t, n):
        return list(((C.c_size_t * 128) * 5).in_dll(self.lib, "table")[t][:n])

    def ints(self):
        return list((C.c_int * 64).in_dll(self.lib, "ints")[:self.value("n_ints")])

    def refused(self, error, call, *args):
        """The call raises `error` and the library is not entered."""
        before = self.value("calls")
        with pytest.raises(error):
            call(*args)
        assert self.value("calls") == before


@pytest.fixture(scope="module")
def binding(tmp_path_factory):
    return Binding(str(tmp_path_factory.mktemp("calls")))


def digits(first, n=BETA):
    return [Tensor(first + i) for i in range(n)]


X = Tensor(0x10)


def test_missing_operands_are_refused(binding):
    """None is an exception wherever an operand is needed: a null address would
    fault on the GPU."""
    b, g = binding, [0]
    k = b.k
    key, gap = digits(0x1000), [X, None]
    calls = [
        (k.ntt, (1, X, X, g, 0), (1, 2)),
        (k.intt, (1, X, X, g, None, 0, 0), (1, 2)),
        (k.binary, (1, 0, X, X, X, g), (2, 3)),
        (k.const_op, (1, 0, X, X, None, [3], g), (2, 3)),
        (k.tensor, (1, X, X, X, X, X, X, X, g), range(1, 8)),
        (k.permute, (1, X, X, None, 5, g), (1, 2)),
        (k.moddown, (1, 1, 0, X, X), (3, 4)),
        (k.keyswitch, (1, 1, X, X, X, None, key, key, 0), (2, 3, 4)),
        (k.hmult, (1, 1, X, X, X, X, X, X, key, key, 0, 1), range(2, 8)),
        (k.hoisted_rotations, (1, 1, X, X, X, [1], [key], [key], 0), (2, 3, 4)),
        (k.linear_transform, (1, 1, X, X, X, X, [0], [None], [0], [None], [[X]], 0, 1), range(2, 6)),
        (k.ctpt_gemm, (1, [X], [X, X], X, g), (3,)),
        (k.sample_uniform, (1, X, g, 1, 0), (1,)),
        (k.sample_error, (1, X, g, 3.2, 1, 0), (1,)),
        (k.encrypt, (1, X, X, X, X, None, g), range(1, 5)),
        (k.encode_coeffs, (1, X, np.zeros(65536), g), (1,)),
    ]
    for call, args, needed in calls:
        assert call(*args) == 0, call
        for i in needed:
            b.refused(AttributeError, call, *args[:i], None, *args[i + 1:])
    # entries of lists
    b.refused(AttributeError, k.ctpt_gemm, 1, gap, [X], X, g)
    b.refused(AttributeError, k.ctpt_gemm, 1, [X], gap, X, g)
    b.refused(AttributeError, k.keyswitch, 1, 1, X, X, X, None, gap, key, 0)
    b.refused(AttributeError, k.keyswitch, 1, 1, X, X, X, None, key, gap, 0)
    b.refused(AttributeError, k.hmult, 1, 1, X, X, X, X, X, X, gap, key, 0, 1)
    b.refused(AttributeError, k.hmult, 1, 1, X, X, X, X, X, X, key, gap, 0, 1)
    b.refused(AttributeError, k.hoisted_rotations, 1, 1, X, X, X, [1], [gap], [key], 0)
    for keys in ((None, key), (key, None)):
        b.refused(TypeError, k.hmult, 1, 1, X, X, X, X, X, X, *keys, 0, 1)
        b.refused(TypeError, k.keyswitch, 1, 1, X, X, X, None, *keys, 0)
        b.refused(TypeError, k.ctpt_gemm, 1, *((None, [X]) if keys[0] is None else ([X], None)), X, g)
    b.refused(TypeError, k.elementwise_multi, 1, 0, 0, None, [X], [X], None, g)
    b.refused(TypeError, k.elementwise_multi, 1, 0, 0, [X], None, [X], None, g)


def test_optional_entries_pass(binding):
    """Steps without a key, empty places of a plaintext table and second operands
    that an operation does not have stay null."""
    b = binding
    k1, k2 = digits(0x1000), digits(0x2000)
    pts = [[Tensor(0x20), Tensor(0x21)], [None, Tensor(0x23)]]
    assert b.k.linear_transform(1, 1, X, X, X, X, [0, 1], [None, (k1, k2)], [0, 2], [None, (k2, k1)], pts, 0, 1) == 0
    assert b.table(0, 4) == [0, 0, 0x1000, 0x1001] and b.table(1, 4) == [0, 0, 0x2000, 0x2001]
    assert b.table(2, 4) == [0, 0, 0x2000, 0x2001] and b.table(3, 4) == [0, 0, 0x1000, 0x1001]
    assert b.table(4, 4) == [0x20, 0x21, 0, 0x23]
    assert b.k.elementwise_multi(1, 0, 2, [X, X], [Tensor(0x30), Tensor(0x31)], [None, None], None, [0]) == 0
    assert b.table(1, 2) == [0x30, 0x31] and b.table(2, 2) == [0, 0]
    assert b.k.elementwise_multi(1, 0, 2, [X], [X], None, None, [0]) == 0


@pytest.mark.parametrize("count", [1, 2, 40])
def test_hoisted_rotation_keys(binding, count):
    """Every rotation gets its own digits, whatever the number of rotations
    (40 of them: more pointers than the binding keeps on the stack)."""
    b = binding
    kb, ka = ([digits(base + 16 * r) for r in range(count)] for base in (0x1000, 0x8000))
    rots = list(range(1, count + 1))
    assert b.k.hoisted_rotations(1, 1, X, X, X, rots, kb, ka, 0) == 0
    assert b.ints() == rots
    assert b.table(0, BETA * count) == [0x1000 + 16 * r + i for r in range(count) for i in range(BETA)]
    assert b.table(1, BETA * count) == [0x8000 + 16 * r + i for r in range(count) for i in range(BETA)]
    # a key with more digits than the level uses (made for a higher level) is used from its first digit on
    assert b.k.hoisted_rotations(1, 1, X, X, X, rots, [digits(0x1000 + 16 * r, 4) for r in range(count)], ka, 0) == 0
    assert b.table(0, BETA * count) == [0x1000 + 16 * r + i for r in range(count) for i in range(BETA)]
    # all digits in one list
    flat = [[t for k in kb for t in k]]
    assert b.k.hoisted_rotations(1, 1, X, X, X, rots, flat, ka, 0) == 0
    assert b.table(0, BETA * count) == [t.addr for t in flat[0]]


def test_hoisted_rotations_refuse_missing_keys(binding):
    b = binding
    k1, k2 = digits(0x1000), digits(0x2000)
    call = b.k.hoisted_rotations
    b.refused(TypeError, call, 1, 1, X, X, X, [1, 2], [None, k2], [k1, k2], 0)
    b.refused(TypeError, call, 1, 1, X, X, X, [1, 2], [k1, k2], [k1, None], 0)
    b.refused(AttributeError, call, 1, 1, X, X, X, [1, 2], [k1, [None, k2[1]]], [k1, k2], 0)
    b.refused(ValueError, call, 1, 1, X, X, X, [1, 2], [k1], [k1, k2], 0)
    b.refused(ValueError, call, 1, 1, X, X, X, [1, 2], [k1, k2], [k1, k2[:1]], 0)
    b.refused(ValueError, call, 1, 1, X, X, X, list(range(1, 41)), [k1] * 40, [k1] * 39, 0)


def test_short_digit_lists_are_refused(binding):
    b = binding
    k1 = digits(0x1000)
    for kb, ka in ((k1[:1], k1), (k1, k1[:1]), ([], k1)):
        b.refused(ValueError, b.k.hmult, 1, 1, X, X, X, X, X, X, kb, ka, 0, 1)
        b.refused(ValueError, b.k.keyswitch, 1, 1, X, X, X, None, kb, ka, 0)
        b.refused(ValueError, b.k.linear_transform, 1, 1, X, X, X, X, [0, 1], [None, (kb, ka)], [0], [None],
                  [[X, X]], 0, 1)
    # more digits than the level uses: a key made for a higher level
    assert b.k.hmult(1, 1, X, X, X, X, X, X, digits(0x1000, 4), digits(0x2000, 4), 0, 1) == 0
    assert b.table(0, 2) == [0x1000, 0x1001] and b.table(1, 2) == [0x2000, 0x2001]
    # an invalid level is the library's own error
    before = b.value("calls")
    assert b.k.hmult(1, 2, X, X, X, X, X, X, k1, k1, 0, 1) < 0
    assert b.k.hoisted_rotations(1, 2, X, X, X, [1], [k1], [k1], 0) < 0
    assert b.value("calls") == before


def test_element_wise_list_lengths(binding):
    """As many operands as destinations count: a shorter list ends in missing
    operands (which the library judges), a longer one is an error."""
    b = binding
    call = b.k.elementwise_multi
    assert call(1, 0, 2, [X, X], [Tensor(0x30), Tensor(0x31)], [Tensor(0x40)], None, [0]) == 0
    assert b.table(1, 2) == [0x30, 0x31] and b.table(2, 2) == [0x40, 0]
    assert call(1, 0, 2, [X, X], [X, X], [], None, [0]) == 0 and b.table(2, 2) == [0, 0]
    many = [Tensor(0x1000 + i) for i in range(70)]
    assert call(1, 0, 0, many, many, many[:65], None, [0]) == 0
    assert b.table(2, 70) == [t.addr for t in many[:65]] + [0] * 5
    b.refused(IndexError, call, 1, 0, 0, [X], [X, X], [X], None, [0])
    b.refused(IndexError, call, 1, 0, 0, [X], [X], [X, X], None, [0])


@pytest.mark.parametrize("gidx", [[3, 0, 7], (3, 0, 7), np.array([3, 0, 7]), np.array([3, 0, 7], dtype=np.int32),
                                  np.array([3, 0, 7], dtype=">i4"), np.array([3, 0, 7], dtype=np.uint32),
                                  np.array([3, 9, 0, 9, 7, 9], dtype=np.int32)[::2], range(3, 12, 4)])
def test_index_lists(binding, gidx):
    """Any sequence or array of integers, whatever its type, order or stride."""
    want = list(int(i) for i in gidx)
    assert binding.k.ntt(1, X, X, gidx, False) == 0
    assert binding.ints() == want
    assert binding.k.const_op(1, 0, X, X, None, gidx, gidx) == 0
    assert binding.ints() == want


def test_index_arrays_count_by_rows(binding):
    """As np.ascontiguousarray and len() count: the rows of a 2-D array, one for a
    number."""
    assert binding.k.ntt(1, X, X, np.arange(6, dtype=np.int32).reshape(2, 3), 0) == 0
    assert binding.ints() == [0, 1]
    for one in (5, np.int32(5), np.array(5, dtype=np.int32)):
        assert binding.k.ntt(1, X, X, one, 0) == 0
        assert binding.ints() == [5]


def test_indices_and_numbers_that_are_refused(binding):
    b, k, key = binding, binding.k, digits(0x1000)
    b.refused(TypeError, k.ntt, 1, X, X, None, 0)
    b.refused(TypeError, k.const_op, 1, 0, X, X, None, None, [0])
    b.refused(TypeError, k.hoisted_rotations, 1, 1, X, X, X, None, [key], [key], 0)
    b.refused(TypeError, k.linear_transform, 1, 1, X, X, X, X, [0], [None], [0], [None], [None], 0, 1)
    # a level, an operation, a stream number with a fraction
    b.refused(TypeError, k.moddown, 1, 1.5, 0, X, X)
    b.refused(TypeError, k.moddown, 1, 1, 0.0, X, X)
    b.refused(TypeError, k.binary, 1, 0.0, X, X, X, [0])
    b.refused(TypeError, k.const_op, 1, 0.5, X, X, None, [1], [0])
    b.refused(TypeError, k.hmult, 1, 1.0, X, X, X, X, X, X, key, key, 0, 1)
    b.refused(TypeError, k.keyswitch, 1, 1.0, X, X, X, None, key, key, 0)
    b.refused(TypeError, k.hoisted_rotations, 1, 1.0, X, X, X, [1], [key], [key], 0)
    b.refused(TypeError, k.linear_transform, 1, 1.0, X, X, X, X, [0], [None], [0], [None], [[X]], 0, 1)
    b.refused(TypeError, k.sample_uniform, 1, X, [0], 1, 2.0)
    b.refused(TypeError, k.sample_uniform, 1, X, [0], 1.0, 2)
    b.refused(TypeError, k.sample_error, 1, X, [0], 3.2, 1, 2.0)


def test_numbers_wrap_as_c_types(binding):
    b = binding
    assert b.k.sample_uniform(1, X, [0], 2 ** 64 + 5, 2 ** 32 + 7) == 0
    assert list((C.c_longlong * 2).in_dll(b.lib, "strides")) == [5, 7]
    assert b.k.sample_uniform(1, X, [0], 2 ** 64 - 1, 0) == 0
    assert list((C.c_longlong * 2).in_dll(b.lib, "strides")) == [-1, 0]
    assert b.k.permute(1, X, X, None, np.uint32(5), [0]) == 0 and b.ints() == [5]
    assert b.k.permute(1, X, X, None, 2 ** 70 + 9, [0]) == 0 and b.ints() == [9]
    # flags take what int() takes
    assert b.k.ntt(1, X, X, [0], np.bool_(True)) == 0 and b.k.ntt(1, X, X, [0], 1.0) == 0


def test_polynomials_and_strides(binding):
    b = binding
    assert b.k.ntt(1, Tensor(1, (5, 2, 65536), 131072), Tensor(2, (5, 2, 65536), 131073), [0, 1], 0) == 0
    assert b.value("polys") == 5 and list((C.c_longlong * 2).in_dll(b.lib, "strides")) == [131072, 131073]
    assert b.k.ntt(1, X, X, [0], 0) == 0 and b.value("polys") == 1


def test_calls_from_several_threads(binding):
    """Conversions keep nothing between calls."""
    import threading
    errors = []

    def work(first):
        keys = [digits(first + 16 * r) for r in range(40)]
        for _ in range(200):
            if binding.k.hoisted_rotations(1, 1, X, X, X, list(range(1, 41)), keys, keys, 0):
                errors.append(first)
            if binding.k.ctpt_gemm(1, [X] * 70, [X] * 90, X, [0, 1]):
                errors.append(first)

    threads = [threading.Thread(target=work, args=(0x10000 * (i + 1),)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
