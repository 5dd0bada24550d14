"""Row classes of a CSR matrix (csrc/csr_classes.cpp), compiled alone and compared with a
plain dictionary over the rows: any number of host threads gives the same classes, and
the limits are 256 classes and 32 entries per row."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "cpu-free-model_b200", "csrc")

WRAP = r"""
#include "csr_classes.h"
extern "C" int classes(int n, const int *rp, const int *col, const double *val, int threads,
                       unsigned char *cls, int *reps, int *count) {
    const cfm::RowClasses r = cfm::find_row_classes(n, rp, col, val, threads);
    for (int i = 0; i < n; ++i) cls[i] = r.kind ? r.cls[i] : 0;
    *count = r.kind ? (int)r.reps.size() : 0;
    for (int c = 0; c < *count; ++c) reps[c] = r.reps[c];
    return r.kind;
}
extern "C" const char *fault(int n, long long nnz, const int *rp, const int *col, int base) {
    return cfm::csr_fault(n, nnz, rp, col, base);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("classes")
    (d / "wrap.cpp").write_text(WRAP)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-fopenmp", "-I", CSRC, str(d / "wrap.cpp"),
                    os.path.join(CSRC, "csr_classes.cpp"), "-o", str(d / "classes.so")], check=True)
    out = ctypes.CDLL(str(d / "classes.so"))
    out.fault.restype = ctypes.c_char_p
    return out


def csr(rows):
    """rows: per row a list of (column, value)."""
    rp = np.zeros(len(rows) + 1, np.int32)
    rp[1:] = np.cumsum([len(r) for r in rows])
    flat = [e for r in rows for e in r]
    return rp, np.array([c for c, _ in flat], np.int32), np.array([v for _, v in flat], np.float64)


def plain(rows, values):
    ids, cls, reps = {}, [], []
    for i, r in enumerate(rows):
        key = tuple((c - i, np.float64(v).tobytes() if values else 0) for c, v in r)
        if key not in ids:
            ids[key] = len(reps)
            reps.append(i)
        cls.append(ids[key])
    return cls, reps


def check(lib, rows, kind, threads, base=0):
    rp, col, val = csr(rows)
    cls, reps, count = np.zeros(len(rows), np.uint8), np.zeros(256, np.int32), ctypes.c_int()
    col = np.ascontiguousarray(col + base)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    got = lib.classes(len(rows), p(rp), p(col), p(val), threads, p(cls), p(reps), ctypes.byref(count))
    assert got == kind
    if kind:
        want_cls, want_reps = plain(rows, kind == 2)
        np.testing.assert_array_equal(cls, want_cls)
        np.testing.assert_array_equal(reps[:count.value], want_reps)


@pytest.mark.parametrize("threads", [1, 2, 3, 7, 16])
def test_classes_of_a_grid_operator(lib, threads):
    n, w = 611, 13
    rng = np.random.default_rng(1)
    rows, varied = [], []
    for i in range(n):
        cols = [c for c in (i - w, i - 1, i, i + 1, i + w) if 0 <= c < n]
        rows.append([(c, 4.0 if c == i else -1.0) for c in cols])
        varied.append([(c, rng.uniform()) for c in cols])
    check(lib, rows, 2, threads)
    check(lib, rows, 2, threads, base=1)
    check(lib, varied, 1, threads)
    rows[n // 2] = []  # an empty row beside others
    check(lib, rows, 2, threads)
    rows[5] = [(c, 0.0 * v) for c, v in rows[5]]
    rows[6] = [(c, -0.0 * v) for c, v in rows[6]]  # zeros of either sign are not alike
    check(lib, rows, 2, threads)


@pytest.mark.parametrize("threads", [1, 2, 5])
def test_limits(lib, threads):
    n = 900
    diag = [[(i, 1.0 + i % 256)] for i in range(n)]
    check(lib, diag, 2, threads)  # exactly 256 classes of values
    diag[-1] = [(n - 1, 0.5)]
    check(lib, diag, 1, threads)  # 257: offsets alone
    offsets = [[((i + i % 256) % n if i + i % 256 < n else i, 1.0)] for i in range(n)]
    check(lib, offsets, 2, threads)
    offsets[0] = [(300, 1.0)]
    offsets[1] = [(700, 1.0)]
    kinds = len(plain(offsets, False)[1])
    assert kinds > 256
    check(lib, offsets, 0, threads)  # too many offsets: none
    full = [[(c, 1.0) for c in range(32)]] + [[(i, 1.0)] for i in range(1, n)]
    check(lib, full, 2, threads)  # 32 entries
    full[0].append((32, 1.0))
    check(lib, full, 0, threads)  # 33


def test_faults(lib):
    rp, col, _ = csr([[(0, 1.0)], [(1, 1.0)], [(2, 1.0)]])
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    assert lib.fault(3, ctypes.c_longlong(3), p(rp), p(col), 0) is None
    for bad in ([0, 1, 3], [0, -1, 2]):
        c = np.array(bad, np.int32)
        assert lib.fault(3, ctypes.c_longlong(3), p(rp), p(c), 0) == b"column index out of range"
    c = np.array([1, 2, 0], np.int32)
    assert lib.fault(3, ctypes.c_longlong(3), p(rp), p(c), 1) == b"column index out of range"
    rp[1] = 3
    assert lib.fault(3, ctypes.c_longlong(3), p(rp), p(col), 0) == b"rowptr must be non-decreasing"
