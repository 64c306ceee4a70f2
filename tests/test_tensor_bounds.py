"""The tests by which the tensor kernels reject combinations (csrc/tensor_bounds.h), compiled for the host and
compared with FP64 over tables of 2 to 81 cells, from 1 : 65 535 to 65 535 : 1 classes: no table's mutual
information exceeds its bound as the kernels sum it in single precision, and the key estimates stay within
their error bounds of the exact fixed-point key."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CLASSES = [(1, 1), (1, 3), (9, 5), (3, 997), (997, 3), (558, 1012), (4000, 4000), (800, 8000), (8000, 800),
           (1000, 20000), (20000, 1000), (600, 60000), (60000, 600), (100, 65535), (65535, 100), (1, 65535),
           (65535, 1), (65535, 65535)]
TINY = np.float32(2.0 ** -20)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("bounds")
    (d / "b.cpp").write_text(
        '#include "tensor_bounds.h"\nextern "C" {\n'
        "void quadratic(int a, int b, int cells, double* o) { fiu::f4_quadratic(a, b, cells, o[0], o[1]); }\n"
        "void quartic(int a, int b, int cells, double* o) {\n"
        "  const fiu::F4Quartic q = fiu::f4_quartic(a, b, cells, o[0], o[1]); o[2] = q.a2; o[3] = q.a3; o[4] = q.a4; }\n"
        "double least(double q) { return fiu::f4_least_ratio(q); }\n"
        "double margin3(int n) { return fiu::t3_margin(n); }\ndouble margin4(int n) { return fiu::t4x_margin(n); }\n}\n")
    so = str(d / "b.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "fiuncho_gb300", "csrc"),
                    str(d / "b.cpp"), "-o", so], check=True)
    L = ctypes.CDLL(so)
    for f in (L.least, L.margin3, L.margin4):
        f.restype = ctypes.c_double
    L.least.argtypes = [ctypes.c_double]
    return L


def _tables(n1, n0, cells, seed, m=400):
    """Tables of both classes: the same frequencies, different ones, and cells of one class or of few samples."""
    rng = np.random.default_rng(seed)
    conc = rng.choice([0.05, 0.3, 1.0, 10.0], (m, 1))
    p = rng.gamma(conc, 1.0, (m, cells)) + 1e-12
    p0 = p * np.where(rng.random((m, 1)) < 0.5, 1.0, rng.gamma(rng.choice([0.3, 2.0], (m, 1)), 1.0, (m, cells)) + 1e-9)
    out = [np.stack([rng.multinomial(n, row / row.sum()) for row in w]) for n, w in ((n1, p), (n0, p0))]
    return out[0].astype(np.float64), out[1].astype(np.float64)


def _xlg(x):
    return x * np.log2(np.maximum(x, 1))


def _nmi(a, b):
    n1, n0 = a.sum(1), b.sum(1)
    return (_xlg(a) + _xlg(b) - _xlg(a + b)).sum(1) + _xlg(n1 + n0) - _xlg(n1) - _xlg(n0)


def _fma(x, y, z):
    return (x.astype(np.float64) * y + z).astype(np.float32)


def _reciprocal(a, b, rng):
    s = (a + b).astype(np.float32) + TINY
    return ((1 / s.astype(np.float64)) * (1 + rng.uniform(-1, 1, s.shape) * 2.0 ** -23)).astype(np.float32)


@pytest.mark.parametrize("n1,n0", CLASSES)
@pytest.mark.parametrize("cells", [2, 3, 9, 27, 81])
def test_no_table_exceeds_its_bounds(lib, n1, n0, cells):
    a, b = _tables(n1, n0, cells, 1000 * cells + n1 % 991 + n0 % 97)
    nmi, rng = _nmi(a, b), np.random.default_rng(5)
    r, b32 = _reciprocal(a, b, rng), b.astype(np.float32)
    o = (ctypes.c_double * 5)()
    lib.quadratic(n1, n0, cells, o)
    acc = np.zeros(len(a), np.float32)
    for c in range(cells):
        acc = _fma(b32[:, c], (b32[:, c] * r[:, c]), acc)
    assert (acc >= o[0] * nmi + o[1]).all()
    lib.quartic(n1, n0, cells, o)
    a2, a3, a4 = (np.float32(x) for x in o[2:5])
    acc = np.zeros(len(a), np.float32)
    for c in range(cells):
        pr = b32[:, c] * r[:, c]
        acc = _fma(b32[:, c] * pr, _fma(pr, _fma(pr, a4, np.full_like(pr, a3)), a2), acc)
    assert (acc >= o[0] * nmi + o[1]).all()


@pytest.mark.parametrize("n1,n0", CLASSES)
def test_the_least_ratio_is_least(lib, n1, n0):
    """Everywhere on a fine grid towards both ends, in extended precision."""
    q = np.longdouble(n0) / (n1 + n0)
    x = np.linspace(-25, 25, 200001).astype(np.longdouble)
    p, p1 = 1 / (1 + np.exp(-x)), 1 / (1 + np.exp(x))
    d = p - q
    far = np.abs(d) > 1e-4 * min(q, 1 - q)
    p, p1, d = p[far], p1[far], d[far]
    l2 = np.log(np.longdouble(2))
    g = (p * np.log1p(d / q) + p1 * np.log1p(-d / (1 - q))) / l2 / d ** 2
    L0, L1 = -np.log1p(-q) / l2 / q ** 2, -np.log(q) / l2 / (1 - q) ** 2
    least = ((L0 + (L1 - L0) * p - g) / (p * p1)).min()
    got = lib.least(float(q))
    assert 0.998 * least - 2e-4 <= got <= least


def _exact_bits(a, b):
    t = lambda c: np.rint(c * np.log(np.maximum(c, 1)) * 2.0 ** 32)
    return (t(a) + t(b) - t(a + b)).sum(1) / (np.log(2) * 2.0 ** 32)


@pytest.mark.parametrize("n1,n0", CLASSES)
@pytest.mark.parametrize("cells", [27, 81])
@pytest.mark.parametrize("err", [-1, 1, 0])
def test_estimates_stay_within_their_error_bounds(lib, n1, n0, cells, err):
    """Logarithms off by 2^-18, all the same way or each its own."""
    a, b = _tables(n1, n0, cells, 7 + cells)
    rng = np.random.default_rng(6)
    a32, b32 = a.astype(np.float32), b.astype(np.float32)
    s32 = a32 + b32

    def lg(x):
        off = rng.uniform(-1, 1, x.shape) if err == 0 else err
        return (np.log2((x + TINY).astype(np.float64)) + off * 2.0 ** -18).astype(np.float32)

    kf = np.zeros(len(a), np.float32)
    for c in range(cells):
        x, y, s = a32[:, c], b32[:, c], s32[:, c]
        if cells == 27:  # order 3: term after term
            kf = _fma(x, lg(x), kf)
            kf = _fma(y, lg(y), kf)
            kf = _fma(-s, lg(s), kf)
        else:            # order 4: a cell's terms first
            kf = kf + (_fma(y, lg(y), x * lg(x)) - s * lg(s))
    margin = lib.margin3(n1 + n0) if cells == 27 else lib.margin4(n1 + n0)
    assert (np.abs(kf - _exact_bits(a, b)) <= margin).all()
