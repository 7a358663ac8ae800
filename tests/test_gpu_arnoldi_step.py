"""One Arnoldi step of the solve's kernel by itself against two classical
Gram-Schmidt projections in FP64: every tile length, tiles that stay on chip and
tiles that stream through the ring, lengths that are no multiple of a tile or of
the streams' alignment, bases of one vector to the most that fit, and every size
of the second projection (none beyond rounding for an orthonormal basis; from
1e-9 to all of w' for one whose first vectors are not orthogonal).

Tolerance: the kernel works in pairs of 48 significant bits, u = 2^-48.  A
projection of n elements is right to a few u of |V_i| |w|, and an element of w''
collects nv rounded products of it: 64 u |w| for the coefficients, and for the
unit vector 64 u |w| / |w''|.  An FP32 sum of the second projection would be wrong
by 2^-24 of it, 1e4 times that for the larger ones here."""
import ctypes as C

import numpy as np
import pytest

from amps_gb300 import _capi

pytestmark = pytest.mark.gpu

U = 2.0 ** -48


def pairs(a):
    """rounded to hi + lo FP32"""
    hi = a.astype(np.float32)
    return hi.astype(np.float64) + (a - hi).astype(np.float32).astype(np.float64)


def step(V, w, d=None, tile=0, ctas=0):
    lib = _capi.load()
    nv, n = V.shape
    h, norm, vn, xf = np.zeros(nv), np.zeros(1), np.zeros(n), np.zeros(n, np.float32)
    ptr = lambda a, t: None if a is None else a.ctypes.data_as(C.POINTER(t))
    st = lib.amps_gpu_arnoldi_step(0, n, nv, ptr(V, C.c_double), ptr(w, C.c_double), ptr(d, C.c_double), tile, ctas,
                                   ptr(h, C.c_double), ptr(norm, C.c_double), ptr(vn, C.c_double),
                                   ptr(xf, C.c_float))
    return st, h, norm[0], vn, xf


def basis(n, nv, g, seed):
    """nv unit vectors, orthogonal but for V_0 . V_1 = g"""
    rng = np.random.default_rng(seed)
    V = np.linalg.qr(rng.standard_normal((n, nv)))[0].T
    if nv > 1:
        V[1] = g * V[0] + np.sqrt(1.0 - g * g) * V[1]
    return pairs(np.ascontiguousarray(V))


def check(n, nv, g, tile, ctas, scaled):
    V = basis(n, nv, g, n + nv)
    rng = np.random.default_rng(n)
    w = pairs(rng.standard_normal(n) + np.sqrt(n) * V.sum(axis=0))  # the larger part in the span
    d = pairs(rng.uniform(0.5, 2.0, n)) if scaled else None
    st, h, norm, vn, xf = step(V, w, d, tile, ctas)
    assert st == 0
    h1 = V @ w
    w1 = w - h1 @ V
    h2 = V @ w1
    w2 = w1 - h2 @ V
    nw, n2 = np.linalg.norm(w), np.linalg.norm(w2)
    assert np.max(np.abs(h - (h1 + h2))) < 64 * U * nw
    assert abs(norm - n2) < 64 * U * nw
    assert np.linalg.norm(vn - w2 / n2) < 64 * U * nw / n2
    ref = vn.astype(np.float32) * (1.0 if d is None else d.astype(np.float32))
    np.testing.assert_allclose(xf, ref, rtol=2.0 ** -23)


# (tile, vectors, length, CTAs): few tiles per CTA (on chip), many (streamed), both in one launch, ragged
SHAPES = [
    (128, 1, 256, 0), (128, 31, 128 * 5 + 5, 2), (128, 31, 128 * 6 + 1, 2), (128, 31, 128 * 12 + 77, 2), (128, 7, 128 * 90 + 3, 3),
    (256, 2, 256 * 3, 2), (256, 25, 256 * 3 + 1, 2), (256, 25, 256 * 11 + 130, 2), (256, 5, 256 * 70 + 2, 3),
    (512, 3, 512 * 3 + 9, 2), (512, 11, 512 * 9 + 300, 2), (512, 2, 512 * 50 + 257, 2),
    (1024, 1, 1024 * 3 + 1, 2), (1024, 4, 1024 * 9 + 1023, 2), (1024, 4, 1024 * 4 + 250, 3), (1024, 2, 1024 * 25, 2),
]


@pytest.mark.parametrize("g", [0.0, 1e-9, 1e-6, 0.3, 0.99])
@pytest.mark.parametrize("tile,nv,n,ctas", SHAPES)
def test_step_matches_fp64(tile, nv, n, ctas, g):
    check(n, nv, g, tile, ctas, scaled=(nv + n) % 2 == 0)
    check(n, nv, g, tile, ctas, scaled=(nv + n) % 2 == 1)


@pytest.mark.parametrize("nv,n", [(20, 320_001), (9, 640_002), (4, 1_250_003)])
def test_lengths_of_the_longer_tiles(nv, n):
    for g in (0.0, 0.3):
        check(n, nv, g, 0, 0, scaled=True)


@pytest.mark.parametrize("tile,nv,n,ctas", [(128, 31, 128 * 5 + 5, 2), (128, 31, 128 * 12 + 77, 2),
                                             (1024, 4, 1024 * 9 + 1023, 2)])
def test_exact_breakdown(tile, nv, n, ctas):
    """w in the span of unit vectors: nothing is left, and the next vector is zero"""
    V = np.zeros((nv, n))
    V[np.arange(nv), np.arange(nv) * (n // nv)] = 1.0
    c = np.arange(1.0, nv + 1.0)
    for w in (c @ V, np.zeros(n)):
        st, h, norm, vn, xf = step(V, w, None, tile, ctas)
        assert st == 0 and norm == 0.0
        np.testing.assert_allclose(h, V @ w, rtol=1e-15)
        assert not vn.any() and not xf.any()


def test_refused_arguments():
    V, w = basis(300, 2, 0.0, 1), np.ones(300)
    assert step(V, w, None, 64)[0] == 1
    assert step(V[:, :255].copy(), w[:255].copy())[0] == 1
    big = np.zeros((5, 2048))
    assert step(big, np.ones(2048), None, 1024)[0] == 1  # two tiles of 5 vectors do not fit on chip
    assert step(np.zeros((32, 2048)), np.ones(2048))[0] == 1


def test_refused_length():
    """beyond a tile copy's 32-bit coordinates; refused before any vector is read"""
    lib, a = _capi.load(), np.zeros(4)
    d, f = a.ctypes.data_as(C.POINTER(C.c_double)), a.ctypes.data_as(C.POINTER(C.c_float))
    assert lib.amps_gpu_arnoldi_step(0, 2 ** 31, 1, d, d, None, 0, 0, d, d, d, f) == 1
