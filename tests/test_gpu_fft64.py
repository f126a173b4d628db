"""The FP64 transforms and the passes fused with them, at the edges of their
tiles, against the oracle: the same operations in the same order, so every
value is equal and the error metric differs by its summation order only
(1e-12 relative, n additions of 2^-53 each for at most 2^20 pixels, sums of
positive terms taken in a tree)."""
import ctypes

import numpy as np
import pytest

import pynadia
import pyoracle as po
import scenarios as sc

pytestmark = pytest.mark.gpu

# one point, every radix and joined pair of radices, primes up to the largest,
# powers of two 64..4096 on either axis beside counts that leave a ragged tile,
# the longest line one block holds
SHAPES = [(1, 1), (1, 2), (2, 3), (3, 5), (5, 7), (7, 9), (6, 10), (12, 15), (14, 16), (11, 13),
          (17, 22), (30, 36), (45, 75), (64, 63), (128, 101), (256, 91), (512, 33), (1024, 5),
          (2048, 3), (4096, 1), (63, 64), (1, 4096), (5, 2048), (9, 1024), (7, 512), (13, 256),
          (11, 128), (1021, 4), (4, 1021), (2042, 3), (7264, 2), (2, 7264), (7263, 1),
          (605, 169), (1000, 48), (1080, 25), (640, 64)]


@pytest.mark.parametrize("nx,ny", SHAPES)
@pytest.mark.parametrize("forward", [True, False])
def test_transform_equals_oracle(nx, ny, forward):
    g = np.random.default_rng(nx * 8191 + ny)
    a = g.standard_normal((nx, ny)) + 1j * g.standard_normal((nx, ny))
    b = np.ascontiguousarray(a.copy())
    pynadia._check(pynadia.load().nadia_fft2d(
        b.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), nx, ny, int(forward)))
    assert np.array_equal(b, po.canon_fft2d(a, forward))


def test_refused_lengths():
    lib = pynadia.load()
    for nx, ny in ((2 * 1031, 4), (4, 8192), (8192, 4)):   # a prime above 1021; past the limit
        a = np.zeros((nx, ny), complex)
        assert lib.nadia_fft2d(a.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), nx, ny, 1) == 1


def gpu(kind, nx, ny, **kw):
    return pynadia.Solver(kind, nx, ny, precision=pynadia.FP64, **kw)


def orc(kind, nx, ny, **kw):
    return po.Oracle(kind, nx, ny, **kw)


def same(fn, exact=True, **kw):
    a, b = fn(gpu, **kw), fn(orc, **kw)
    assert sc.rel_err(a["errors"], b["errors"]) <= 1e-12
    for k in ("esw", "support", "transmission", "to_detector", "from_detector"):
        if k in b and exact:
            assert np.array_equal(a[k], b[k], equal_nan=True), k
        elif k in b:
            assert sc.rel_err(a[k], b[k]) <= 1e-10, k


@pytest.mark.parametrize("n,ny", [(128, 64), (512, 256), (1024, 66), (2048, 64), (4096, 34),
                                  (66, 512), (34, 2048), (34, 4096), (600, 90), (38, 1000)])
def test_planar_iterations(n, ny):
    same(sc.planar_mixed, n=n, ny=ny, hio=3, raar=2, er=2, n_best=0)


@pytest.mark.parametrize("n,ny", [(256, 256), (512, 128), (64, 1024), (90, 120)])
def test_fresnel_iterations(n, ny):
    same(sc.fresnel_mixed, n=n, ny=ny)


@pytest.mark.parametrize("n", [60, 256])
def test_fresnel_wf_iterations(n):
    same(sc.fresnel_wf_mixed, n=n, iterations=4)


@pytest.mark.parametrize("n,padding", [(120, 4), (60, 3), (90, 8)])
def test_poly_iterations(n, padding):
    same(sc.poly_mixed, exact=False, n=n, padding=padding)
