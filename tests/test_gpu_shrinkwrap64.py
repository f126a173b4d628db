"""The FP64 shrinkwrap and soften at the edges of their tiles, against the
oracle: every sum has the reference's terms in the reference's order, so the
support is equal to the bit (0/0 included, where nothing passes the threshold)."""
import numpy as np
import pytest

import pynadia
import pyoracle as po

pytestmark = pytest.mark.gpu

SIZES = [(2, 2), (7, 7), (9, 5), (31, 31), (32, 32), (33, 33), (40, 64), (64, 40), (96, 96),
         (131, 129), (256, 256)]


def both(nx, ny):
    g = np.random.default_rng(nx * 997 + ny)
    sup = (g.random((nx, ny)) > 0.3).astype(float)
    x = g.standard_normal((nx, ny)) * np.exp(2j * np.pi * g.random((nx, ny)))
    out = []
    for make in (lambda: pynadia.Solver("planar", nx, ny, precision=pynadia.FP64),
                 lambda: po.Oracle("planar", nx, ny)):
        s = make()
        s.set_support(sup, True)
        s.set_exit_surface_wave(x)
        out.append(s)
    return out


@pytest.mark.parametrize("nx,ny", SIZES)
def test_shrinkwrap_equals_oracle(nx, ny):
    a, b = both(nx, ny)
    assert np.array_equal(a.get_support(), b.get_support())     # softened: cut-off 5
    for width, t in ((1.5, 0.1), (1.5, 0.0), (3.0, 0.9), (0.4, 1.0), (1.5, 1.5), (2.0, 0.3)):
        a.apply_shrinkwrap(width, t)
        b.apply_shrinkwrap(width, t)
        assert np.array_equal(a.get_support(), b.get_support(), equal_nan=True), (width, t)


def test_fp32_error_and_flag_after_many_steps():
    """get_error waits for the work before it and returns the last iteration's
    metric in both forms."""
    g = np.random.default_rng(3)
    for prec in (pynadia.FP64, pynadia.FP32):
        s = pynadia.Solver("planar", 256, 256, precision=prec)
        assert s.get_error() == 0.0
        s.set_support((g.random((256, 256)) > 0.5).astype(float))
        s.set_intensity(g.random((256, 256)))
        s.initialise_estimate(1)
        errs = []
        for _ in range(5):
            s.iterate()
            errs.append(s.get_error())
        assert np.array_equal(s.get_error_history(5), errs)
