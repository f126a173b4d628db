"""FP64 PolyCDI and FresnelCDI_WF on grids whose sides (and, for PolyCDI, whose
paddings) differ, against the oracle: the fused passes index rows, columns,
pitches and tables per axis.

The operations and their order are the oracle's, so the bounds are those of the
square grids: the error metric differs by its summation order (1e-12 relative),
FresnelCDI_WF's values are equal, and PolyCDI's estimate, whose expansion squares
a magnitude the oracle also squares, stays within 1e-10."""
import numpy as np
import pytest

import pynadia
import pyoracle as po
import scenarios as sc
from pynadia import synth

pytestmark = pytest.mark.gpu


def gpu(kind, nx, ny, **kw):
    return pynadia.Solver(kind, nx, ny, precision=pynadia.FP64, **kw)


def orc(kind, nx, ny, **kw):
    return po.Oracle(kind, nx, ny, **kw)


def poly(make, nx, ny, spread, stop):
    g = np.random.default_rng(nx * 1000 + ny)
    s = make("poly", nx, ny)
    sup = np.zeros((nx, ny))
    sup[nx // 3:2 * nx // 3, ny // 4:3 * ny // 4] = 1
    s.set_support(sup)
    s.set_intensity(g.random((nx, ny)) * 100)
    # longest wavelength first: paddings int(spread * nx / 2) and int(spread * ny / 2)
    s.set_spectrum(np.array([[1e-10 * (1 + d), w] for d, w in
                             ((spread, 0.4), (spread / 3, 0.8), (0.0, 1.0), (-spread, 0.3))]))
    if stop:
        bs = np.ones((nx, ny))
        bs[nx // 2 - 3:nx // 2 + 2, ny // 2 - 2:ny // 2 + 4] = 0
        s.set_beam_stop(bs)
    s.set_exit_surface_wave(sup * (g.random((nx, ny)) + 1j * g.random((nx, ny))))
    errs = []
    for alg, count in ((sc.ER, 2), (sc.HIO, 4), (sc.RAAR, 2)):
        s.set_algorithm(alg)
        for _ in range(count):
            s.iterate()
            errs.append(s.get_error())
    return np.array(errs), s.get_exit_surface_wave()


@pytest.mark.parametrize("nx,ny,spread,stop", [(64, 200, 0.071, False), (200, 64, 0.071, True),
                                               (90, 160, 0.101, True), (146, 22, 0.2, False)])
def test_poly(nx, ny, spread, stop):
    ea, a = poly(gpu, nx, ny, spread, stop)
    eb, b = poly(orc, nx, ny, spread, stop)
    assert sc.rel_err(ea, eb) <= 1e-12
    assert sc.rel_err(a, b) <= 1e-10


def wf(make, nx, ny):
    f = synth.FresnelWFCase(64, seed=6)  # its geometry
    g = np.random.default_rng(nx * 1000 + ny)
    s = make("fresnel_wf", nx, ny, wavelength=f.wavelength, zone_focal_length=f.z12,
             focal_detector_length=f.z23, pixel_size=f.pixel)
    s.set_support(synth.disk_mask(nx, ny, 0.3 * min(nx, ny)).astype(float))
    s.set_intensity(g.random((nx, ny)) * 100)
    field = g.standard_normal((nx, ny)) + 1j * g.standard_normal((nx, ny))
    s.set_exit_surface_wave(field)
    errs = []
    for _ in range(4):
        s.iterate()
        errs.append(s.get_error())
    return (np.array(errs), s.get_exit_surface_wave(), s.propagate_to_detector(field),
            s.propagate_from_detector(field))


@pytest.mark.parametrize("nx,ny", [(60, 256), (256, 90), (128, 64), (34, 1000)])
def test_fresnel_wf(nx, ny):
    a, b = wf(gpu, nx, ny), wf(orc, nx, ny)
    assert sc.rel_err(a[0], b[0]) <= 1e-12
    for x, y in zip(a[1:], b[1:]):
        assert np.array_equal(x, y)
