"""Arrays between the host and the device: they pass through pinned slots in
pieces of whole rows, several threads at a time, and the FP32 form's panel
order is made on the way, so what comes back is what was set, to the bit."""
import threading

import numpy as np
import pytest

import pynadia
from pynadia import FP32, FP64

pytestmark = pytest.mark.gpu


def field(nx, ny, seed):
    g = np.random.default_rng(seed)
    return (g.standard_normal((nx, ny)) + 1j * g.standard_normal((nx, ny)))


def round_trip(kind, nx, ny, prec, seed=1):
    s = pynadia.Solver(kind, nx, ny, precision=prec)
    x = field(nx, ny, seed)
    s.set_exit_surface_wave(x)
    want = x.astype(np.complex64).astype(np.complex128) if prec == FP32 else x
    assert np.array_equal(s.get_exit_surface_wave(), want)
    assert np.array_equal(s.get_exit_surface_wave_f32(), x.astype(np.complex64))
    x32 = field(nx, ny, seed + 1).astype(np.complex64)
    s.set_exit_surface_wave_f32(x32)
    assert np.array_equal(s.get_exit_surface_wave_f32(), x32)
    assert np.array_equal(s.get_exit_surface_wave(), x32.astype(np.complex128))
    return s


# below, at and above one piece; long and short rows; grids of the PolyCDI form
@pytest.mark.parametrize("kind,nx,ny,prec", [
    ("planar", 256, 256, FP32), ("planar", 256, 4096, FP32), ("planar", 4096, 256, FP32),
    ("planar", 768, 1536, FP32), ("planar", 2048, 2048, FP32), ("poly", 240, 244, FP32),
    ("poly", 1008, 1020, FP32), ("planar", 33, 7, FP64), ("planar", 362, 362, FP64),
    ("planar", 363, 361, FP64), ("planar", 1000, 1050, FP64), ("planar", 4096, 512, FP64)])
def test_estimate_round_trip(kind, nx, ny, prec):
    round_trip(kind, nx, ny, prec)


@pytest.mark.parametrize("nx,ny", [(256, 512), (1536, 2048)])
def test_support_round_trip_fp32(nx, ny):
    """A shrinkwrap's support comes from the device (real values in panels)."""
    s = round_trip("planar", nx, ny, FP32)
    d = pynadia.Solver("planar", nx, ny, precision=FP64)
    sup = np.zeros((nx, ny))
    sup[nx // 4:nx // 2, ny // 4:ny // 2] = 1
    x = np.where(sup > 0, 1.0 + 0j, 0j)
    for h in (s, d):
        h.set_support(sup)
        h.set_exit_surface_wave(x)
        h.apply_shrinkwrap(1.5, 0.5)
    a, b = s.get_support(), d.get_support()
    # a box blurred by a symmetric window: the threshold at half the maximum
    # runs between pixels, so no rounding decides a pixel; columns from nx on
    # are not thresholded (apply_threshold's j < nx) and keep their blurred
    # values, 81 products and sums and a division in FP32 (85 roundings of
    # 2^-24 on either side of the division)
    assert np.array_equal(a == 0, b == 0)
    assert np.all(np.abs(a - b) <= 2 * 85 * 2.0 ** -24 * np.abs(b))


def test_threads_at_once():
    """Reconstructions on their own threads share the slots and the copying
    threads."""
    errors = []

    def work(k):
        try:
            for r in range(3):
                round_trip("planar", 1024, 1024 if k % 2 else 512, FP32 if k % 3 else FP64,
                           seed=10 * k + r)
        except Exception as e:  # reported by the main thread
            errors.append(e)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors


def test_error_history_past_the_ring():
    """The history keeps the last 65536 errors; a read that straddles the
    ring's end is put together in order."""
    s = pynadia.Solver("planar", 8, 8, precision=FP64)
    g = np.random.default_rng(0)
    s.set_support(np.ones((8, 8)))
    s.set_intensity(g.random((8, 8)) + 1)
    s.set_exit_surface_wave(field(8, 8, 3))
    s.set_algorithm("RAAR")
    s.iterate(65530)
    errs = []
    for _ in range(12):
        s.iterate()
        errs.append(s.get_error())
    assert np.array_equal(s.get_error_history(12), np.array(errs))
    assert np.array_equal(s.get_error_history(3), np.array(errs[-3:]))
