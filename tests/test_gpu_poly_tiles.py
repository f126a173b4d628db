"""PolyCDI's FP32 passes on the 1080-point tiles whose threads hold one
butterfly per pass, at the paddings and windows where their index ranges end:
narrow and wide padding, a window whose edge falls inside a panel run of the
tile, and axes of different padding; one iteration against the FP64 form at
the per-step bar of the FP32 tests (2e-5), and the column and row transforms
through it in every algorithm's combine."""
import numpy as np
import pytest

import pynadia
from pynadia import synth

pytestmark = pytest.mark.gpu

STEP_TOL = 2e-5


def pair(nx, ny, spectrum, seed=5):
    g = np.random.default_rng(seed)
    i = np.arange(nx)[:, None] - nx / 2
    j = np.arange(ny)[None, :] - ny / 2
    r = 0.16 * min(nx, ny)
    inside = i * i + j * j <= r * r
    obj = np.where(inside, (0.5 + 0.5 * g.random((nx, ny))) * np.exp(1j * g.random((nx, ny))), 0)
    out = []
    for prec in (pynadia.FP64, pynadia.FP32):
        s = pynadia.Solver("poly", nx, ny, precision=prec)
        s.set_spectrum(spectrum)
        s.set_support((i * i + j * j <= (1.2 * r) ** 2).astype(float))
        out.append(s)
    # data of a different object of the same kind, so the modulus does work
    px, py = out[0].get_padding()
    f = np.zeros((nx + 2 * px, ny + 2 * py), complex)
    f[px:px + nx, py:py + ny] = obj * np.exp(0.3j * g.random((nx, ny)))
    inten = np.abs(np.fft.fftshift(np.fft.fft2(f)))[px:px + nx, py:py + ny] ** 2 / f.size
    for s in out:
        s.set_intensity(inten + 1e-3 * inten.mean())
        s.set_exit_surface_wave(obj)
    return out, (px, py)


@pytest.mark.parametrize("n,padding", [(1024, 28), (1072, 4), (1040, 20), (1008, 36), (960, 60)])
@pytest.mark.parametrize("alg", ["ER", "HIO", "RAAR"])
def test_one_iteration_matches_fp64(n, padding, alg):
    (a, b), pad = pair(n, n, synth.gaussian_spectrum(10, 0.05, 1e-10, padding, n))
    assert pad == (padding, padding)
    for s in (a, b):
        s.set_algorithm(alg)
        s.iterate(1)
    assert abs(b.get_error() - a.get_error()) <= STEP_TOL * a.get_error()
    xa, xb = a.get_exit_surface_wave(), b.get_exit_surface_wave()
    assert np.linalg.norm(xb - xa) <= STEP_TOL * np.linalg.norm(xa)
    # a second iteration starts from the rows the first one transformed
    for s in (a, b):
        s.set_exit_surface_wave(xa)
        s.iterate(2)
    xa, xb = a.get_exit_surface_wave(), b.get_exit_surface_wave()
    assert np.linalg.norm(xb - xa) <= 2 * STEP_TOL * np.linalg.norm(xa)


def test_batch_equals_alone():
    spectrum = synth.gaussian_spectrum(10, 0.05, 1e-10, 28, 1024)
    batch = [pair(1024, 1024, spectrum, seed)[0][1] for seed in (1, 2, 3)]
    alone = [pair(1024, 1024, spectrum, seed)[0][1] for seed in (1, 2, 3)]
    for s in batch + alone:
        s.set_algorithm("HIO")
    pynadia.iterate_many(batch, 18)
    for s in alone:
        s.iterate(18)
    for x, y in zip(batch, alone):
        assert np.array_equal(x.get_exit_surface_wave_f32(), y.get_exit_surface_wave_f32())
        assert np.array_equal(x.get_error_history(18), y.get_error_history(18))
