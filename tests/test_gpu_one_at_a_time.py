"""A program that holds one reconstruction at a time pays for the process's
pinned memory and helper threads once, not with each reconstruction."""
import gc
import time

import numpy as np
import pytest

import pynadia
from pynadia import FP32, FP64

pytestmark = pytest.mark.gpu


def life(nx, ny, prec, data):
    """Milliseconds from the construction of a reconstruction to its end."""
    sup, intensity, x = data
    t = time.perf_counter()
    s = pynadia.Solver("planar", nx, ny, precision=prec)
    s.set_support(sup)
    s.set_intensity(intensity)
    s.set_exit_surface_wave(x)
    s.iterate(1)
    s.get_error()
    s.get_exit_surface_wave()
    del s
    gc.collect()
    return (time.perf_counter() - t) * 1e3


@pytest.mark.parametrize("nx,ny,prec", [(256, 256, FP64), (645, 475, FP64), (512, 512, FP32)])
def test_alone_as_beside_another(nx, ny, prec):
    """At most twice the time it takes while another reconstruction exists."""
    g = np.random.default_rng(0)
    sup = np.zeros((nx, ny))
    sup[nx // 4:nx // 2, ny // 4:ny // 2] = 1
    data = sup, g.random((nx, ny)) + 1, sup + 0j
    life(nx, ny, prec, data)
    gc.collect()
    alone = np.median([life(nx, ny, prec, data) for _ in range(9)])
    other = pynadia.Solver("planar", 64, 64, precision=FP64)
    beside = np.median([life(nx, ny, prec, data) for _ in range(9)])
    del other
    assert alone <= 2 * beside, (alone, beside)
