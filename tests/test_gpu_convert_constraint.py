"""nadia_convert_to_fp64 keeps a transmission constraint whole: its regions, their
parameters and the per-pixel part act in the FP64 form as if set there."""
import numpy as np
import pytest

import pynadia
import scenarios as sc
from pynadia import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("regions", [0, 1, 3])
@pytest.mark.parametrize("fixed", [False, True])
def test_constraint_carries_over(regions, fixed):
    n = 256
    c = synth.PlanarCase(n, 40, 2, 1e8, seed=3, support_side=100)
    masks, alphas, fixed_c = sc.constraint_regions(n)
    args = (True, True, -1, masks[:regions], alphas[:regions],
            np.full(regions, 0.25) if fixed else None)
    a = pynadia.Solver("planar", n, n, precision=pynadia.FP32)
    b = pynadia.Solver("planar", n, n, precision=pynadia.FP64)
    for s in (a, b):
        s.set_support(c.support)
        s.set_intensity(c.intensity)
        s.set_transmission_constraint(*args)
    a.initialise_estimate(1)
    a.iterate(3)
    esw = a.get_exit_surface_wave()
    a.convert_to_fp64()
    b.set_exit_surface_wave(esw)
    for alg in (sc.ER, sc.HIO):
        for s in (a, b):
            s.set_algorithm(alg)
            s.iterate(2)
    assert a.get_error() == b.get_error()
    assert np.array_equal(a.get_exit_surface_wave(), b.get_exit_surface_wave())
    # and without it
    for s in (a, b):
        s.clear_transmission_constraint()
        s.iterate(1)
    assert np.array_equal(a.get_exit_surface_wave(), b.get_exit_surface_wave())
