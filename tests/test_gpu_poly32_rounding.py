"""One FP32 PolyCDI iteration is as close to the FP64 form as it was when the
compiler contracted every product of the inverse column pass.  The distances are
those of that form on these inputs (deterministic: one tile shape per size); 0.1%
is left for the summation of the norm."""
import numpy as np
import pytest

import pynadia

pytestmark = pytest.mark.gpu

DISTANCE = {(240, 0): 2.5251e-07, (240, 3): 2.9770e-07, (480, 0): 2.7096e-07, (480, 3): 3.1911e-07,
            (232, 0): 2.4851e-07, (232, 3): 2.9295e-07, (496, 0): 2.7396e-07, (496, 3): 3.2279e-07}
PADDED = {240: 17, 480: 33, 232: 25, 496: 17}  # twice the padding and one


def step(n, precision, algorithm):
    g = np.random.default_rng(8 * n)
    s = pynadia.Solver("poly", n, n, precision=precision)
    r = PADDED[n] / n
    s.set_spectrum(np.array([(1e-10 * (1 + r), .4), (1e-10, 1.0), (1e-10 * (1 - r / 2), .5)]))
    s.set_support((g.random((n, n)) < .6).astype(float) * g.choice([1, .5], size=(n, n)))
    s.set_intensity(g.random((n, n)) * 50)
    x = g.standard_normal((n, n)) + 1j * g.standard_normal((n, n))
    s.set_exit_surface_wave(x.astype(np.complex64).astype(complex))
    s.set_algorithm(algorithm)
    s.iterate(1)
    return s.get_exit_surface_wave()


@pytest.mark.parametrize("n,algorithm", sorted(DISTANCE))
def test_one_step_distance(n, algorithm):
    a, b = step(n, pynadia.FP32, algorithm), step(n, pynadia.FP64, algorithm)
    assert np.linalg.norm(a - b) / np.linalg.norm(b) <= DISTANCE[n, algorithm] * 1.001
