"""nadia_convert_to_fp64 on FresnelCDI_WF: the FP64 form gets its zone-plate
factors and goes on as an FP64 reconstruction from the same state does."""
import numpy as np
import pytest

import pynadia
from pynadia import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(256, 256), (512, 256)])
@pytest.mark.parametrize("steps", [0, 3])
def test_fresnel_wf_continues_as_fp64(nx, ny, steps):
    f = synth.FresnelWFCase(64, seed=6)  # its geometry
    g = np.random.default_rng(nx + ny)
    kw = dict(wavelength=f.wavelength, zone_focal_length=f.z12, focal_detector_length=f.z23,
              pixel_size=f.pixel)
    sup = synth.disk_mask(nx, ny, 0.3 * min(nx, ny)).astype(float)
    intensity = g.random((nx, ny)) * 100
    field = g.standard_normal((nx, ny)) + 1j * g.standard_normal((nx, ny))
    a = pynadia.Solver("fresnel_wf", nx, ny, precision=pynadia.FP32, **kw)
    b = pynadia.Solver("fresnel_wf", nx, ny, precision=pynadia.FP64, **kw)
    for s in (a, b):
        s.set_support(sup)
        s.set_intensity(intensity)
    a.set_exit_surface_wave(field)
    a.iterate(steps)
    esw = a.get_exit_surface_wave()
    a.convert_to_fp64()
    assert np.array_equal(a.get_exit_surface_wave(), esw)
    b.set_exit_surface_wave(esw)
    for _ in range(3):
        a.iterate()
        b.iterate()
        assert a.get_error() == b.get_error()
    assert np.array_equal(a.get_exit_surface_wave(), b.get_exit_surface_wave())
    assert np.array_equal(a.propagate_to_detector(field), b.propagate_to_detector(field))
    assert np.array_equal(a.propagate_from_detector(field), b.propagate_from_detector(field))
