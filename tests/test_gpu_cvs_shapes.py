"""The launch shapes belong to the full matrix: on a CVS matrix setting or tuning
them is refused (status 16), and products go on."""
import ctypes as C

import numpy as np
import pytest

from tests.conftest import system

pytestmark = pytest.mark.gpu


def test_launch_shapes_are_refused_on_a_cvs_matrix(gpu):
    from adc_ottawa_gb300 import AdcGpu
    from adc_ottawa_gb300._native import lib

    e, eri = system(3, 12, 4)
    g = AdcGpu(0)
    g.set_orbitals(3, 12, e)
    g.set_eri_packed(eri)
    g.write_fspace_adc2_1_cvs([1])
    x = np.ones((g.ndim, 2), order="F")
    w = g.sigma(x)
    assert lib().adcgpu_sigma_set_shape(g._h, 64, 2, 4) == 16
    ch, mc, ms = C.c_int(0), C.c_int(0), C.c_double(0.0)
    assert lib().adcgpu_sigma_autotune(g._h, 2, C.byref(ch), C.byref(mc), C.byref(ms)) == 16
    assert np.abs(g.sigma(x) - w).max() <= 1e-13 * np.abs(w).max()
    g.close()
