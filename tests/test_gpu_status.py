"""A pipeline wait of the tensor-core sigma kernels that gave up reaches the
caller of every entry point that runs sigma products: as ADCGPU_DEVICE_TIMEOUT,
whatever the rows it left behind led to, and once, not again in the next call.

The status word is set from the host (adcgpu_test_set_status): the kernels then
return at once, as after a lost wait, and nothing on the device waits.
"""
import numpy as np
import pytest

from tests.conftest import system

pytestmark = pytest.mark.gpu

TIMEOUT = 14
NO, NV = 3, 12


def _calls(g, precision):
    n = g.ndim
    r = np.random.RandomState(1)
    x = np.asfortranarray(r.standard_normal((n, 4)))
    psi = r.standard_normal(n) + 0j
    psi /= np.linalg.norm(psi)
    dtpsi = -1j * g.sigma(psi.real[:, None])[:, 0]
    return {
        "sigma": lambda: g.sigma(x),
        "davidson": lambda: g.davdiag_block(3, 1e-6, precision=precision),
        "lanczos": lambda: g.lancdiag_block(x, 6),
        "autocorr": lambda: g.propagate_fvec(x[:, :2], 1.0, 5.0, 8, 1e-6),
        "silstep": lambda: g.silstep(psi, dtpsi, 0.5, 8, 1e-6),
        "chebyshev_auto": lambda: g.chebyshev_auto(x, np.array([0.0, 8.0]), 20),
        "chebyshev_project": lambda: g.project_psi0(x[:, :1], np.array([0.0, 8.0]), 20, 1.0),
        "spectral_bounds": lambda: g.spectral_bounds(),
    }


@pytest.mark.parametrize("kind", ["fp64", "cvs", "mixed", "direct"])
def test_lost_wait_is_reported_once_by_every_entry_point(gpu, kind):
    from adc_ottawa_gb300 import ADCGPU_DIRECT, ADCGPU_FP64, ADCGPU_MIXED, AdcGpu, AdcGpuError
    from adc_ottawa_gb300._native import lib

    e, eri = system(NO, NV, 4)
    g = AdcGpu(0)
    g.set_orbitals(NO, NV, e)
    g.set_eri_packed(eri)
    precision = {"fp64": ADCGPU_FP64, "mixed": ADCGPU_MIXED, "direct": ADCGPU_DIRECT, "cvs": ADCGPU_FP64}[kind]
    if kind == "cvs":
        g.write_fspace_adc2_1_cvs([1, 2])
    else:
        g.write_fspace_adc2_1(None, precision=precision)
    calls = _calls(g, ADCGPU_FP64 if kind == "direct" else precision)
    if kind == "mixed":             # the propagators and Lanczos run on FP64 matrices
        calls = {n: calls[n] for n in ("sigma", "davidson")}
    if kind in ("cvs", "direct"):   # its guess needs a stored full matrix
        del calls["spectral_bounds"]
    for name, call in calls.items():
        call()
        assert lib().adcgpu_test_set_status(g._h, 5) == 0
        with pytest.raises(AdcGpuError) as err:
            call()
        assert err.value.code == TIMEOUT, (name, str(err.value))
        call()


def _cvs():
    from adc_ottawa_gb300 import AdcGpu

    e, eri = system(NO, NV, 4)
    g = AdcGpu(0)
    g.set_orbitals(NO, NV, e)
    g.set_eri_packed(eri)
    g.write_fspace_adc2_1_cvs([1, 2])
    return g


def test_lost_wait_comes_before_the_error_it_led_to(gpu):
    """A zero start vector ends a propagation with an error of its own (its
    norm is 0); after a lost wait the wait is reported, and not by the next call."""
    from adc_ottawa_gb300 import AdcGpuError
    from adc_ottawa_gb300._native import lib

    g = _cvs()
    call = lambda: g.propagate_fvec(np.zeros((g.ndim, 1)), 1.0, 5.0, 2, 1e-6)
    with pytest.raises(AdcGpuError) as err:
        call()
    assert err.value.code != TIMEOUT
    assert lib().adcgpu_test_set_status(g._h, 5) == 0
    with pytest.raises(AdcGpuError) as err:
        call()
    assert err.value.code == TIMEOUT, str(err.value)
    g.sigma(np.ones((g.ndim, 1)))


def test_no_product_follows_a_lost_wait_for_long(gpu):
    from adc_ottawa_gb300 import AdcGpuError
    from adc_ottawa_gb300._native import lib

    g = _cvs()
    x = np.asfortranarray(np.random.RandomState(2).standard_normal((g.ndim, 2)))
    n0 = lib().adcgpu_kernel_launches()
    g.lancdiag_block(x, 60)
    n1 = lib().adcgpu_kernel_launches()
    assert lib().adcgpu_test_set_status(g._h, 5) == 0
    with pytest.raises(AdcGpuError):
        g.lancdiag_block(x, 60)
    # the second cycle's product finds the first one's status
    assert lib().adcgpu_kernel_launches() - n1 < (n1 - n0) // 4
