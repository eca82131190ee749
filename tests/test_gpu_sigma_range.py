"""The sliced sigma products (csrc/sigma_slices.cu) over the range of their type.

H (s x) = s H x exactly for a power of two s, as long as nothing leaves the
normal range, and to the grain of the smallest subnormal beyond: a product of
scaled columns has the accuracy of the unscaled one.

Tolerance: that of the unscaled product (tests/test_gpu_sigma_slices.py; the
FP32 one on top of FP32's rounding of the values), plus one half grain for each
of the at most N products and sums of an element.
"""
import ctypes as C

import numpy as np
import pytest

import oracle
from tests.conftest import system

pytestmark = pytest.mark.gpu


def _system(no, nv, precision=0, core=None):
    from adc_ottawa_gb300 import AdcGpu

    e, eri = system(no, nv, 3 * no + nv)
    g = AdcGpu(0)
    g.set_orbitals(no, nv, e)
    g.set_eri_packed(eri)
    if core:
        g.write_fspace_adc2_1_cvs(core)
        return g, oracle.Matrix.build_cvs(no, nv, e, eri, core)
    g.write_fspace_adc2_1(None, precision=precision)
    return g, oracle.Matrix.build(no, nv, e, eri)


def _vectors(N, m, seed):
    r = np.random.RandomState(seed)
    return r.standard_normal((m, N)) * 10.0 ** r.uniform(-3, 0, (m, N))


def _sigma(g, x):
    import torch

    from adc_ottawa_gb300._native import lib

    v = torch.from_numpy(x).cuda()
    w = torch.full_like(v, 3.0)
    torch.cuda.synchronize()
    st = lib().adcgpu_sigma_device(g._h, x.shape[0], C.c_void_p(v.data_ptr()), C.c_void_p(w.data_ptr()), x.shape[1])
    assert st == 0, lib().adcgpu_last_error(g._h)
    return w.cpu().numpy().astype(np.float64)


@pytest.mark.parametrize("scale", [-1040, -1015, -985, -940, -890, 980])
@pytest.mark.parametrize("no,nv,m,core", [(3, 9, 3, None), (5, 33, 17, None), (5, 33, 4, [1, 4])])
def test_fp64_columns_of_any_scale(gpu, no, nv, m, core, scale):
    from adc_ottawa_gb300 import ADCGPU_FP64

    g, ref = _system(no, nv, ADCGPU_FP64, core)
    x = np.ldexp(_vectors(g.ndim, m, nv), scale)
    w = _sigma(g, x)
    # the reference at a harmless scale, from the columns as they were rounded
    r = np.ldexp(ref.matvec(np.asfortranarray(np.ldexp(x, -scale).T)).T, scale)
    for c in range(m):
        assert (np.abs(w[c] - r[c]) <= 1e-13 * np.abs(r[c]).max() + g.ndim * 2.0 ** -1074).all()


@pytest.mark.parametrize("scale", [-125, -110, -95, -85, -60, 100])
@pytest.mark.parametrize("no,nv,m", [(3, 9, 3), (5, 33, 17)])
def test_fp32_columns_of_any_scale(gpu, no, nv, m, scale):
    """FP32 values and vectors (shape flag 256: the ladder's FP32 store)."""
    from adc_ottawa_gb300 import ADCGPU_MIXED
    from adc_ottawa_gb300._native import lib

    g, ref = _system(no, nv, ADCGPU_MIXED)
    assert lib().adcgpu_sigma_set_shape(g._h, 64, 2 | 8, 4 | 8 | 256) == 0
    x = np.ldexp(_vectors(g.ndim, m, nv), scale).astype(np.float32)
    w = _sigma(g, x)
    r = ref.matvec(np.asfortranarray(x.astype(np.float64).T)).T
    for c in range(m):
        assert (np.abs(w[c] - r[c]) <= 1e-6 * np.abs(r[c]).max() + g.ndim * 2.0 ** -149).all()
