"""The digits of a small matrix stay with the context for its next one
(csrc/sigma_slices.cu, OZ_SPARE_BYTES): products of matrices that follow each
other agree with the oracle (1e-13, tests/test_gpu_sigma_slices.py), the memory
is held once, given back when something else needs it, and freed with the context.
"""
import numpy as np
import pytest

import oracle
from tests.conftest import system
from tests.test_gpu_digit_memory import MB, _Held

pytestmark = pytest.mark.gpu


def _product(g, ref, m):
    r = np.random.RandomState(m)
    x = np.asfortranarray(r.standard_normal((g.ndim, m)) * 10.0 ** r.uniform(-3, 0, (g.ndim, m)))
    want = ref.matvec(x)
    assert (np.abs(g.sigma(x) - want).max(axis=0) <= 1e-13 * np.abs(want).max(axis=0)).all()


def test_matrices_that_follow_each_other(gpu):
    from adc_ottawa_gb300 import AdcGpu, ADCGPU_DIRECT, ADCGPU_FP64

    g = AdcGpu(0)
    # smaller, larger, another kind, the first again
    for no, nv, kind, m in ((5, 19, "fp64", 2), (3, 10, "fp64", 17), (6, 30, "fp64", 4), (4, 17, "direct", 3),
                            (8, 40, "cvs", 16), (5, 19, "fp64", 1)):
        e, eri = system(no, nv, 31)
        g.set_orbitals(no, nv, e)
        g.set_eri_packed(eri)
        if kind == "cvs":
            g.write_fspace_adc2_1_cvs([2])
            ref = oracle.Matrix.build_cvs(no, nv, e, eri, [2])
        else:
            g.write_fspace_adc2_1(None, precision=ADCGPU_DIRECT if kind == "direct" else ADCGPU_FP64)
            ref = oracle.Matrix.build(no, nv, e, eri)
        _product(g, ref, m)
        _product(g, ref, m + 1)
    g.close()


def test_kept_once_given_back_and_freed(gpu):
    import torch

    from adc_ottawa_gb300 import AdcGpu

    no, nv = 5, 19
    e, eri = system(no, nv, 31)
    ref = oracle.Matrix.build(no, nv, e, eri)
    g = AdcGpu(0)
    g.set_orbitals(no, nv, e)
    g.set_eri_packed(eri)
    g.write_fspace_adc2_1(None)
    built = g.device_bytes()
    _product(g, ref, 1)
    one = g.device_bytes()
    for _ in range(3):
        g.write_fspace_adc2_1(None)
        assert g.device_bytes() >= built + 4 * MB        # 9.5 MB of digits
        _product(g, ref, 1)
        assert g.device_bytes() == one
    g.write_fspace_adc2_1(None)
    with _Held(24 * MB):                                   # the integrals take 61 MB
        # fails, but first the digits went
        b = AdcGpu(0)
        b.set_orbitals(8, 80, system(8, 80, 17)[0])
        with pytest.raises(Exception):
            b.set_eri_packed(system(8, 80, 17)[1])
        b.close()
        assert g.device_bytes() < built + MB
    _product(g, ref, 1)
    g.write_fspace_adc2_1(None)
    free0, _ = torch.cuda.mem_get_info()
    held = g.device_bytes()
    g.close()
    assert torch.cuda.mem_get_info()[0] - free0 >= held // 2
