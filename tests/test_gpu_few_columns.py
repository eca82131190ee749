"""Products of few columns, where the sliced tensor-core pass is slower than the
kernels that it replaces, take those; both agree with the oracle on either side
of the line (csrc/sigma_slices.cu, oz_faster).

adcgpu_test_set_status makes the sliced pass take every later product of a
context; its digits show in device_bytes.  Tolerances: as in
tests/test_gpu_sigma_slices.py (1e-13; FP32 values 1e-6).
"""
import numpy as np
import pytest

import oracle
from tests.conftest import system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,no,nv,m,sliced", [
    ("fp64", 3, 7, 1, False), ("fp64", 3, 8, 1, True), ("fp64", 2, 4, 2, True), ("fp64", 17, 9, 1, False),
    ("fp64", 17, 9, 2, True), ("fp64", 16, 9, 1, True),
    ("fp32", 5, 33, 2, False), ("fp32", 5, 33, 3, True), ("fp32", 2, 12, 4, False), ("fp32", 2, 13, 4, True),
    ("fp32", 3, 12, 16, False), ("fp32", 3, 13, 17, True), ("fp32", 17, 9, 5, False), ("fp32", 17, 9, 6, True),
    ("direct", 4, 17, 1, False), ("direct", 4, 17, 2, True),
    ("cvs", 3, 12, 4, False), ("cvs", 8, 40, 5, False), ("cvs", 8, 40, 8, True)])
def test_the_kernel_follows_the_columns(gpu, kind, no, nv, m, sliced):
    from adc_ottawa_gb300 import ADCGPU_DIRECT, ADCGPU_FP64, ADCGPU_MIXED, AdcGpu, AdcGpuError
    from adc_ottawa_gb300._native import lib

    e, eri = system(no, nv, 5 * no + nv)
    g = AdcGpu(0)
    g.set_orbitals(no, nv, e)
    g.set_eri_packed(eri)
    if kind == "cvs":
        g.write_fspace_adc2_1_cvs([2])
        ref = oracle.Matrix.build_cvs(no, nv, e, eri, [2])
    else:
        g.write_fspace_adc2_1(None, precision={"fp64": ADCGPU_FP64, "fp32": ADCGPU_MIXED, "direct": ADCGPU_DIRECT}[kind])
        ref = oracle.Matrix.build(no, nv, e, eri)
    if kind == "fp32":
        assert lib().adcgpu_sigma_set_shape(g._h, 64, 2, 4 | 256) == 0
    r = np.random.RandomState(m)
    x = r.standard_normal((g.ndim, m)) * 10.0 ** r.uniform(-3, 0, (g.ndim, m))
    x = np.asfortranarray(x.astype(np.float32 if kind == "fp32" else np.float64).astype(np.float64))
    want = ref.matvec(x)
    tol = 1e-6 if kind == "fp32" else 1e-13

    def product():
        w = g.sigma(x)
        assert (np.abs(w - want).max(axis=0) <= tol * np.abs(want).max(axis=0)).all()
        return g.device_bytes()

    first = product()
    assert lib().adcgpu_test_set_status(g._h, 5) == 0
    with pytest.raises(AdcGpuError):
        g.sigma(x)
    digits = product() - first          # those that were not there
    assert (digits == 0) == sliced
    g.close()


@pytest.mark.parametrize("prec", [0, 1])
def test_tuning_few_columns_leaves_the_others_alone(gpu, tmp_path, prec):
    """One column takes the per-warp pass at nocc=17 whatever the flag for it
    (bit 4) says; set, the flag would take it for every later product."""
    from adc_ottawa_gb300 import AdcGpu, autotune

    e, eri = system(17, 9, 94)
    g = AdcGpu(0)
    g.set_orbitals(17, 9, e)
    g.set_eri_packed(eri)
    g.write_fspace_adc2_1(None, precision=prec)
    for i in range(4):
        r = autotune.tune(g, 1, prec, cache=str(tmp_path / f"{i}.json"))
        assert r["mc"] & 16 == 0
    g.close()
