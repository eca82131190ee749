"""The work space of the matrix build and of the integral blocks fits itself to
the memory that is left: a matrix is not refused for want of larger batches.

The device is filled with a torch buffer up to what the results and the smallest
work space take; 32 MB more allow for the allocator's 2 MB pieces.
"""
import numpy as np
import pytest

from tests.conftest import system
from tests.test_gpu_digit_memory import MB, _Held, _context

pytestmark = pytest.mark.gpu


def test_build_in_little_room(gpu):
    """nocc=8, nvirt=80: full batches of the second-order terms take 145 MB."""
    from adc_ottawa_gb300 import AdcGpu

    no, nv = 8, 80
    a = _context(no, nv)
    e, eri = system(no, nv, 17)
    b = AdcGpu(0)
    b.set_orbitals(no, nv, e)
    b.set_eri_packed(eri)
    store = a.device_bytes() - b.device_bytes()
    tables = 2 * 8 * (no * nv) ** 2 + 8 * nv * nv * no      # and the terms of one sum
    with _Held(store + tables + 32 * MB):
        assert b.write_fspace_adc2_1(None) == a.write_fspace_adc2_1(None)
    assert np.array_equal(a.get_diag(), b.get_diag())
    for x, y in zip(a.export_coo(), b.export_coo()):
        assert np.array_equal(x, y)
    a.close()
    b.close()


def test_integrals_in_little_room(gpu):
    """nocc=32, nvirt=96: a second copy of the (vv|ov) block takes 226 MB, which
    is 134 MB more than the blocks that are filled after it."""
    from adc_ottawa_gb300 import AdcGpu

    no, nv = 32, 96
    n = no + nv
    npair = n * (n + 1) // 2
    eri = np.random.RandomState(0).standard_normal(npair * (npair + 1) // 2)
    e = np.concatenate([-2.0 + np.arange(no) / no, 0.5 + np.arange(nv) / nv])
    g = AdcGpu(0)
    g.set_orbitals(no, nv, e)
    empty = g.device_bytes()
    g.set_eri_packed(eri)
    blocks = g.device_bytes() - empty
    g.close()
    g = AdcGpu(0)
    g.set_orbitals(no, nv, e)
    with _Held(blocks + eri.nbytes + 32 * MB):
        g.set_eri_packed(eri)
    assert g.device_bytes() - empty == blocks
    g.close()
