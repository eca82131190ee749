"""The digit stores of the sliced sigma products are a cache: what else the
library needs the memory for comes first, in the same context and in others on
the device, and a matrix whose digits find no room keeps its other kernels.

The device is filled with a torch buffer (never touched) up to the room that a
case leaves; a product is compared with the one before at 1e-13 of its largest
element, the accuracy of either kernel (tests/test_gpu_sigma_slices.py).
"""
import threading

import numpy as np
import pytest

from tests.conftest import system

pytestmark = pytest.mark.gpu

MB = 1 << 20


class _Held:
    """Holds all of the free device memory but 'room' bytes."""

    def __init__(self, room):
        import torch

        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        self.buf = torch.empty(max(0, free - room), dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *a):
        import torch

        self.buf = None
        torch.cuda.empty_cache()


def _context(no=8, nv=80, cvs=None):
    from adc_ottawa_gb300 import AdcGpu

    e, eri = system(no, nv, 17)
    g = AdcGpu(0)
    g.set_orbitals(no, nv, e)
    g.set_eri_packed(eri)
    if cvs:
        g.write_fspace_adc2_1_cvs(cvs)
    else:
        g.write_fspace_adc2_1(None)
    return g


def _x(g, m=3):
    return np.asfortranarray(np.random.RandomState(m).standard_normal((g.ndim, m)))


def _same(w, ref):
    assert (np.abs(w - ref).max(axis=0) <= 1e-13 * np.abs(ref).max(axis=0)).all()


@pytest.mark.parametrize("cvs", [None, [1, 2, 3]])
def test_a_solver_gets_the_memory_of_the_digits(gpu, cvs):
    """The Lanczos basis does not fit beside the digits."""
    g = _context(cvs=cvs)
    x = _x(g, 4)
    w = g.sigma(x)
    t, _, _ = g.lancdiag_block(x, 8, orthotype=1)
    before = g.device_bytes()
    basis = 8 * g.ndim * 4 * 8
    with _Held(basis + 16 * MB):
        t2, _, _ = g.lancdiag_block(x, 24, orthotype=1, want_evals=False)     # three times the basis
        assert g.device_bytes() < before
        _same(g.sigma(x), w)
    assert np.abs(t2[:32, :32] - t).max() <= 1e-9 * np.abs(t).max()


def test_another_context_gets_the_memory_of_the_digits(gpu):
    a = _context()
    x = _x(a)
    w = a.sigma(x)
    before = a.device_bytes()
    with _Held(200 * MB):
        # refused before the digits of a are given back: its store alone is larger
        b = _context()
        assert a.device_bytes() < before
        _same(b.sigma(x), w)
        _same(a.sigma(x), w)
    b.close()


def test_refused_digits_stay_refused(gpu):
    """The kernel does not change between the products of a matrix when memory
    comes free; the next matrix asks again."""
    g = _context()
    x = _x(g)
    with _Held(300 * MB):
        w = g.sigma(x)
        held = g.device_bytes()
    _same(g.sigma(x), w)
    assert g.device_bytes() <= held + 16 * MB       # no digits
    g.write_fspace_adc2_1(None)
    _same(g.sigma(x), w)
    assert g.device_bytes() > held + 100 * MB


def test_digits_given_back_while_another_thread_computes(gpu):
    """Each product of b needs more than the room that is left beside a's
    digits (133 MB here), which fit again when it is done."""
    a, b = _context(6, 60), _context(6, 60)
    x, many = _x(a), _x(b, 300)         # 299 MB on the device, in and out
    w = a.sigma(x)
    errors = []

    def work():
        try:
            for _ in range(60):
                _same(a.sigma(x), w)
        except BaseException as err:
            errors.append(err)

    with _Held(290 * MB):
        ref = b.sigma(many)
        t = threading.Thread(target=work)
        t.start()
        for _ in range(5):
            _same(b.sigma(many), ref)
        t.join()
    assert not errors, errors
