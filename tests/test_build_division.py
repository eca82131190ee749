"""The builder's division by sqrt(2.0) (csrc/build_kernels.cu, div_sqrt2):
two operations in place of an FP64 division, which must round every quotient
as the division does, because the kept structure of the matrix is bit-exact.

The method's error before its final rounding is below 2^-105 relative, so it
can differ only for dividends whose quotient lies within that distance of a
midpoint of two doubles.  With x = X and sqrt(2.0) = C as 53-bit integers
(powers of two aside) these are the solutions of X 2^s = d (mod C), s = 53 or
54, for the smallest remainders d: all of them up to 64 are enumerated here
and rounded exactly with rationals, beside random dividends.
"""
import math
import random
from fractions import Fraction as F

import pytest


def _div(x, zh, zl):
    q1 = float(F(x) * F(zl))               # one rounding: __dmul_rn
    return float(F(x) * F(zh) + F(q1))     # one rounding: __fma_rn


def test_division_by_sqrt2_rounds_correctly():
    c = math.sqrt(2.0)
    zh = float.fromhex("0x1.6a09e667f3bccp-1")
    zl = float.fromhex("0x1.08b2fb1366eaap-56")
    assert zh == float(1 / F(c)) and zl == float(1 / F(c) - F(zh))
    C = int(math.frexp(c)[0] * 2 ** 53)
    assert C % 2 == 1
    near = set()
    for s in (53, 54):
        inv = pow(pow(2, s, C), -1, C)
        for d in range(-64, 65):
            X = d * inv % C
            while X < 2 ** 53:
                if X >= 2 ** 52:
                    near.add(X)
                X += C
    assert len(near) > 100
    for X in near:
        assert _div(float(X), zh, zl) == float(F(X) / F(c))
    r = random.Random(1)
    for _ in range(20000):
        x = r.uniform(-1, 1) * 10.0 ** r.uniform(-13, 2)
        assert _div(x, zh, zl) == x / c


@pytest.mark.gpu
def test_vvov_layout_from_both_inputs(gpu):
    """The (vv|ov) block is stored in another order than it is gathered in:
    both input layouts give the same matrix, and the kept count the oracle's."""
    import numpy as np

    import oracle
    from adc_ottawa_gb300 import AdcGpu
    from tests.conftest import system

    no, nv = 3, 33
    e, eri = system(no, nv, 5)
    n = no + nv
    i, j = np.tril_indices(n)
    pair = np.zeros((n, n), np.int64)
    pair[i, j] = pair[j, i] = np.arange(len(i))
    a, b = np.maximum(pair[:, :, None, None], pair[None, None]), np.minimum(pair[:, :, None, None], pair[None, None])
    full = eri[a * (a + 1) // 2 + b]
    out = []
    for complex_layout in (False, True):
        g = AdcGpu(0)
        g.set_orbitals(no, nv, e)
        if complex_layout:
            g.set_eri_mo_complex(np.asfortranarray(full.astype(np.complex128)))
        else:
            g.set_eri_packed(eri)
        out.append((g.write_fspace_adc2_1(None), g.get_diag(), *g.export_coo()))
    for x, y in zip(*out):
        assert np.array_equal(x, y)
    ref = oracle.Matrix.build(no, nv, e, eri)
    assert out[0][0] == ref.nnz and np.array_equal(out[0][1], ref.coo()[0])
