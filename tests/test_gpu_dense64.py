"""The tall-skinny FP64 products of the solvers (csrc/dense.cu: k_tn64, k_nn64)
through block Lanczos (lancdiag_block, block_lanczos.f90:28-81), whose every
step is built of them, at block sizes with one column, odd columns, exactly
and just over 32 columns (the column split) and over 8 (the row kernel's),
in both arithmetics.

Reference: the same recurrence in numpy with LAPACK's QR, B_j with a positive
diagonal.  Each product is accurate to sqrt(N) 2^-53 ~ 1e-14 relative (FP64;
the double-float option: 1e-14 per product, its documented accuracy); three
cycles with a QR each lose at most the condition of the residual block, 1e2
here: 1e-11 (FP64) and 1e-10 (double-float) of max|T|.
"""
import numpy as np
import pytest

import oracle
from tests.conftest import system

pytestmark = pytest.mark.gpu

NO, NV = 4, 14


def _reference(H, q0, cycles):
    b = q0.shape[1]

    def qr(x):
        q, r = np.linalg.qr(x)
        s = np.sign(np.diag(r))
        return q * s, s[:, None] * r

    q, _ = qr(q0 / np.linalg.norm(q0, axis=0))
    T = np.zeros((b * cycles, b * cycles))
    basis = []
    for j in range(cycles):
        basis.append(q)
        u = H @ q
        T[j * b:(j + 1) * b, j * b:(j + 1) * b] = q.T @ u
        for _ in range(2):
            for p in basis:
                u = u - p @ (p.T @ u)
        q, r = qr(u)
        if j + 1 < cycles:
            T[(j + 1) * b:(j + 2) * b, j * b:(j + 1) * b] = r
            T[j * b:(j + 1) * b, (j + 1) * b:(j + 2) * b] = r.T
    return T


@pytest.mark.parametrize("df", [0, 1])
@pytest.mark.parametrize("b", [1, 2, 7, 8, 9, 32, 33, 41])
def test_block_lanczos_matches_numpy(gpu, b, df):
    from adc_ottawa_gb300 import AdcGpu

    e, eri = system(NO, NV, 31)
    d, h, oi, oj = oracle.Matrix.build(NO, NV, e, eri).coo()
    H = np.diag(d)
    H[oi - 1, oj - 1] = h
    H[oj - 1, oi - 1] = h
    g = AdcGpu(0)
    g.set_orbitals(NO, NV, e)
    g.set_eri_packed(eri)
    g.write_fspace_adc2_1(None)
    g.set_fp64_arith(df)
    q0 = np.random.RandomState(b).rand(len(d), b)
    T, ev, R = g.lancdiag_block(q0, 3, orthotype=1, want_ritz=True)
    ref = _reference(H, q0, 3)
    tol = (1e-10 if df else 1e-11) * np.abs(ref).max()
    assert np.abs(T - ref).max() <= tol
    assert np.abs(ev - np.linalg.eigvalsh(ref)).max() <= 10 * tol
    # Ritz vectors: unit norm, Rayleigh quotients equal to the Ritz values
    assert np.abs(np.linalg.norm(R, axis=0) - 1.0).max() <= 1e-12
    rq = np.einsum("ij,ij->j", R, H @ R)
    assert np.abs(rq - ev).max() <= 1e-8 * np.abs(ev).max()
