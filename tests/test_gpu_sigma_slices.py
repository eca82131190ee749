"""The FP64 sigma product's sliced tensor-core pass (csrc/sigma_slices.cu).

W = H V (hxvec_incore, block_davidson.f90:844-883) at the sizes where the pass
changes shape: rows of exactly and just over 64, 128 and 384 values, tiles and
work items with a remainder, one to four 128-value groups, 8- and 16-column
operands with one to three column groups, vectors whose entries spread over
many decades, and a leading dimension larger than N.

Tolerance: both sides round every multiply-add or sum of a row at 2^-53 of a
partial sum; a singles row sums at most N = 1.6e5 products, so |W - W_ref| is
below sqrt(N) 2^-53 max|W| = 4.5e-14 max|W| on either side: 1e-13.
"""
import ctypes as C

import numpy as np
import pytest

import oracle
from tests.conftest import system

pytestmark = pytest.mark.gpu

TOL = 1e-13


def _build(no, nv, seed):
    from adc_ottawa_gb300 import AdcGpu

    e, eri = system(no, nv, seed)
    g = AdcGpu(0)
    g.set_orbitals(no, nv, e)
    g.set_eri_packed(eri)
    g.write_fspace_adc2_1(None)
    return g, e, eri


def _vectors(N, m, ld, seed):
    r = np.random.RandomState(seed)
    x = np.zeros((m, ld))
    x[:, :N] = r.standard_normal((m, N)) * 10.0 ** r.uniform(-6, 0, (m, N))
    return x


def _sigma(g, x, flag=0):
    import torch

    from adc_ottawa_gb300._native import lib

    # flag 32: the CUDA-core tile instead of the tensor-core pass
    assert lib().adcgpu_sigma_set_shape(g._h, 64, 2 | 8 | flag, 4 | 8 | flag) == 0
    v = torch.from_numpy(x).cuda()
    w = torch.full_like(v, 3.0)
    torch.cuda.synchronize()
    st = lib().adcgpu_sigma_device(g._h, x.shape[0], C.c_void_p(v.data_ptr()), C.c_void_p(w.data_ptr()), x.shape[1])
    assert st == 0, lib().adcgpu_last_error(g._h)
    w = w.cpu().numpy()
    assert (w[:, g.ndim:] == 3.0).all()
    return w[:, :g.ndim]


@pytest.mark.parametrize("no,nv,m,pad", [
    (2, 2, 1, 0), (1, 20, 3, 0), (3, 8, 8, 3), (3, 16, 9, 0), (4, 17, 16, 0), (2, 32, 17, 1), (5, 33, 3, 0), (3, 64, 33, 0),
    (3, 65, 5, 0), (2, 96, 16, 0), (9, 40, 2, 0), (7, 53, 31, 0), (16, 20, 18, 2), (17, 18, 5, 0),
    (32, 7, 16, 0)])
def test_sliced_product_matches_oracle(gpu, no, nv, m, pad):
    g, e, eri = _build(no, nv, 11 * no + nv)
    x = _vectors(g.ndim, m, g.ndim + pad, nv)
    ref = oracle.Matrix.build(no, nv, e, eri).matvec(np.asfortranarray(x[:, :g.ndim].T)).T
    w = _sigma(g, x)
    for c in range(m):
        assert np.abs(w[c] - ref[c]).max() <= TOL * np.abs(ref[c]).max()


@pytest.mark.parametrize("no,nv,m", [(2, 192, 17), (2, 193, 9), (10, 110, 20)])
def test_sliced_product_matches_tile(gpu, no, nv, m):
    """Up to 384 values a row: 16-column operands; above: 8-column ones."""
    g, _, _ = _build(no, nv, no + nv)
    x = _vectors(g.ndim, m, g.ndim, nv)
    w, ref = _sigma(g, x), _sigma(g, x, 32)
    for c in range(m):
        assert np.abs(w[c] - ref[c]).max() <= TOL * np.abs(ref[c]).max()


def test_nonfinite_column_stays_in_its_column(gpu):
    g, _, _ = _build(4, 20, 5)
    x = _vectors(g.ndim, 4, g.ndim, 1)
    clean = _sigma(g, x)
    for at, bad in ((3, np.nan), (g.ndim - 1, np.inf)):
        y = x.copy()
        y[2, at] = bad
        w, ref = _sigma(g, y), _sigma(g, y, 32)
        for c in (0, 1, 3):
            assert np.abs(w[c] - clean[c]).max() <= TOL * np.abs(clean[c]).max()
        # wherever the multiply-add product is not finite, so is the sliced one
        assert not np.isfinite(w[2][~np.isfinite(ref[2])]).any()


@pytest.mark.parametrize("no,nv,m,pad", [
    (2, 2, 1, 0), (1, 20, 3, 0), (4, 17, 16, 1), (2, 32, 17, 0), (5, 33, 3, 2), (3, 64, 33, 0), (3, 65, 20, 0),
    (16, 20, 18, 0), (17, 18, 5, 0), (2, 200, 7, 0)])
def test_sliced_fp32_values_match_oracle(gpu, no, nv, m, pad):
    """FP32 values and vectors (shape flag 256: the ladder's FP32 store).  The
    result is rounded to FP32 and the values were: 2^-24 of |W| and of
    sum |h| |x|, which stays below 8 max|W| for these vectors: 5e-7, 1e-6 with
    the accumulation."""
    import torch

    from adc_ottawa_gb300 import ADCGPU_MIXED, AdcGpu
    from adc_ottawa_gb300._native import lib

    e, eri = system(no, nv, 7 * no + nv)
    g = AdcGpu(0)
    g.set_orbitals(no, nv, e)
    g.set_eri_packed(eri)
    g.write_fspace_adc2_1(None, precision=ADCGPU_MIXED)
    x = _vectors(g.ndim, m, g.ndim + pad, nv).astype(np.float32)
    v = torch.from_numpy(x).cuda()
    w = {}
    for flag in (0, 32):
        assert lib().adcgpu_sigma_set_shape(g._h, 64, 2 | 8, 4 | 8 | 256 | flag) == 0
        o = torch.full_like(v, 3.0)
        torch.cuda.synchronize()
        st = lib().adcgpu_sigma_device(g._h, m, C.c_void_p(v.data_ptr()), C.c_void_p(o.data_ptr()), x.shape[1])
        assert st == 0, lib().adcgpu_last_error(g._h)
        assert (o.cpu().numpy()[:, g.ndim:] == 3.0).all()
        w[flag] = o.cpu().numpy()[:, :g.ndim].astype(np.float64)
    if nv <= 100:
        ref = oracle.Matrix.build(no, nv, e, eri).matvec(np.asfortranarray(x[:, :g.ndim].T.astype(np.float64))).T
    else:
        ref = w[32]     # the CUDA-core tile
    for c in range(m):
        assert np.abs(w[0][c] - ref[c]).max() <= 1e-6 * np.abs(ref[c]).max()


@pytest.mark.parametrize("no,nv,core,m", [(3, 9, [2], 1), (5, 33, [1, 4], 17), (19, 6, list(range(1, 18)), 9)])
def test_sliced_cvs_rows_match_oracle(gpu, no, nv, core, m):
    """The CVS pair rows (one to seventeen core holes per segment)."""
    from adc_ottawa_gb300 import AdcGpu

    e, eri = system(no, nv, no + nv)
    g = AdcGpu(0)
    g.set_orbitals(no, nv, e)
    g.set_eri_packed(eri)
    g.write_fspace_adc2_1_cvs(core)
    x = _vectors(g.ndim, m, g.ndim, 3)
    ref = oracle.Matrix.build_cvs(no, nv, e, eri, core).matvec(np.asfortranarray(x.T)).T
    w = g.sigma(np.asfortranarray(x.T)).T
    for c in range(m):
        assert np.abs(w[c] - ref[c]).max() <= TOL * np.abs(ref[c]).max()
