"""The singles block's product W1 = A V1 (csrc/sigma.cu: k_singles_gemm) where
the FP64 tile follows the column count: at the smallest singles space that
takes it (512) and one that no tile divides, with one column, column counts at
and just over a tile's, and over 32 (two column tiles).

Tolerance: at most n1 = 531 products a sum, in any order and split, each
rounded at 2^-53 of a partial sum on either side: below 2 sqrt(531) 2^-53 =
5.1e-15 of max|W1|; 1e-14.
"""
import ctypes as C

import numpy as np
import pytest

import oracle
from tests.conftest import system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("no,nv", [(2, 256), (3, 177)])
def test_singles_product_matches_oracle(gpu, no, nv):
    import torch

    from adc_ottawa_gb300 import AdcGpu
    from adc_ottawa_gb300._native import lib

    e, eri = system(no, nv, 5)
    g = AdcGpu(0)
    g.set_orbitals(no, nv, e)
    g.set_eri_packed(eri)
    g.write_fspace_adc2_1(None)
    n1 = no * nv
    x = np.zeros((41, g.ndim))
    x[:, :n1] = np.random.RandomState(nv).standard_normal((41, n1))
    ref = oracle.Matrix.build(no, nv, e, eri).matvec(np.asfortranarray(x.T)).T[:, :n1]
    v = torch.from_numpy(x).cuda()
    for m in (1, 7, 8, 9, 10, 17, 32, 33, 41):
        w = torch.full_like(v, 3.0)
        torch.cuda.synchronize()
        st = lib().adcgpu_sigma_device(g._h, m, C.c_void_p(v.data_ptr()), C.c_void_p(w.data_ptr()), g.ndim)
        assert st == 0, lib().adcgpu_last_error(g._h)
        d = np.abs(w[:m, :n1].cpu().numpy() - ref[:m]).max(axis=1)
        assert (d <= 1e-14 * np.abs(ref[:m]).max(axis=1)).all(), m
