"""The FP64 sliced sigma product on values and vectors whose digits share their
sign and size.

The slices' group sums are whole numbers in FP32 accumulators.  With random
digits they stay far below 2^24; with every base-256 digit of every operand
near 127 they reach (g + 1) K 127^2 for group g of a row of K values, above
2^24 from g = 2 on at K = 512.  Integrals and vectors here are such numbers, at
the widths of one to four 128-value groups.

Reference: the CUDA-core tile's multiply-adds.  All products of the rows looked
at (the doubles with a' = b', whose values are plain integrals, and the singles)
are positive but those of the diagonal and of segment A, so each side's error is
at most n 2^-53 of a sum of n terms, on average sqrt(n) 2^-54: with n = 2 nvirt
for a double, below 1e-14, and the digits' own rounding, 2^-55 a product: 2e-14
of the row's largest result.  The singles sum up to N = 1.3e5 terms: 1e-13.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _structured(r, n):
    """n numbers in (0.75, 1), base-256 digits 100..127 down to the last bit."""
    u = np.zeros(n, np.uint64)
    for i in range(7):
        u = u * np.uint64(256) + r.randint(100, 128, n).astype(np.uint64)
    u &= ~np.uint64(3)                      # 53 of the 55 bits below 1
    return u.astype(np.float64) * 2.0 ** -55


@pytest.mark.parametrize("nv,m", [(60, 10), (128, 10), (136, 10), (180, 10), (192, 16), (200, 10), (256, 10), (256, 3)])
def test_structured_digits(gpu, nv, m):
    import torch

    from adc_ottawa_gb300 import AdcGpu
    from adc_ottawa_gb300._native import lib

    no, r = 2, np.random.RandomState(nv)
    nb = no + nv
    npair = nb * (nb + 1) // 2
    # integrals (pq|rs), symmetric in all eight ways by the packing
    g = AdcGpu(0)
    g.set_orbitals(no, nv, np.concatenate([[-200.0, -100.0], np.linspace(100.0, 200.0, nv)]))
    g.set_eri_packed(_structured(r, npair * (npair + 1) // 2))
    g.write_fspace_adc2_1(None)
    x = _structured(r, 16 * g.ndim).reshape(16, g.ndim)
    v = torch.from_numpy(x).cuda()
    w = []
    for flag, cols in ((0, m), (32, 16)):        # 32: the CUDA-core tile (from 16 columns on)
        assert lib().adcgpu_sigma_set_shape(g._h, 64, 2 | 8 | flag, 4 | 8 | flag) == 0
        o = torch.empty_like(v)
        torch.cuda.synchronize()
        st = lib().adcgpu_sigma_device(g._h, cols, C.c_void_p(v.data_ptr()), C.c_void_p(o.data_ptr()), g.ndim)
        assert st == 0, lib().adcgpu_last_error(g._h)
        w.append((o - torch.from_numpy(g.get_diag()).cuda() * v)[:m])
    n1, pv = no * nv, nv * (nv - 1) // 2
    c2 = slice(n1 + n1 + no * pv, n1 + n1 + no * pv + nv)      # doubles (a, a, k' < l')
    d = (w[0] - w[1]).abs()
    for rows, tol in ((c2, 2e-14), (slice(0, n1), 1e-13)):
        rel = (d[:, rows].amax(1) / w[1][:, rows].abs().amax(1)).max().item()
        print(f"nvirt={nv} m={m} rows {rows.start}..: {rel:.1e}")
        assert rel <= tol
