"""Workloads of the ADC(2)-s library, at the sizes it is used at.

Every case goes through the package's public entry points on one synthetic
closed-shell system: orbital energies U(-1.4, -0.4) Ha (occupied) and
U(0.1, 3.0) Ha (virtual), real MO integrals (pq|rs) of 8-fold symmetry,
N(0,1) * 0.3 * exp(-0.15|p-r| - 0.15|q-s|).  A case's "kind" is the call:

  sigma     W = H V for m columns on the resident matrix, device buffers: the
            product every solver spends its time in.  "precision": fp64 (the
            drop-in path), mixed (BF16 values, FP32 vectors), direct (coupling
            block recomputed in every product) or cvs (core-valence-separated
            space of the ncore deepest orbitals); "df": the double-float
            arithmetic option of the FP64 block products
  build     orbital energies and packed integrals up from the host, matrix
            build, diagonal back: what a new geometry costs
  lanczos   block Lanczos from a dipole-like start block, host block in, T
            matrix and its eigenvalues out
  davidson  the lowest excitation energies on the resident matrix

The random state of a case is made on the device from its seed alone.
"""
import numpy as np
import torch

from adc_ottawa_gb300 import api

PRECISION = {"fp64": api.ADCGPU_FP64, "mixed": api.ADCGPU_MIXED, "direct": api.ADCGPU_DIRECT, "cvs": api.ADCGPU_FP64}


def listed():
    return [
        # one Ritz vector of a small molecule: launches and latency
        {"name": "sigma_fp64_one", "kind": "sigma", "nocc": 5, "nvirt": 19, "m": 1, "precision": "fp64", "df": False},
        # a Lanczos block of ten dipole-like vectors
        {"name": "sigma_fp64_block10", "kind": "sigma", "nocc": 10, "nvirt": 110, "m": 10, "precision": "fp64", "df": False},
        # 32 wavepackets carried as 64 real columns
        {"name": "sigma_fp64_packets", "kind": "sigma", "nocc": 10, "nvirt": 110, "m": 64, "precision": "fp64", "df": False},
        # the default block of a 20-root Davidson on the largest system
        {"name": "sigma_fp64_large", "kind": "sigma", "nocc": 16, "nvirt": 180, "m": 40, "precision": "fp64", "df": False},
        # the FP64 refinement block of the mixed-precision ladder, odd sizes
        {"name": "sigma_df_refine", "kind": "sigma", "nocc": 13, "nvirt": 131, "m": 30, "precision": "fp64", "df": True},
        # the mixed ladder's block on the largest system
        {"name": "sigma_mixed_large", "kind": "sigma", "nocc": 16, "nvirt": 180, "m": 40, "precision": "mixed", "df": False},
        # a few unconverged roots left, ragged sizes
        {"name": "sigma_mixed_ragged", "kind": "sigma", "nocc": 9, "nvirt": 101, "m": 5, "precision": "mixed", "df": False},
        # the matrix-free path of a memory-bound user
        {"name": "sigma_direct", "kind": "sigma", "nocc": 10, "nvirt": 110, "m": 10, "precision": "direct", "df": False},
        # K-edge block
        {"name": "sigma_cvs", "kind": "sigma", "nocc": 9, "nvirt": 107, "m": 7, "precision": "cvs", "df": False, "ncore": 3},
        # a new geometry
        {"name": "build", "kind": "build", "nocc": 10, "nvirt": 110, "precision": "fp64"},
        # a short band Lanczos spectrum
        {"name": "lanczos", "kind": "lanczos", "nocc": 10, "nvirt": 110, "m": 10, "cycles": 12},
        # ten excitation energies to 1e-6 by the mixed-precision ladder
        {"name": "davidson_mixed", "kind": "davidson", "nocc": 10, "nvirt": 110, "roots": 10, "precision": "mixed"},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["fp64", "fp64", "fp64", "df", "mixed", "mixed", "direct", "cvs", "build", "lanczos", "davidson"])
    if kind in ("lanczos", "davidson"):
        no, nv = rng.randint(5, 10), _log_int(rng, 19, 110)
        if kind == "lanczos":
            return {"kind": kind, "nocc": no, "nvirt": nv, "m": rng.randint(2, 12), "cycles": rng.randint(6, 12)}
        return {"kind": kind, "nocc": no, "nvirt": nv, "roots": rng.randint(4, 10), "precision": rng.choice(["fp64", "mixed"])}
    if kind == "build":
        return {"kind": kind, "nocc": rng.randint(4, 12), "nvirt": _log_int(rng, 19, 120), "precision": rng.choice(["fp64", "mixed"])}
    if kind == "direct":
        return {"kind": "sigma", "nocc": rng.randint(4, 10), "nvirt": _log_int(rng, 19, 110), "m": _log_int(rng, 1, 20),
                "precision": kind, "df": False}
    if kind == "cvs":
        return {"kind": "sigma", "nocc": rng.randint(5, 12), "nvirt": _log_int(rng, 19, 120), "m": _log_int(rng, 1, 20),
                "precision": kind, "df": False, "ncore": rng.randint(1, 4)}
    no, nv = rng.randint(4, 16), _log_int(rng, 19, 150)
    return {"kind": "sigma", "nocc": no, "nvirt": nv, "m": _log_int(rng, 1, 64), "precision": "mixed" if kind == "mixed" else "fp64",
            "df": kind == "df"}


# ---------------------------------------------------------------------------
# Inputs.
# ---------------------------------------------------------------------------
def _system(case, seed):
    """Orbital energies (host) and canonical packed integrals (device)."""
    no, nv = case["nocc"], case["nvirt"]
    nb = no + nv
    r = np.random.RandomState(seed % (1 << 32))
    e = np.concatenate([np.sort(r.uniform(-1.4, -0.4, no)), np.sort(r.uniform(0.1, 3.0, nv))])
    gen = torch.Generator(device="cuda").manual_seed(seed)
    npair = nb * (nb + 1) // 2
    p, q = torch.tril_indices(nb, nb, device="cuda")
    eri = torch.randn(npair * (npair + 1) // 2, generator=gen, device="cuda", dtype=torch.float64)
    row = 0
    while row < npair:      # rows pq of the packed triangle, about 2^25 values at a time
        end = row + 1
        while end < npair and (end + 1) * (end + 2) // 2 - row * (row + 1) // 2 <= 1 << 25:
            end += 1
        i0, i1 = row * (row + 1) // 2, end * (end + 1) // 2
        n = torch.arange(row + 1, end + 1, device="cuda")
        pq = torch.repeat_interleave(torch.arange(row, end, device="cuda"), n)
        rs = torch.arange(i0, i1, device="cuda") - pq * (pq + 1) // 2
        d = (p[pq] - p[rs]).abs() + (q[pq] - q[rs]).abs()
        eri[i0:i1] *= 0.3 * torch.exp(-0.15 * torch.arange(2 * nb, device="cuda", dtype=torch.float64))[d]
        row = end
    return e, eri


def _dim(case):
    no, nv = case["nocc"], case["nvirt"]
    if case.get("precision") == "cvs":
        return api.cvs_dim(no, nv, list(range(1, case["ncore"] + 1)))
    return api.adc2s_dim(no, nv)[0]


def _vectors(case, seed, ndim):
    """Unit columns whose amplitudes spread over three decades, as those of
    Ritz and Krylov vectors do."""
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    v = torch.randn(case["m"], ndim, generator=gen, device="cuda", dtype=torch.float64)
    v *= 10.0 ** (-3.0 * torch.rand(case["m"], ndim, generator=gen, device="cuda", dtype=torch.float64))
    v /= v.norm(dim=1, keepdim=True)
    return v.float() if case["precision"] == "mixed" else v


def _start_block(case, seed, ndim):
    return np.asfortranarray(np.random.RandomState((seed + 2) % (1 << 32)).random_sample((case["m"], ndim)).T)


def prepare(case, seed):
    e, eri = _system(case, seed)
    s = {"case": case, "e": e, "eri": eri.cpu().numpy()}
    g = s["g"] = api.AdcGpu(0)
    if case["kind"] == "build":
        return s
    g.set_orbitals(case["nocc"], case["nvirt"], e)
    g.set_eri_packed(s.pop("eri"))
    if case.get("precision") == "cvs":
        g.write_fspace_adc2_1_cvs(list(range(1, case["ncore"] + 1)))
    else:
        g.write_fspace_adc2_1(precision=PRECISION[case.get("precision", "fp64")])
    if case["kind"] == "sigma":
        if case["df"]:
            g.set_fp64_arith(1)
        s["v"] = _vectors(case, seed, g.ndim)
        s["w"] = torch.empty_like(s["v"])
    elif case["kind"] == "lanczos":
        s["q0"] = _start_block(case, seed, g.ndim)
    torch.cuda.synchronize()
    return s


def run(s):
    case, g = s["case"], s["g"]
    if case["kind"] == "sigma":
        g.sigma_device(case["m"], s["v"].data_ptr(), s["w"].data_ptr(), g.ndim)
        return s["w"]
    if case["kind"] == "build":
        g.set_orbitals(case["nocc"], case["nvirt"], s["e"])
        g.set_eri_packed(s["eri"])
        n = g.write_fspace_adc2_1(precision=PRECISION[case["precision"]])
        return {"noffdel": n, "diag": g.get_diag()}
    if case["kind"] == "lanczos":
        t, ev, _ = g.lancdiag_block(s["q0"], case["cycles"], orthotype=1)
        return {"t": t, "evals": ev}
    r = g.davdiag_block(case["roots"], 1e-6, maxiter=200, precision=PRECISION[case["precision"]], want_vectors=False)
    return {"evals": r.evals}


def work(case):
    """Kept couplings (each multiplied into both sides), the dense singles
    block and the vectors; a solver's products at the columns it cannot do
    without (one block a cycle; four blocks of the roots for a Davidson)."""
    no, nv = case["nocc"], case["nvirt"]
    n1, pv, po = no * nv, nv * (nv - 1) // 2, no * (no - 1) // 2
    if case.get("precision") == "cvs":
        nc = case["ncore"]
        pairs, n1 = nc * (no - nc), nc * nv
        nnz = pairs * (nv * (nc + nv - 1) + 2 * pv * (2 * nc + nv - 2))
        ndim = n1 + pairs * (nv + 2 * pv)
    else:
        ndim = n1 + no * nv + no * pv + po * nv + 2 * po * pv
        nnz = no * nv * (no + nv - 1) + no * pv * (2 * no + nv - 2) + po * nv * (no + 2 * nv - 2) + 2 * po * pv * (2 * no + 2 * nv - 4)
    val, vec = (2, 4) if case.get("precision") == "mixed" else (8, 8)
    matrix = val * nnz + 2 * val * n1 * n1 + vec * ndim

    def sigma(m):
        return {"bytes": matrix + 2 * vec * m * ndim, "flops": (4 * nnz + 2 * n1 * n1 + 2 * ndim) * m}

    if case["kind"] == "sigma":
        s = sigma(case["m"])
        if case["precision"] == "direct":       # integrals in, values never stored
            s["bytes"] = 8 * (nv * nv * no * nv + no ** 3 * nv + n1 * n1) + 8 * ndim + 16 * case["m"] * ndim
            s["flops"] += 4 * nnz
        return s
    nb = no + nv
    eri = (nb * (nb + 1) // 2) * (nb * (nb + 1) // 2 + 1) // 2
    if case["kind"] == "build":
        return {"bytes": 8 * eri + matrix + 8 * ndim, "flops": 4 * nnz + 2 * n1 ** 3}
    n = case["cycles"] if case["kind"] == "lanczos" else 4
    s = sigma(case["m"] if case["kind"] == "lanczos" else 2 * case["roots"])
    return {"bytes": n * s["bytes"], "flops": n * s["flops"]}


# ---------------------------------------------------------------------------
# The same outputs in 64 bits from the formulas of the method.
# ---------------------------------------------------------------------------
class _Exact:
    """The ADC(2)-s matrix of a system as blocks of integrals, torch FP64."""

    MINC = 1e-12

    def __init__(self, no, nv, e, eri):
        self.no, self.nv = no, nv
        o, v = torch.arange(no, device="cuda"), torch.arange(no, no + nv, device="cuda")

        def block(p, q, r, s):
            def pair(x, y):
                x, y = torch.broadcast_tensors(x[:, None], y[None, :])
                return torch.maximum(x, y) * (torch.maximum(x, y) + 1) // 2 + torch.minimum(x, y)

            b, a = torch.broadcast_tensors(pair(r, s)[None], pair(p, q)[:, :, None, None])
            return eri[torch.maximum(a, b) * (torch.maximum(a, b) + 1) // 2 + torch.minimum(a, b)]

        self.vvov = torch.stack([block(x[None], v, o, v)[0] for x in v])      # (a b|i c)
        self.ooov = block(o, o, o, v)                                          # (i j|k a)
        ovov, vvoo = block(o, v, o, v), block(v, v, o, o)
        e = torch.as_tensor(e, device="cuda")
        eo, ev = e[:no], e[no:]
        pa, pb = torch.triu_indices(nv, nv, 1, device="cuda")
        self.pa, self.pb = pa, pb
        n1 = no * nv
        vovo = ovov.permute(1, 0, 3, 2)                                        # (a i|b j)
        m = 2.0 * vovo - vvoo.permute(0, 2, 1, 3)                              # C1: [a,k,a1,k1]
        # second-order terms, each denominator the mean of its two one-sided forms
        g, g2 = vovo, vovo.permute(0, 3, 2, 1)                                 # (a u|r v), (a v|r u)
        den = eo[None, :, None, None] + eo[None, None, None, :] - ev[None, None, :, None] - ev[:, None, None, None]
        x, y = (g / den).reshape(nv, -1), (2 * g - g2).reshape(nv, -1)
        ca = -0.5 * (x @ y.T + g.reshape(nv, -1) @ ((2 * g - g2) / den).reshape(nv, -1).T)
        f = ovov.permute(0, 1, 3, 2)                                           # f[k,r,s,u] = (r k|s u)
        f2 = f.permute(0, 2, 1, 3)
        den = eo[None, None, None, :] - ev[None, :, None, None] - ev[None, None, :, None] + eo[:, None, None, None]
        cb = -0.5 * ((f / den).reshape(no, -1) @ (2 * f - f2).reshape(no, -1).T
                     + f.reshape(no, -1) @ ((2 * f - f2) / den).reshape(no, -1).T)
        t = (2.0 * vovo - g2).reshape(n1, n1)                                  # 2(ak|rs) - (as|rk) over [r,s]
        d = (eo[None, :] - ev[:, None]).reshape(-1)
        td = t / (d[:, None] + d[None, :])
        cc = 0.5 * (td @ t.T + t @ td.T)
        m = m.reshape(nv, no, nv, no).clone()
        m += ca[:, None, :, None] * torch.eye(no, device="cuda", dtype=m.dtype)[None, :, None, :]
        m += torch.eye(nv, device="cuda", dtype=m.dtype)[:, None, :, None] * cb[None, :, None, :]
        m = m.reshape(n1, n1) + cc
        dd = torch.diagonal(m)
        dd += -d
        diag = dd.clone()
        m[m.abs() <= self.MINC] = 0.0
        torch.diagonal(m).copy_(diag)
        self.h11 = m
        k, l = torch.triu_indices(no, no, 1, device="cuda")
        vv = ev[pa] + ev[pb]
        c4 = (vv[None, :] - (eo[k] + eo[l])[:, None]).reshape(-1)
        self.diag = torch.cat([diag, (2 * ev[None, :] - 2 * eo[:, None]).reshape(-1), (vv[:, None] - 2 * eo[None, :]).reshape(-1),
                               (2 * ev[None, :] - (eo[k] + eo[l])[:, None]).reshape(-1), c4, c4])
        self.ndim = self.diag.numel()

    def _cut(self, x):
        return torch.where(x.abs() <= self.MINC, 0.0, x)

    def _slab(self, k, l, kind):
        """(C, D, Y, Z) of the rows of hole pair (k, l): couplings to (a,k),
        (a,l), and to (a',kk), (b',kk) as tables over b' and a'."""
        o, pa, pb, n = self.ooov, self.pa, self.pb, self.nv
        ml, mk = self.vvov[:, :, l, :], self.vvov[:, :, k, :]
        s1, s2 = o[k, :, l, :].T, o[l, :, k, :].T                              # [virtual, kk]
        if kind in ("II", "I"):
            f, g = (2 ** -0.5, 1.0) if kind == "I" else ((3 / 2) ** 0.5, -1.0)
            c, d = f * (ml + g * ml.transpose(1, 2)), f * g * (mk + g * mk.transpose(1, 2))
            y, z = -f * (s1 + g * s2), -f * g * (s1 + g * s2)
        elif kind == "2":
            c, d = -(mk + mk.transpose(1, 2)), None
            y = z = s1
        elif kind == "3":
            c, d = torch.diagonal(ml, dim1=1, dim2=2), torch.diagonal(mk, dim1=1, dim2=2)
            y, z = -(s1 + s2), None
        else:
            c, d = -2 ** 0.5 * torch.diagonal(mk, dim1=1, dim2=2), None
            y, z = 2 ** 0.5 * s1, None
        two = z is not None
        ra = pa if two else torch.arange(n, device="cuda")
        rb = pb if two else ra
        rows = torch.arange(ra.numel(), device="cuda")
        out = []
        for t, h in ((c, k), (d, l)):
            if t is None:
                continue
            t = (t[:, pa, pb] if two else t).T.clone()
            t[rows, ra] += y[rb, h]
            if two:
                t[rows, rb] += z[ra, h]
            out.append((self._cut(t), h))
        keep = torch.ones(self.no, device="cuda", dtype=y.dtype)
        keep[k] = keep[l] = 0.0
        return out, self._cut(y) * keep, self._cut(z) * keep if two else None, ra, rb

    def rows(self):
        """(kind, k, l, store indices of the slab's rows) of every slab."""
        no, nv = self.no, self.nv
        n1, pv, po = no * nv, nv * (nv - 1) // 2, no * (no - 1) // 2
        s2, s3 = n1 + n1, n1 + n1 + no * pv
        s4 = s3 + po * nv
        for k in range(no):
            yield "1", k, k, n1 + k * nv + torch.arange(nv, device="cuda")
            yield "2", k, k, s2 + k + no * torch.arange(pv, device="cuda")
        p = 0
        for k in range(no):
            for l in range(k + 1, no):
                yield "3", k, l, s3 + p * nv + torch.arange(nv, device="cuda")
                yield "I", k, l, s4 + p * pv + torch.arange(pv, device="cuda")
                yield "II", k, l, s4 + (po + p) * pv + torch.arange(pv, device="cuda")
                p += 1

    def product(self, v):
        """H v for the rows of v (m x ndim)."""
        no, nv, m = self.no, self.nv, v.shape[0]
        n1 = no * nv
        w = v * self.diag
        h = self.h11.clone()
        torch.diagonal(h).zero_()
        w[:, :n1] += v[:, :n1] @ h
        x = v[:, :n1].reshape(m, nv, no)
        w1 = w[:, :n1].reshape(m, nv, no)
        for kind, k, l, at in self.rows():
            blocks, y, z, ra, rb = self._slab(k, l, kind)
            v2 = v[:, at]
            w2 = torch.zeros_like(v2)
            for t, hole in blocks:
                w2 += x[:, :, hole] @ t.T
                w1[:, :, hole] += v2 @ t
            if z is None:
                w2 += torch.einsum("mak,ak->ma", x, y)
                w1 += v2[:, :, None] * y[None]
            else:
                u = torch.zeros(m, nv, nv, device="cuda", dtype=v.dtype)
                u[:, ra, rb] = v2
                w2 += (x @ y.T)[:, ra, rb] + (x @ z.T).transpose(1, 2)[:, ra, rb]
                w1 += u @ y + u.transpose(1, 2) @ z
            w[:, at] += w2
        return w

    def cvs(self, ncore):
        """Indices of the CVS configurations in the full list."""
        no, nv = self.no, self.nv
        idx = [(torch.arange(nv, device="cuda")[:, None] * no + torch.arange(ncore, device="cuda")[None, :]).reshape(-1)]
        for want in ("3", "I", "II"):
            idx += [at for kind, k, l, at in self.rows() if kind == want and (k < ncore) != (l < ncore)]
        return torch.cat(idx)


def _lanczos(h, q0, cycles):
    """Block Lanczos with full orthogonalisation: T and its eigenvalues."""
    b = q0.shape[0]
    q = q0 / q0.norm(dim=1, keepdim=True)

    def ortho(x, basis):
        for y in basis:
            x = x - (x @ y.T) @ y
        return x

    def qr(x):
        r = torch.eye(b, device="cuda", dtype=x.dtype)
        for _ in range(2):
            c = torch.linalg.cholesky(x @ x.T)
            x, r = torch.linalg.solve_triangular(c, x, upper=False), c.T @ r
        return x, r

    q, _ = qr(q)
    basis, n = [], b * cycles
    t = torch.zeros(n, n, device="cuda", dtype=q.dtype)
    for j in range(cycles):
        basis.append(q)
        u = h(q)
        a = q @ u.T
        t[j * b:(j + 1) * b, j * b:(j + 1) * b] = a
        q, r = qr(ortho(ortho(u, basis), basis))
        if j + 1 < cycles:
            t[(j + 1) * b:(j + 2) * b, j * b:(j + 1) * b] = r
            t[j * b:(j + 1) * b, (j + 1) * b:(j + 2) * b] = r.T
    return t, torch.linalg.eigvalsh(t)


def exact(case, seed):
    no, nv = case["nocc"], case["nvirt"]
    if case["kind"] == "davidson" and _dim(case) > 8000:
        return None         # no dense diagonalisation of this size in the time
    e, eri = _system(case, seed)
    m = _Exact(no, nv, e, eri)
    if case["kind"] == "sigma":
        ndim = _dim(case)
        v = _vectors(case, seed, ndim).double()
        if case["precision"] != "cvs":
            return m.product(v)
        at = m.cvs(case["ncore"])
        full = torch.zeros(case["m"], m.ndim, device="cuda", dtype=torch.float64)
        full[:, at] = v
        return m.product(full)[:, at]
    if case["kind"] == "build":
        return {"noffdel": None, "diag": m.diag.cpu().numpy()}
    if case["kind"] == "lanczos":
        q0 = torch.from_numpy(np.ascontiguousarray(_start_block(case, seed, m.ndim).T)).cuda()
        t, ev = _lanczos(m.product, q0, case["cycles"])
        return {"t": t.cpu().numpy(), "evals": ev.cpu().numpy()}
    h = m.product(torch.eye(m.ndim, device="cuda", dtype=torch.float64))
    return {"evals": torch.linalg.eigvalsh(0.5 * (h + h.T))[:case["roots"]].cpu().numpy()}
