"""Overlap and kinetic sums by rows of the lattice sphere against the plain
formula (products of 1D integrals, torch FP64): boxes whose sphere has one to
some ten thousand vectors, a cube instead of a sphere, a set that is not
symmetric (which takes the sums vector by vector), atoms far outside the box,
one atom, bases with and without p functions, Gamma and k-point.  The sums
vector by vector, which one vector moved by 1e-14 of its length selects, must
agree with the rows as well, to the rounding of their longer chains.

Tolerance: the rows round every term exp(-x) h to about (x + 4) eps of itself
(x exp(-x) < 0.4) and add a few dozen partial sums: 64 eps of the sum of the
absolute values of the terms, element by element (the elements themselves
cancel); one eps a vector more for sums in sequence.  Both forms leave out
images beyond exp(-60), below 1e-18 of any diagonal element: CUT."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CUT = 1e-18


def _overlap(basis, lat, xp, kpts):
    import torch
    from hqc_gb300 import _lib
    from hqc_gb300.basis import basis_tables
    lib = _lib.load()
    al, co, ls, ca = basis_tables(basis)
    lat = np.ascontiguousarray(lat)
    B, n, _ = xp.shape
    nao = n * co.shape[0]
    x = torch.tensor(xp, device="cuda")
    ty = torch.float64 if kpts is None else torch.complex128
    S = torch.zeros(B, nao, nao, dtype=ty, device="cuda")
    T = torch.zeros_like(S)
    d, i = lambda v: v.ctypes.data_as(_lib.c_double_p), lambda v: v.ctypes.data_as(_lib.c_int_p)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    _lib.check(lib.hqcgb_overlap(n, co.shape[0], al.size, d(al), d(co), i(ls), i(ca), lat.shape[0], d(lat), B, p(x),
                                 None if kpts is None else d(kpts), p(S), p(T),
                                 ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return S.cpu().numpy(), T.cpu().numpy()


def _set(kind, L, rcut):
    from hqc_gb300.solver import lattice_sphere
    if kind == "sphere":
        return lattice_sphere(L, rcut)
    m = np.arange(-2, 3) * L
    cube = np.array(np.meshgrid(m, m, m)).reshape(3, -1).T
    return cube if kind == "cube" else cube[cube[:, 0] >= 0]


def _plain(basis, lat, x, kpt, absolute):
    """S and T of one configuration x (n, 3), or the sums of their terms' absolute values."""
    import torch
    from hqc_gb300.basis import basis_tables
    al, co, ls, ca = basis_tables(basis)
    x, t = torch.tensor(x, device="cuda"), torch.tensor(np.ascontiguousarray(lat), device="cuda")
    u = x[:, None, None] - x[None, :, None] + t
    phase = 1.0 if kpt is None or absolute else torch.exp(-1j * (t @ torch.tensor(kpt, device="cuda")))
    mag, sgn = (torch.abs, 1) if absolute else (lambda v: v, -1)
    n, nb = x.shape[0], len(ls)
    S = torch.zeros(n, nb, n, nb, dtype=torch.float64 if kpt is None or absolute else torch.complex128, device="cuda")
    T = torch.zeros_like(S)
    for a in range(len(al)):
        for b in range(len(al)):
            p, c = al[a] + al[b], al[b]
            pa, pb = mag(-al[b] / p * u), mag(al[a] / p * u)
            one = torch.exp(-al[a] * al[b] / p * u * u) * np.sqrt(np.pi / p)
            I = {(0, 0): one, (1, 0): pa * one}
            for j in range(3):
                for i in (0, 1):
                    v = pb * I[i, j]
                    v = v + (j / (2 * p) * I[i, j - 1] if j else 0) + (i / (2 * p) * I[0, j] if i else 0)
                    I[i, j + 1] = v
            for k in range(nb):
                for q in range(nb):
                    w = co[k, a] * co[q, b]
                    w = abs(w) if absolute else w
                    if w == 0:
                        continue
                    lk = [int(ls[k] == 1 and ca[k] == d) for d in range(3)]
                    lq = [int(ls[q] == 1 and ca[q] == d) for d in range(3)]
                    o = [I[lk[d], lq[d]][..., d] for d in range(3)]
                    e = [((3 if lq[d] else 1) * c * I[lk[d], lq[d]] + sgn * 2 * c * c * I[lk[d], lq[d] + 2])[..., d]
                         for d in range(3)]
                    S[:, k, :, q] += w * (o[0] * o[1] * o[2] * phase).sum(-1)
                    T[:, k, :, q] += w * ((e[0] * o[1] * o[2] + o[0] * e[1] * o[2] + o[0] * o[1] * e[2]) * phase).sum(-1)
    return S.reshape(n * nb, n * nb).cpu().numpy(), T.reshape(n * nb, n * nb).cpu().numpy()


@pytest.mark.parametrize("basis", ["gth-szv", "gth-dzvp"])
@pytest.mark.parametrize("kind,L,rcut", [("sphere", 1.6, 24.0), ("sphere", 2.6, 18.0), ("sphere", 6.5, 24.0),
                                         ("sphere", 8.0, 18.0), ("sphere", 30.0, 24.0), ("cube", 5.0, 0.0),
                                         ("half", 5.0, 0.0)])
@pytest.mark.parametrize("kpoint", [False, True])
def test_rows_match_plain_sums(basis, kind, L, rcut, kpoint):
    rng = np.random.default_rng(int(100 * L))
    lat = _set(kind, L, rcut)
    moved = lat.copy()
    if len(lat) > 1:
        moved[np.argmax((lat ** 2).sum(1))] *= 1 + 1e-14
    else:
        moved = np.concatenate([lat, [[1e3, 0.0, 0.0]], [[0.0, 1.7e3, 0.0]]])  # vectors that add nothing
    for n in (1, 5):
        xp = rng.uniform(-0.5, 1.5, (2, n, 3)) * L
        kpts = rng.uniform(-np.pi / L, np.pi / L, (2, 3)) if kpoint else None
        new, old = _overlap(basis, lat, xp, kpts), _overlap(basis, moved, xp, kpts)
        for b in range(2):
            k = kpts[b] if kpoint else None
            for got, vec, want, terms in zip(new, old, _plain(basis, lat, xp[b], k, False),
                                             _plain(basis, lat, xp[b], k, True)):
                far = np.abs(got[b] - want) / (2.2e-16 * terms + CUT)
                assert far.max() <= 64 + (len(lat) if kind == "half" else 0)
                assert (np.abs(got[b] - vec[b]) / (2.2e-16 * terms + CUT)).max() <= 64 + len(lat)
