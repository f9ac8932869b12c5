"""Quadratures and exchange of at most 64 AOs, which run on narrow tiles, where
the tile, the ring and the sums have their edges: 1 to 65 AOs around the multiples
of 16 and 32 (65 takes the wide tiles), sums shorter than a stage, of one, of
several parts with a remainder, drains every and every fourth stage.

Tolerance of the quadratures: FP32-accurate products and sums, 1e-6 of the sum of
the absolute values of the terms.  Of the exchange, whose pairs and transforms are
FP32: a transform's error is within 20 eps of its norm and the pieces drop 2^-22,
2 (20 x 6e-8 + 2.4e-7) = 3e-6 of the largest diagonal element."""
import numpy as np
import pytest

from test_gpu_tc import _operands

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nao", [1, 15, 16, 17, 31, 32, 33, 48, 49, 63, 64, 65])
@pytest.mark.parametrize("N", [5, 32, 1000, 29791])
@pytest.mark.parametrize("drain", [1, 4])
def test_quadratures(nao, N, drain):
    import torch
    from hqc_gb300._lib import tc_quadrature
    phi, _, ld = _operands(nao, N, 100 + nao)
    w = torch.zeros(ld, dtype=torch.float32, device="cuda")
    w[:N] = torch.randn(N, device="cuda", generator=torch.Generator(device="cuda").manual_seed(5))
    M = tc_quadrature(phi, w, drain=drain)
    p64, w64 = phi[:, :N].double(), w[:N].double()
    terms = (p64.abs() * w64.abs()) @ p64.abs().T
    assert ((M - (p64 * w64) @ p64.T).abs() / terms).max() < 1e-6
    assert bool((M == M.T).all()) and bool((M == tc_quadrature(phi, w, drain=drain)).all())


@pytest.mark.parametrize("n,basis,grid", [(3, "gth-szv", 25), (8, "gth-dzv", 33), (17, "gth-szv", 31), (16, "gth-dzv", 27),
                                          (10, "gth-dzvp", 25), (32, "gth-dzv", 25), (33, "gth-dzv", 25)])
def test_exchange(n, basis, grid):
    import torch
    from hqc_gb300 import make_solver
    rng = np.random.default_rng(n)
    rs, L = 1.5, (4 * np.pi * n / 3) ** (1 / 3)
    sites = np.array(np.meshgrid(*[np.arange(4)] * 3)).reshape(3, -1).T[np.arange(n) * 64 // max(n, 1) % 64] * (L / 4)
    xp = sites + rng.normal(0, 0.05, (n, 3))
    s = make_solver(n, L, rs, basis, grid_length=L * rs / (grid - 0.5), max_cycle=2, precision="mixed", smearing=True,
                    smearing_sigma=0.05)
    s(xp)
    plan = s.plan
    q = lambda k: torch.as_tensor(plan.query(k), device="cuda").double()
    D = q("D")
    nao = int(round(D.numel() ** 0.5))
    D, K, St = D.reshape(nao, nao), q("K").reshape(nao, nao), q("St").reshape(nao, nao)
    ph = q("phi")
    phi = ph[: nao * (ph.numel() // nao)].reshape(nao, -1)[:, : grid ** 3].reshape(nao, grid, grid, grid)
    box = L * rs
    m = torch.fft.fftfreq(grid, 1.0 / grid, dtype=torch.float64, device="cuda") * (2 * np.pi / box)
    G2 = m[:, None, None] ** 2 + m[:, None] ** 2 + m ** 2
    coul = torch.where(G2 > 0, 4 * np.pi / G2.clamp_min(1e-9), 0.0)
    occ, U = torch.linalg.eigh(D)
    want = 4 * np.pi / box * 0.22578495 * St @ D @ St
    for i in range(nao):
        psi = torch.tensordot(U[:, i], phi, 1)
        P = (torch.fft.fftn(phi * psi, dim=(1, 2, 3)) * (coul / grid ** 3).sqrt()).reshape(nao, -1)
        want += occ[i] * (box / grid) ** 3 * (P @ P.conj().T).real
    assert (K - want).abs().max() <= 3e-6 * want.diagonal().abs().max()
