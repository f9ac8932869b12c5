"""The FP64 k-point plan's grid contractions and exchange against plain torch
complex128 of the same formulas (K and the Madelung term from the density
matrix, V and S~ from the AO grid), where the tiles of 16 AOs and the grids'
factors have their edges: 16 AOs (the fewest that take the tiles), 20, 32 and 36;
grids 21 = 3 x 7, 23 and 31 (primes), 25 and 33 (fixed factors), 27 = 3 x 9 and
51 = 3 x 17 (a factor above 16), 35 = 5 x 7; both sides of the 16.

Tolerance: a transform of n points errs by at most 3 n eps of its norm and a sum of N
products in parts by some hundred eps of the sum of their absolute values, on
either side: (12 n + 2000) eps of the largest diagonal element."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.2e-16


@pytest.mark.parametrize("n,basis,grid", [(8, "gth-dzv", 21), (8, "gth-dzv", 23), (8, "gth-dzv", 27), (10, "gth-dzv", 25),
                                          (16, "gth-dzv", 33), (18, "gth-dzv", 35), (4, "gth-dzvp", 51),
                                          (16, "gth-szv", 31), (14, "gth-szv", 31)])
def test_exchange_and_quadratures(n, basis, grid):
    import torch
    from hqc_gb300 import make_solver
    rng = np.random.default_rng(n + grid)
    rs, L = 1.5, (4 * np.pi * n / 3) ** (1 / 3)
    edge = np.arange(8).reshape(-1, 1) >> np.arange(3) & 1
    sites = np.vstack([edge, edge + [0.5, 0.25, 0.25], edge + [0.25, 0.25, 0.75]])[:n] * (L / 2)
    xp = sites + rng.normal(0, 0.05, (n, 3))
    s = make_solver(n, L, rs, basis, gamma=False, grid_length=L * rs / (grid - 0.5), max_cycle=3)
    s(xp, rng.uniform(-np.pi / L / rs, np.pi / L / rs, 3))
    q = lambda k: torch.as_tensor(s.plan.query(k), device="cuda")
    z = lambda k: torch.view_as_complex(q(k).reshape(-1, 2).contiguous())
    D = z("D")
    nao = int(round(D.numel() ** 0.5))
    D, K, V, St = (t.reshape(nao, nao) for t in (D, z("K"), z("V"), z("St")))
    phi = z("phi").reshape(nao, grid, grid, grid)
    vloc, rho, vh = (q(k).reshape(grid, grid, grid) for k in ("vloc", "rho", "vh"))
    box = L * rs
    dV = (box / grid) ** 3
    m = torch.fft.fftfreq(grid, 1.0 / grid, dtype=torch.float64, device="cuda") * (2 * np.pi / box)
    G2 = m[:, None, None] ** 2 + m[:, None] ** 2 + m ** 2
    coul = torch.where(G2 > 0, 4 * np.pi / G2.clamp_min(1e-9), 0.0)
    f = phi.reshape(nao, -1)
    tol = (12 * grid + 2000) * EPS

    def close(got, want):
        assert (got - want).abs().max() <= tol * want.diagonal().abs().max()

    close(V, dV * (f * vloc.reshape(-1)) @ f.conj().T)
    close(St, dV * f @ f.conj().T)
    close(St, St.conj().T)
    want = torch.fft.ifftn(coul * torch.fft.fftn(rho)).real
    assert (vh - want).abs().max() <= tol * want.abs().max()
    occ, U = torch.linalg.eigh(D)
    pair = torch.zeros_like(K)
    for i in range(nao):
        psi = (U[:, i].conj() @ f).reshape(grid, grid, grid)
        P = torch.fft.fftn(phi * psi.conj(), dim=(1, 2, 3)) * (coul / grid ** 3).sqrt()
        P = P.reshape(nao, -1)
        pair += occ[i] * dV * P @ P.conj().T
    want = pair + 4 * np.pi / box * 0.22578495 * St @ D @ St
    close(K, want)
