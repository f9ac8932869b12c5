"""The Hartree-Fock plan's exchange matrix against plain torch FP64 of the same sum
where the plane kernel changes form: grids whose shared field fits beside the plane
buffers (several orbitals a block) and grids where it does not, one, few and many
orbitals, FP32 and FP64.

Tolerance: FP64 a transform errs by at most 3 n eps of its norm and the sum by some
hundred eps, on either side: (12 n + 2000) eps of the largest diagonal element.
Mixed: FP32 pairs and transforms within 20 eps of their norm, pieces to 2^-22:
2 (20 x 6e-8 + 2.4e-7) = 3e-6 of it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp64", None), ("mixed", 3e-6)])
@pytest.mark.parametrize("n,basis,grid,sigma", [(2, "gth-szv", 21, 0.0), (3, "gth-dzv", 41, 0.3), (6, "gth-dzvp", 49, 0.3),
                                                (20, "gth-dzv", 27, 0.05), (3, "gth-dzv", 57, 0.3),
                                                (3, "gth-dzv", 69, 0.3), (2, "gth-szv", 81, 0.3)])
def test_exchange_matrix(precision, tol, n, basis, grid, sigma):
    import torch
    from hqc_gb300 import make_solver
    rng = np.random.default_rng(n + grid)
    rs, L = 1.5, (4 * np.pi * n / 3) ** (1 / 3)
    sites = np.array(np.meshgrid(*[np.arange(3)] * 3)).reshape(3, -1).T[(np.arange(n) * 27) // n] * (L / 3)
    s = make_solver(n, L, rs, basis, grid_length=L * rs / (grid - 0.5), max_cycle=2, precision=precision,
                    smearing=sigma > 0, smearing_sigma=sigma)
    s(sites + rng.normal(0, 0.05, (n, 3)))
    q = lambda k: torch.as_tensor(s.plan.query(k), device="cuda").double()
    D = q("D")
    nao = int(round(D.numel() ** 0.5))
    D, K, St = D.reshape(nao, nao), q("K").reshape(nao, nao), q("St").reshape(nao, nao)
    phi = q("phi").reshape(nao, grid, grid, grid)
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
    bound = (12 * grid + 2000) * 2.2e-16 if tol is None else tol
    assert (K - want).abs().max() <= bound * want.diagonal().abs().max()
