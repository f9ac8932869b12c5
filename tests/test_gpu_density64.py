"""The FP64 orbital density on the tensor cores against the sum over the
density matrix in torch FP64, at the edges of its tiles: AO counts around 8,
32 and 64, more than 64 orbitals (two column blocks), grids that end inside a
tile of 128 points, LDA, smeared and PBE runs; and beyond 512 AOs, where the
sum over D stays.

Tolerance: psi is exact to 2^-55 sqrt(n) of max|phi(g)| max|Y| a point and the
sum over D to n eps of the sum of its absolute terms, which bounds both:
64 n eps sum_pq |D_pq phi_p phi_q| with |D| = |C| f |C|^T."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,basis,grid,kw", [
    (2, "gth-szv", 9, {}), (8, "gth-szv", 25, {}), (14, "gth-dzv", 19, {}), (16, "gth-dzv", 21, {}),
    (14, "gth-dzvp", 17, dict(xc="pbe")), (8, "gth-dzvp", 25, dict(xc="pbe", kelvin=20000)),
    (34, "gth-dzv", 15, dict(kelvin=60000)), (66, "gth-szv", 15, dict(kelvin=200000)),
    (54, "gth-dzvp", 15, dict(xc="pbe")), (8, "gth-dzv", 15, dict(hf=True)), (104, "gth-dzvp", 9, {})])
def test_density_matches_density_matrix(n, basis, grid, kw):
    import torch
    from hqc_gb300 import make_solver
    from hqc_gb300.workloads import box
    L = box(n)
    rng = np.random.default_rng(n + grid)
    m = int(np.ceil(n ** (1 / 3)))
    sites = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] / m * L
    args = dict(n_grid=grid, max_cycle=0, diis=False, dft=not kw.get("hf"), xc=kw.get("xc", "lda,vwn"))
    if "kelvin" in kw:
        args.update(smearing=True, smearing_method="fermi", smearing_sigma=0.5 * kw["kelvin"] / 157888.09,
                    search_method="newton")
    s = make_solver(n, L, 1.4, basis, **args)
    out = s(sites + rng.uniform(-0.1, 0.1, (n, 3)))
    nao, N = s.plan.nao, grid ** 3
    phi = s.plan.query("phi").reshape(nao, N)
    rho = s.plan.query("rho")
    C, D = out[0], out[1]
    want = (phi * (D @ phi)).sum(0)
    d = torch.diagonal(torch.linalg.solve(C, D) @ torch.linalg.inv(C).T).clamp(min=0)  # occupations of D = C f C^T
    terms = (phi.abs() * (((C.abs() * d) @ C.abs().T) @ phi.abs())).sum(0)
    assert ((rho - want).abs() <= 64 * nao * 2.2e-16 * terms).all()
    assert float((rho - want).norm() / want.norm()) < 1e-12
