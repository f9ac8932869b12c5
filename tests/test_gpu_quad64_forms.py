"""The FP64 quadratures' forms against plain sums.

Elements: AOs far apart, whose products are small next to the largest element,
keep the accuracy of an FP64 sum of their own terms.  An AO's values are held to
2^-57 of twice its largest in a brick of at most 8 points a side, on either side;
where the brick's |w phi_p phi_q| sum to 1/256 of its points times the maxima at
least (two p Gaussians of exponent 0.73, 5 Bohr apart, in a brick 1.4 Bohr wide:
1/160) and every point errs the same way, that is 64 eps of the sum of absolute
terms.  The reference's own rounding (products, pairwise sums): 36 eps.

PBE: the Fock matrix's two-electron part (J + V_xc) of the density the engine
returns, against the oracle's quadratures of it: rho and grad rho agree to some
1e-13 of their largest values, PBE's potentials pass that on with factors of order
ten, and the sum is 1e-14 itself: 1e-11 of the norm.

Exchange on grids beyond the fused kernels (FP64: planes of 119 points), where the
pair form contracts two operands: as test_gpu_exchange_planes.py."""
import numpy as np
import pytest
from test_gpu_exchange_planes import test_exchange_matrix as _exchange_matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,basis,box,grid", [(3, "gth-szv", 12.0, 47), (5, "gth-dzvp", 10.0, 57),
                                              (4, "gth-dzvp", 14.0, 81), (14, "gth-dzvp", 9.0, 51)])
def test_small_elements_keep_their_digits(n, basis, box, grid):
    import torch
    from hqc_gb300 import make_solver
    rng = np.random.default_rng(n)
    s = make_solver(n, box / 1.4, 1.4, basis, n_grid=grid, max_cycle=0, diis=False)
    s(rng.uniform(0, box / 1.4, (n, 3)))
    nao, N = s.plan.nao, grid ** 3
    phi = s.plan.query("phi").reshape(nao, N)
    dV = box ** 3 / N
    for name, w in (("V", s.plan.query("vloc")), ("St", torch.ones(N, dtype=torch.float64, device="cuda"))):
        M = s.plan.query(name).reshape(nao, nao)
        want, terms = torch.zeros_like(M), torch.zeros_like(M)
        for p in range(nao):
            t = phi * (phi[p] * w)
            want[p], terms[p] = dV * t.sum(1), dV * t.abs().sum(1)
        seen = terms > 1e-10 * terms.max()
        assert bool(((M - want).abs() <= 100 * 2.2e-16 * terms)[seen].all())


@pytest.mark.parametrize("n,basis,grid", [(2, "gth-szv", 15), (8, "gth-szv", 17), (13, "gth-dzvp", 17),
                                          (32, "gth-dzv", 21), (26, "gth-dzvp", 15), (54, "gth-dzvp", 15)])
def test_pbe_fock_matrix_matches_the_oracle(n, basis, grid):
    from hqc_gb300 import make_solver
    from hqc_gb300.workloads import box
    from oracle.gpw import Solver
    L = box(n)
    m = int(np.ceil(n ** (1 / 3)))
    sites = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] / m * L
    xp = sites + np.random.default_rng(n).uniform(-0.1, 0.1, (n, 3))
    s = make_solver(n, L, 1.4, basis, dft=True, xc="pbe", n_grid=grid, max_cycle=0, diis=False)
    D = s(xp)[1].cpu().numpy()
    F2e = s.plan.query("J").cpu().numpy().reshape(D.shape)
    o = Solver(n, L, 1.4, basis, dft=True, xc="pbe", n_grid=grid)
    g = o.setup_geometry(xp)
    rho, _, _ = o.density(D, g["phi"])
    want = o.hartree(rho, g["phi"])[0] + o.xc_terms(D, g["phi"], g["grad"])[1]
    assert np.linalg.norm(F2e - want) <= 1e-11 * np.linalg.norm(want)


@pytest.mark.parametrize("precision,tol,grid", [("fp64", None, 119), ("mixed", 3e-6, 169)])
def test_exchange_of_large_grids(precision, tol, grid):
    _exchange_matrix(precision, tol, 2, "gth-szv", grid, 0.0)
