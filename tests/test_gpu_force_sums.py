"""The nuclear sums that do not touch the AO grid, at the atom counts and cut-offs
where their kernels change form: the structure-factor force term in groups of 10
atoms and passes of 40 (through the FP64 gradient against the oracle's), and the
Ewald energy and gradient with its table of Gaussians (|G|^2 <= 1023) and without.

Tolerances: gradient 1e-7 Ha/Bohr, as the other comparisons with the
oracle at SCF tol 1e-10; Ewald 1e-13 of the sum of the terms' absolute
values, some hundred eps for sums of up to 10^5 terms in blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 10, 12, 42])
def test_gradient_matches_oracle(n):
    from hqc_gb300 import make_solver
    from oracle.forces import electronic_gradient
    from oracle.gpw import Solver
    rng = np.random.default_rng(n)
    rs, L = 1.6, (4 * np.pi * n / 3) ** (1 / 3)
    m = 2 if n <= 4 else 3 if n <= 14 else 4
    sites = np.array(np.meshgrid(*[np.arange(m)] * 3)).reshape(3, -1).T[(np.arange(n) * m ** 3) // n] * (L / m)
    xp = sites + rng.normal(0, 0.04, (n, 3))
    kw = dict(dft=True, xc="lda,vwn", tol=1e-10, max_cycle=200, grid_length=0.45, smearing=True, smearing_sigma=0.05,
              search_method="newton", search_tol=1e-12)
    s = make_solver(n, L, rs, "gth-szv", forces=True, **kw)
    s(xp)
    got = s.plan.forces().cpu().numpy()
    ref = Solver(n, L, rs, "gth-szv", **kw)
    ref.solve(xp)
    assert np.abs(got - electronic_gradient(ref)).max() < 1e-7


@pytest.mark.parametrize("n,kappa,gmax", [(1, 10.0, 15), (2, 4.0, 31), (2, 4.0, 32), (11, 4.0, 31), (11, 4.0, 32),
                                          (11, 10.0, 3), (41, 10.0, 15)])
def test_ewald_matches_oracle(n, kappa, gmax):
    from hqc_gb300.potential import potential_energy_pp_and_grad
    from oracle.ewald import vpp
    rng = np.random.default_rng(10 * n + gmax)
    rs, L = 1.4, (4 * np.pi * n / 3) ** (1 / 3)
    x = rng.uniform(-L, 2 * L, (n, 3))
    e, g = potential_energy_pp_and_grad(x, L, rs, kappa, gmax)
    ref, gref = vpp(x, L, rs, kappa, gmax, grad=True)
    pairs = n * n / L / rs * 60.0  # kappa / sqrt(pi) and 1 / r of the closest pairs bound a term
    assert abs(float(e) - ref) <= 1e-13 * max(pairs, abs(ref))
    assert np.abs(g.cpu().numpy() - gref).max() <= 1e-13 * max(pairs * 100, np.abs(gref).max())
