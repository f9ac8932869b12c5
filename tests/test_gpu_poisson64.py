"""The FP64 Hartree potential (half spectrum, paired transforms) against numpy's
FFT of the same density on the grid sizes where its transforms differ: primes
(direct sums), the fixed two-factor sizes, composite sizes through the generic
routine, sizes whose columns do not fill a chunk of 8, and an even size (the
complex passes).  Tolerance: three transforms forth and back of length n round
each term to a few eps and the Coulomb kernel weights them alike: 1e-13 of the
largest value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [3, 5, 9, 15, 21, 24, 25, 27, 31, 33, 35, 41, 45, 49, 51, 65, 81])
def test_hartree_potential_matches_numpy(grid):
    from hqc_gb300 import make_solver
    from hqc_gb300.workloads import box
    n, rs = 4, 1.4
    L = box(n)
    x = np.array([[0, 0, 0], [.5, .5, 0], [.5, 0, .5], [0, .5, .5]]) * L + np.random.default_rng(grid).normal(0, .05, (4, 3))
    s = make_solver(n, L, rs, "gth-dzv", dft=True, n_grid=grid, max_cycle=2, diis=False)
    s(x)
    rho = s.plan.query("rho").cpu().numpy().reshape((grid,) * 3)
    vh = s.plan.query("vh").cpu().numpy().reshape((grid,) * 3)
    m = np.where(np.arange(grid) <= grid // 2, np.arange(grid), np.arange(grid) - grid) * 2 * np.pi / (L * rs)
    G2 = m[:, None, None] ** 2 + m[None, :, None] ** 2 + m[None, None] ** 2
    k = np.where(G2 > 0, 4 * np.pi / np.where(G2 > 0, G2, 1.0), 0.0)
    want = np.fft.ifftn(k * np.fft.fftn(rho)).real
    assert np.abs(vh - want).max() < 1e-13 * np.abs(want).max()
