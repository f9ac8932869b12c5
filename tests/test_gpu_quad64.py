"""The FP64 quadrature on the tensor cores (digits of 7 bits) at the edges of
its tiles: AO counts around 8, 16, 64, 128 and 256 rows, grids whose point
count is no multiple of a stage, a chain or a maxima block, with a weight (V)
and without (S~), against torch FP64 products of the same AO grid.

Tolerance, elementwise: a digit string ends 2^-57 of 2^e, e at most two above
the row's largest element, on either side, and products below 2^-56 of
2^(eA + eB) are left out: N 2^-50 max|w phi_p| max|phi_q| dV bounds the sum if
every point errs the same way.  The errors are independent, so the Frobenius
norm of the whole must be near FP64 rounding: 1e-14 (an FP64 product of N terms
is allowed sqrt(N) eps = 3e-14 at these N)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,basis,grid", [
    (2, "gth-szv", 3), (2, "gth-szv", 15), (8, "gth-szv", 25), (10, "gth-szv", 21), (16, "gth-szv", 17),
    (14, "gth-dzvp", 19), (32, "gth-dzv", 25), (66, "gth-szv", 15), (126, "gth-szv", 15), (64, "gth-dzv", 15),
    (130, "gth-szv", 15), (26, "gth-dzvp", 15), (54, "gth-dzvp", 21), (200, "gth-szv", 15)])
def test_weighted_products_match_fp64(n, basis, grid):
    from hqc_gb300 import make_solver
    from hqc_gb300.workloads import box
    L = box(n)
    rng = np.random.default_rng(n + grid)
    m = int(np.ceil(n ** (1 / 3)))  # spread out: the geometry alone is of interest
    sites = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] / m * L
    xp = sites + rng.uniform(-0.1, 0.1, (n, 3))
    s = make_solver(n, L, 1.4, basis, n_grid=grid, max_cycle=0, diis=False)
    s(xp)
    nao = s.plan.nao
    N = grid ** 3
    phi = s.plan.query("phi").reshape(nao, N)
    vloc = s.plan.query("vloc")
    dV = (L * 1.4) ** 3 / N
    for name, w in (("V", vloc), ("St", None)):
        M = s.plan.query(name).reshape(nao, nao)
        A = phi if w is None else phi * w
        want = dV * (A @ phi.T)
        top = A.abs().amax(1) if w is None else phi.abs().amax(1) * w.abs().max()
        bound = N * 2.0 ** -50 * dV * top[:, None] * phi.abs().amax(1)[None]
        assert ((M - want).abs() <= bound).all()
        assert float((M - want).norm() / want.norm()) < 1e-14
        assert bool((M == M.T).all())
