"""Device memory of plans, and the forms that FP64 plans take to stay within it.

A plan holds its AO grids, the vectors of the grid and what a product forms at a
time; the bound leaves a quarter of the AO grids for the latter.  An FP64 plan keeps
the digits of its AOs for a geometry only within a limit that it shares with its batch
workers; whether it does changes no bit of a result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _used():
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, total = torch.cuda.mem_get_info()
    return total - free


def _solver(n, grid, basis="gth-dzvp", **kw):
    from hqc_gb300 import make_solver
    from hqc_gb300.workloads import box
    return make_solver(n, box(n), 1.4, basis, n_grid=grid, **kw)


# bytes a value of an AO on the grid: phi, grad phi, D phi and the GGA force's two operands in FP64;
# phi, grad phi and the two pieces of phi and of the quadrature's operand in FP32, and bytes a
# point of the orbitals and their gradients that mixed forces keep (64 of them)
@pytest.mark.parametrize("precision,value_bytes,point_bytes", [("fp64", 7 * 8, 0), ("mixed", 8 * 4, 4 * 64 * 4)])
def test_a_plan_holds_little_more_than_its_grids(precision, value_bytes, point_bytes):
    n, grid = 54, 61
    before = _used()
    s = _solver(n, grid, dft=True, xc="pbe", forces=True, precision=precision)
    held = _used() - before
    assert held <= 1.25 * grid ** 3 * (s.plan.nao * value_bytes + point_bytes)


# four workers: the digits of the first plan are kept, those of the others do not fit the limit any more
@pytest.mark.parametrize("n,basis,grid,kw", [
    (14, "gth-dzvp", 49, dict(xc="pbe", forces=True)),
    (32, "gth-dzv", 65, dict(smearing=True, smearing_sigma=0.02, search_method="newton"))])
def test_kept_digits_change_no_bit(n, basis, grid, kw):
    import torch
    from hqc_gb300.workloads import box
    m = int(np.ceil(n ** (1 / 3)))
    sites = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] / m * box(n)
    xp = sites + np.random.default_rng(n).uniform(-0.1, 0.1, (n, 3))
    s = _solver(n, grid, basis, dft=True, max_cycle=2, concurrency=4, **kw)
    batch = torch.tensor(np.broadcast_to(xp, (8,) + xp.shape).copy(), device="cuda")
    one = s(batch[0])
    for t, b in zip(one[1:4], s(batch)[1:4]):
        assert bool((b == t).all())
