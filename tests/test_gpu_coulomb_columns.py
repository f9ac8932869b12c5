"""The column form of the walkers' reciprocal sums (hqcgb_coulomb_energy)
against the pairwise oracle where it can go wrong: G lists that are not
spheres (duplicates, one of a pair G, -G, single vectors, the largest index
of the phase tables and one beyond it, which takes the general kernel), both
dimensions, particle counts around the chunk of 32, few and many walkers
(runs of 2 and of 8).  Tolerance as for the spheres: 1e-10, FP64 sums of up
to 1e4 terms of order one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lists(dim, kind, rng):
    from hqc_gb300 import kpoints
    if kind == "sphere":
        return kpoints(dim, 7)
    if kind == "random":
        G = rng.integers(-6, 7, (60, dim))
        return G[(G ** 2).sum(1) > 0]
    if kind == "edge":
        return np.concatenate([np.eye(dim, dtype=int) * 31, -np.eye(dim, dtype=int) * 31, np.ones((1, dim), int)])
    if kind == "beyond":
        return np.concatenate([np.eye(dim, dtype=int) * 32, kpoints(dim, 4)])
    return np.concatenate([kpoints(dim, 3), kpoints(dim, 3)[:5], -kpoints(dim, 3)[7:9]])  # duplicates


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("kind", ["sphere", "random", "edge", "beyond", "twice"])
@pytest.mark.parametrize("n,B", [(1, 3), (31, 2), (33, 5), (14, 700)])
def test_column_sums_match_oracle(dim, kind, n, B):
    from hqc_gb300 import potential_energy
    from oracle.ewald import potential_energy as ref
    rng = np.random.default_rng(n + B + dim)
    L, rs = 4.7, 1.3
    x = rng.uniform(-L, 2 * L, (B, 2 * n, dim))
    G = _lists(dim, kind, rng)
    out = [v.cpu().numpy() for v in potential_energy(x, 1.5, G, L, rs)]
    some = slice(0, 2)
    want = ref(x[some], 1.5, G, L, rs)
    for v, r in zip(out, want):
        np.testing.assert_allclose(v[some], r, rtol=1e-10, atol=1e-10)


def test_non_finite_positions_stay_visible():
    from hqc_gb300 import kpoints, potential_energy
    x = np.random.default_rng(0).uniform(0, 3, (2, 8, 3))
    x[1, 2, 0] = np.nan
    out = [v.cpu().numpy() for v in potential_energy(x, 5.0, kpoints(3, 5), 3.0, 1.4)]
    assert all(np.isfinite(v[0]) for v in out) and np.isnan(out[0][1])
