"""The FP64 path's refined eigensolver inside the SCF, where its spectra are
awkward: below and above the size it starts at (12 AOs), a liquid's bands, a
perfect lattice's degenerate ones and nearly degenerate ones.  The orbitals
must be S-orthonormal and diagonalise nothing but what the FP64 solver would:
F C = S C diag(bands).

Tolerance: a backward-stable solve of the orthogonalised problem leaves
C^T S C - 1 and C^T F C - diag(bands) at n eps cond(S) (of the largest band);
100 times that bounds the constants of both factors."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _positions(kind, n, L, seed):
    from hqc_gb300.workloads import bcc
    if kind == "liquid":
        rng = np.random.default_rng(seed)
        x = rng.uniform(0, L, (n, 3))
        for _ in range(200):
            d = x[:, None] - x[None]
            d -= L * np.round(d / L)
            x = x + 0.25 * (d * np.exp(-(d ** 2).sum(-1) / 1.44)[..., None]).sum(1)
        return x % L
    return bcc(round((n / 2) ** (1 / 3)), 1.4, {"perfect": 0.0, "nearly": 1e-6, "warm": 0.05}[kind], seed)


@pytest.mark.parametrize("kind,n,basis,grid", [
    ("liquid", 10, "gth-szv", 25), ("liquid", 12, "gth-szv", 25), ("liquid", 14, "gth-dzvp", 25),
    ("liquid", 32, "gth-dzv", 31), ("perfect", 16, "gth-szv", 25), ("perfect", 16, "gth-dzvp", 25),
    ("nearly", 16, "gth-dzvp", 25), ("warm", 16, "gth-dzvp", 25), ("perfect", 54, "gth-dzvp", 27)])
def test_orbitals_solve_the_generalised_problem(kind, n, basis, grid):
    import torch
    from hqc_gb300 import make_solver
    from hqc_gb300.workloads import box
    L = box(n)
    s = make_solver(n, L, 1.4, basis, dft=True, n_grid=grid, max_cycle=0, diis=False)
    out = s(_positions(kind, n, L, 3))  # no cycles: the orbitals are the core Hamiltonian's
    C, w = out[0], out[2] / 2
    nao = C.shape[0]
    S, H = [s.plan.query(k).reshape(nao, nao) for k in ("S", "H")]
    S, H = 0.5 * (S + S.T), 0.5 * (H + H.T)
    sw = torch.linalg.eigvalsh(S.cpu())
    tol = 100 * nao * 2.2e-16 * float(sw[-1] / sw[0])
    top = max(1.0, float(w.abs().max()))
    one = torch.eye(nao, dtype=torch.float64, device="cuda")
    assert (C.T @ S @ C - one).abs().max() < tol
    assert (C.T @ H @ C - torch.diag(w)).abs().max() < tol * top
    assert bool((w[1:] >= w[:-1]).all())
