"""The FP64 orbital density where a CTA takes several tiles of 128 points (more than
152 of them): every role goes on to the next tile, field and column block in step.
Bounds and references of test_gpu_density64.py (rho) and test_gpu_quad64_forms.py (the
PBE Fock matrix, which reads the gradient)."""
import pytest
from test_gpu_density64 import test_density_matches_density_matrix as _density
from test_gpu_quad64_forms import test_pbe_fock_matrix_matches_the_oracle as _fock

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,basis,grid,kw", [
    (2, "gth-szv", 29, {}), (9, "gth-dzv", 39, {}), (14, "gth-dzvp", 35, dict(xc="pbe")),
    (66, "gth-szv", 29, dict(xc="pbe", kelvin=200000)), (34, "gth-dzv", 31, dict(kelvin=60000)),
    (54, "gth-dzvp", 35, dict(xc="pbe"))])
def test_density_of_several_tiles(n, basis, grid, kw):
    _density(n, basis, grid, kw)


@pytest.mark.parametrize("n,basis,grid", [(8, "gth-dzvp", 33), (26, "gth-szv", 31), (13, "gth-dzvp", 35)])
def test_gradient_of_several_tiles(n, basis, grid):
    _fock(n, basis, grid)
