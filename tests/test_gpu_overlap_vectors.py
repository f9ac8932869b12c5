"""Overlap and kinetic sums over lists of lattice vectors that are no sphere, at
the lengths where the warps' queue of 32 vectors is empty, full or has a
remainder, some of the vectors too far to add anything, against the plain
formula (torch FP64), Gamma and k-point.

Tolerance: every term is rounded to a few eps of itself and the sums run in
sequence: 64 + (number of vectors) eps of the sum of the terms' absolute values."""
import numpy as np
import pytest

from test_gpu_overlap_rows import CUT, _overlap, _plain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("basis", ["gth-szv", "gth-dzvp"])
@pytest.mark.parametrize("nvec", [1, 2, 31, 32, 33, 63, 64, 65, 97, 200])
@pytest.mark.parametrize("kpoint", [False, True])
def test_vector_lists(basis, nvec, kpoint):
    rng = np.random.default_rng(nvec)
    lat = np.vstack([np.zeros((1, 3)), rng.uniform(-6.0, 6.0, (nvec - 1, 3))])
    lat[rng.random(nvec) < 0.3] *= 40.0  # queued in their order around far ones
    for n in (1, 3):
        xp = rng.uniform(0.0, 4.0, (1, n, 3))
        kpts = rng.uniform(-0.5, 0.5, (1, 3)) if kpoint else None
        k = kpts[0] if kpoint else None
        for got, want, terms in zip(_overlap(basis, lat, xp, kpts), _plain(basis, lat, xp[0], k, False),
                                    _plain(basis, lat, xp[0], k, True)):
            assert (np.abs(got[0] - want) / (2.2e-16 * terms + CUT)).max() <= 64 + nvec
