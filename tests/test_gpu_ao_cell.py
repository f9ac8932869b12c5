"""AO values through the images of a box (one exponential a primitive for the
nearest image, ratios for the others) against the plain image sums, which the
same images in another order select: bases of 1 to 13 AOs an atom, boxes with
1 to 37 images an axis, electrons far outside the box, Gamma and k-point.

Tolerance: the exponents are at most 41 below the nearest image's, so each
form is within 41 eps and a few roundings of the sum: 1e-13 of the largest
value."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ao(basis, lat, xp, xe, kpt):
    import torch
    from hqc_gb300 import _lib
    from hqc_gb300.basis import basis_tables
    lib = _lib.load()
    al, co, ls, ca = basis_tables(basis)
    lat = np.ascontiguousarray(lat)
    n, npts = xp.shape[0], xe.shape[0]
    x, e = torch.tensor(xp, device="cuda"), torch.tensor(xe, device="cuda")
    out = torch.zeros(npts, n * co.shape[0], 1 if kpt is None else 2, dtype=torch.float64, device="cuda")
    d, i = lambda v: v.ctypes.data_as(_lib.c_double_p), lambda v: v.ctypes.data_as(_lib.c_int_p)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    head = (n, co.shape[0], al.size, d(al), d(co), i(ls), i(ca), lat.size, d(lat))
    tail = (p(x), npts, npts, p(e), p(out), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    if kpt is None:
        _lib.check(lib.hqcgb_ao_points(*head, *tail))
    else:
        _lib.check(lib.hqcgb_ao_points_kpt(*head, d(kpt), *tail))
    return out.cpu().numpy()


@pytest.mark.parametrize("basis", ["gth-szv", "gth-dzv", "gth-dzvp", "gth-tzvp", "gth-qzv3p"])
@pytest.mark.parametrize("L", [1.3, 3.0, 8.0, 30.0])
@pytest.mark.parametrize("kpoint", [False, True])
def test_box_images_match_image_sums(basis, L, kpoint):
    rng = np.random.default_rng(int(10 * L))
    tm = 24.0 // L
    lat = np.arange(-tm, tm + 1) * L
    xp = rng.uniform(0, L, (5, 3))
    xe = np.concatenate([rng.uniform(-0.5, 1.5, (40, 3)) * L, rng.uniform(-40, 40, (20, 3)), xp,
                         xp + 0.5 * L, xp - 1e-9])
    kpt = rng.uniform(-np.pi / L, np.pi / L, 3) if kpoint else None
    got = _ao(basis, lat, xp, xe, kpt)
    want = _ao(basis, np.concatenate([lat[1:], lat[:1]]) if lat.size > 1 else np.array([0.0, 1e6]), xp, xe, kpt)
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-13 * np.abs(want).max())
