"""Rounding of AO values: against the image sums in extended precision at the same
electron-proton differences.

A value takes about twelve roundings in a row (the exponential's table entry and its
last multiply-add, the three axes' factors, coefficient, the sum over primitives and
over other images), each 2^-53 / sqrt(3) of its value at the worst mantissa and 0.72 of
that on average: sqrt(12) 4.6e-17 = 1.6e-16 of the values' norm.  At a k-point the phases and the two
products of a complex part make it half as many again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _exact(xp, xe, a, basis, kpt, rcut=24.0):
    from hqc_gb300.basis import basis_tables
    ld = np.longdouble
    alpha, coef, ls, carts = [np.asarray(v) for v in basis_tables(basis)]
    t = np.arange(-(rcut // a), rcut // a + 1) * a
    u = (xe[:, None, :] - xp[None])[..., None].astype(ld) - t.astype(ld)
    phase = 1
    if kpt is not None:
        arg = kpt[:, None].astype(ld) * t.astype(ld)
        phase = np.cos(arg) + 1j * np.sin(arg)
    f = [[(u ** l * np.exp(-ld(x) * u * u) * phase).sum(-1) for x in alpha] for l in (0, 1)]
    out = []
    for k in range(len(ls)):
        v = 0
        for q in range(len(alpha)):
            w = ld(coef[k, q])
            for d in range(3):
                w = w * f[1 if ls[k] == 1 and carts[k] == d else 0][q][..., d]
            v = v + w
        out.append(v)
    return np.stack(out, -1).reshape(xe.shape[0], -1)


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="no extended precision here")
@pytest.mark.parametrize("n,rs,basis", [(8, 1.4, "gth-dzv"), (14, 1.6, "gth-dzvp"), (32, 1.25, "gth-szv")])
@pytest.mark.parametrize("k", [None, (0.21, -0.13, 0.34)])
def test_ao_values_round_like_a_chain_of_twelve(n, rs, basis, k):
    from hqc_gb300 import make_slater
    from hqc_gb300.workloads import box
    rng = np.random.default_rng(n)
    L = box(n)
    xp, xe = rng.uniform(0, L, (n, 3)), rng.uniform(0, L, (100, 3))
    kpt = None if k is None else np.array(k) / L
    got = make_slater(n, L, rs, basis, gamma=k is None).ao_values(xp, xe, kpt).cpu().numpy()
    want = _exact(xp * rs, xe * rs, L * rs, basis, kpt)
    bound = 1.6e-16 if k is None else 1.6e-16 * 1.5 ** 0.5
    assert np.sqrt((abs(got - want) ** 2).sum() / (abs(want) ** 2).sum()) <= bound
