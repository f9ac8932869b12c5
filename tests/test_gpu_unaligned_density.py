"""hqcgb_tc_orbital_density on arrays that start off 16 bytes, which TMA does not
take: they go through a copy (resident-Y form) or the transposition (more orbitals
or AOs), and the results are the aligned call's bit for bit, as the values, kernels
and order of the sums are the same."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nao,N,nuse,gga,off_phi,off_dphi", [
    (1, 129, 1, False, 1, 0), (20, 4097, 10, True, 1, 0), (20, 4097, 10, True, 0, 3), (33, 1000, 17, True, 2, 2),
    (288, 515, 32, True, 3, 1), (130, 4097, 64, False, 1, 0), (300, 515, 20, True, 1, 3)])
def test_unaligned_arrays_give_the_aligned_bits(nao, N, nuse, gga, off_phi, off_dphi):
    import torch
    from hqc_gb300._lib import tc_orbital_density
    g = torch.Generator(device="cuda").manual_seed(nao + N)
    ld = (N + 63) // 64 * 64

    def shifted(x, off):
        big = torch.empty(x.numel() + 4, dtype=x.dtype, device="cuda")
        y = big[off:off + x.numel()].view(x.shape)
        y.copy_(x)
        assert y.data_ptr() % 16 == 4 * off
        return y

    def rows(n):
        x = torch.zeros(n, ld, device="cuda")
        x[:, :N] = torch.randn(n, N, generator=g, device="cuda")
        return x

    phi, dphi = rows(nao), rows(3 * nao) if gga else None
    C = torch.randn(nao, nao, generator=g, dtype=torch.float64, device="cuda") / nao ** 0.5
    occ = torch.zeros(nao, dtype=torch.float64, device="cuda")
    occ[:nuse] = 2.0
    want = tc_orbital_density(phi, C, occ, N, nuse, dphi)
    got = tc_orbital_density(shifted(phi, off_phi), C, occ, N, nuse, shifted(dphi, off_dphi) if gga else None)
    for a, b in zip(want if gga else (want,), got if gga else (got,)):
        assert bool((a == b).all())
