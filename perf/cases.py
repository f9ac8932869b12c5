"""Performance cases of hqc_gb300: what its users have it compute, through its public entry points.

Whole calculations at the sizes of the test suite and the benchmark
configurations, and the blocks they share:

* SCFs at fixed protons (``make_solver``, double precision: the default);
* energy and gradient (``make_pes(..., forces=True)``), double precision;
* energy and gradient in mixed precision through the torch autograd wrapper
  (``pes_energy``), one configuration and concurrent batches, with float32
  positions as a sampler or a molecular-dynamics driver on the GPU holds them
  (the wrapper returns what the positions are: float32);
* a k-point mesh;
* Slater matrices, Coulomb energies and overlap matrices of walker batches;
* the tensor-core grid contractions on their own (orbital density with its
  gradient, GGA Fock quadrature).

Protons are those of a compressed liquid (uniformly random positions put
protons on top of one another, where an SCF need not converge), and runs
without smearing take the atom counts that fill a shell of plane waves
(8, 14, 38, 54), as periodic hydrogen is simulated.  Smeared runs use the
Newton search for the chemical potential: bisection at its default tolerance
leaves occupations that step with the last digits of the Fock matrix.  Orbital coefficients are left out of the outputs: eigenvectors are
defined up to a sign, the density matrix is not.
"""
import numpy as np
import torch

import hqc_gb300 as hqc
from hqc_gb300 import _lib
from hqc_gb300.basis import basis_tables

NAO = {"gth-szv": 1, "gth-dzv": 2, "gth-dzvp": 5}  # AOs per hydrogen
KELVIN = 0.5 / 157888.09  # Hartree, as the smearing widths of the benchmark workloads
TYPICAL_CYCLES = 15  # SCF iterations of a converged run with the default DIIS settings


def listed():
    return [
        # the smallest everyday run: eight atoms, minimal basis, exact exchange; launches and latency count
        dict(name="scf h8 szv hf 41", kind="scf", n=8, rs=1.25, basis="gth-szv", dft=False, xc="", kelvin=0, grid=41),
        # a smeared LDA run of the middle size in the default precision
        dict(name="scf h32 dzv lda 65", kind="scf", n=32, rs=1.4, basis="gth-dzv", dft=True, xc="lda,vwn",
             kelvin=10000, grid=65),
        # energy and forces in double precision with the polarised basis: the reference for mixed runs
        dict(name="forces h14 dzvp pbe 49", kind="forces", n=14, rs=1.4, basis="gth-dzvp", dft=True, xc="pbe",
             kelvin=0, grid=49),
        # one step of molecular dynamics: the H54 PBE benchmark system, one configuration at a time
        dict(name="md h54 dzvp pbe 81", kind="mixed", n=54, rs=1.31, basis="gth-dzvp", dft=True, xc="pbe", kelvin=0,
             grid=81, batch=1),
        # a sampler's batch: eight concurrent configurations of the middle size
        dict(name="batch8 h38 dzvp pbe 65", kind="mixed", n=38, rs=1.31, basis="gth-dzvp", dft=True, xc="pbe",
             kelvin=0, grid=65, batch=8),
        # smeared Hartree-Fock energies and forces, a concurrent batch (the exchange build)
        dict(name="batch4 h14 dzv hf 49", kind="mixed", n=14, rs=1.4, basis="gth-dzv", dft=False, xc="", kelvin=5000,
             grid=49, batch=4),
        # two k-points of a mesh, double precision, exact exchange
        dict(name="kmesh2 h8 dzv hf 33", kind="kpt", n=8, rs=1.4, basis="gth-dzv", dft=False, xc="", kelvin=10000,
             grid=33, batch=2),
        # Slater matrices of a variational Monte Carlo walker batch
        dict(name="slater h54 dzvp 2048", kind="slater", n=54, rs=1.31, basis="gth-dzvp", walkers=2048, kpoint=False),
        # Coulomb energies of the walkers of one such step
        dict(name="coulomb h54 1024", kind="coulomb", n=54, rs=1.31, gmax=15, walkers=1024),
        # overlap and kinetic matrices of a batch of configurations
        dict(name="overlap h54 dzvp 16", kind="overlap", n=54, rs=1.31, basis="gth-dzvp", batch=16, kpoint=False),
        # the mixed path's grid contractions at the H54 sizes: density with its gradient ...
        dict(name="density 270x81 occ27", kind="density", nao=270, grid=81, occ=27),
        # ... and the GGA Fock quadrature
        dict(name="quadrature 270x81", kind="quadrature", nao=270, grid=81),
    ]


def draw(rng):
    """One more case of the same ranges: atom counts up to the listed ones, odd grids, densities, bases,
    functionals, smearing and batch sizes."""
    def odd(lo, hi):
        return rng.randrange(lo // 2, hi // 2 + 1) * 2 + 1 if lo < hi else lo

    def log(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    rs = round(rng.uniform(1.25, 1.6), 3)
    kind = rng.choice(["scf", "scf", "forces", "mixed", "mixed", "kpt", "slater", "coulomb", "overlap", "density",
                       "quadrature"])
    if kind in ("scf", "forces"):
        dft, kelvin = rng.random() < 0.6, rng.choice([0, 5000, 10000])
        if kelvin:
            n, basis = rng.choice([(4, "gth-dzvp"), (8, "gth-szv"), (8, "gth-dzvp"), (16, "gth-dzv"),
                                   (16, "gth-szv"), (32, "gth-szv")])
        else:
            n, basis = rng.choice([(8, "gth-szv"), (8, "gth-dzvp"), (14, "gth-dzv"), (14, "gth-dzvp")])
        xc = rng.choice(["lda,vwn", "lda,hl", "pbe"]) if dft else ""
        top = 41 if kind == "forces" or not dft else 49
        return dict(kind=kind, n=n, rs=rs, basis=basis, dft=dft, xc=xc, kelvin=kelvin, grid=odd(25, top))
    if kind == "mixed":
        n, lo, hi, most = rng.choice([(8, 31, 49, 8), (14, 39, 57, 8), (38, 49, 65, 6), (54, 65, 81, 1)])
        if n <= 14 and rng.random() < 0.4:
            return dict(kind=kind, n=n, rs=rs, basis="gth-dzv", dft=False, xc="", kelvin=5000, grid=odd(31, 49),
                        batch=rng.randrange(1, 5))
        return dict(kind=kind, n=n, rs=rs, basis="gth-dzvp", dft=True, xc=rng.choice(["pbe", "pbe", "lda,vwn"]),
                    kelvin=0, grid=odd(lo, hi), batch=rng.randrange(1, most + 1))
    if kind == "kpt":
        dft = rng.random() < 0.5
        return dict(kind=kind, n=rng.choice([4, 8]), rs=rs, basis="gth-dzv", dft=dft, xc="lda,vwn" if dft else "",
                    kelvin=10000, grid=odd(21, 33), batch=rng.choice([1, 2]))
    if kind == "slater":
        return dict(kind=kind, n=rng.choice([8, 14, 16, 32, 54]), rs=rs, basis=rng.choice(["gth-dzv", "gth-dzvp"]),
                    walkers=log(4, 2048), kpoint=rng.random() < 0.3)
    if kind == "coulomb":
        return dict(kind=kind, n=rng.choice([8, 14, 16, 32, 54]), rs=rs, gmax=rng.choice([9, 12, 15]),
                    walkers=log(4, 1024))
    if kind == "overlap":
        return dict(kind=kind, n=rng.choice([4, 8, 14, 16, 32, 54]), rs=rs,
                    basis=rng.choice(["gth-szv", "gth-dzv", "gth-dzvp"]), batch=log(1, 16), kpoint=rng.random() < 0.3)
    nao = rng.randrange(16, 271)
    if kind == "density":
        return dict(kind=kind, nao=nao, grid=odd(33, 81), occ=rng.randrange(2, max(3, min(32, nao // 2)) + 1))
    return dict(kind=kind, nao=nao, grid=odd(33, 81))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _box(n):
    return (4.0 / 3.0 * np.pi * n) ** (1.0 / 3.0)


def _protons(n, rng, batch=None):
    """Protons of a compressed liquid, in rs units: random positions moved apart by a soft pair repulsion until
    neighbours are about one lattice spacing away."""
    L = _box(n)
    x = rng.uniform(0, L, (1 if batch is None else batch, n, 3))
    for _ in range(200):
        d = x[:, :, None] - x[:, None]
        d -= L * np.round(d / L)
        r2 = (d ** 2).sum(-1)
        x = x + 0.25 * (d * np.exp(-r2 / 1.2 ** 2)[..., None]).sum(2)
    x = x % L
    return x[0] if batch is None else x


def _electrons(xp, L, walkers, rng):
    """Walkers' electrons: one near each proton, at the distances of the 1s density."""
    return (xp + rng.normal(0.0, 0.7, (walkers,) + xp.shape)) % L


def _method(case):
    kw = dict(dft=case["dft"], n_grid=case["grid"])
    if case["dft"]:
        kw["xc"] = case["xc"]
    if case["kelvin"]:
        kw.update(smearing=True, smearing_method="fermi", smearing_sigma=KELVIN * case["kelvin"],
                  search_method="newton")
    return kw


def _on_grid(case, seed, derivatives):
    """AO-like functions on a periodic grid, float32, rows padded to a multiple of 64: s and p Gaussians of the
    basis' exponents on random centres of a box with the H54 system's grid spacing; with their gradients."""
    rng = np.random.default_rng(seed)
    ng, nao = case["grid"], case["nao"]
    N, h = ng ** 3, 0.129
    ld = (N + 63) // 64 * 64
    dev = torch.device("cuda")
    alpha = torch.tensor(rng.choice([8.374, 1.806, 0.4530, 0.1658, 0.727], nao), dtype=torch.float64, device=dev)
    power = torch.tensor(rng.integers(-2, 3, nao), device=dev)  # < 0: an s function, 0..2: p along that axis
    centre = torch.tensor(rng.uniform(0, ng * h, (nao, 3)), dtype=torch.float64, device=dev)
    x = torch.arange(ng, dtype=torch.float64, device=dev) * h
    norm = (2 * alpha / np.pi) ** 0.75
    f, df = [], []
    for d in range(3):
        u = x[None] - centre[:, d:d + 1]
        u = u - ng * h * torch.round(u / (ng * h))
        g = torch.exp(-alpha[:, None] * u * u)
        p = (power == d)[:, None]
        f.append(torch.where(p, u * g, g).float())
        df.append(torch.where(p, (1 - 2 * alpha[:, None] * u * u) * g, -2 * alpha[:, None] * u * g).float())
    f[0], df[0] = f[0] * norm[:, None].float(), df[0] * norm[:, None].float()

    def product(a, b, c):
        out = torch.zeros(nao, ld, dtype=torch.float32, device=dev)
        out[:, :N] = (a[:, :, None, None] * b[:, None, :, None] * c[:, None, None, :]).reshape(nao, N)
        return out

    phi = product(*f)
    if not derivatives:
        return phi, None, N, rng
    dphi = torch.cat([product(df[0], f[1], f[2]), product(f[0], df[1], f[2]), product(f[0], f[1], df[2])])
    return phi, dphi, N, rng


def prepare(case, seed):
    kind, rng = case["kind"], np.random.default_rng(seed)
    s = dict(case=case)
    if kind in ("density", "quadrature"):
        phi, dphi, N, rng = _on_grid(case, seed, True)
        s.update(phi=phi, dphi=dphi, N=N)
        nao, ld = phi.shape
        if kind == "density":
            C = np.linalg.qr(rng.normal(size=(nao, nao)))[0]
            occ = np.zeros(nao)
            occ[:case["occ"]] = 2.0
            s.update(C=torch.tensor(C, device="cuda"), occ=torch.tensor(occ, device="cuda"))
        else:
            gen = torch.Generator(device="cuda").manual_seed(seed)
            # the xc + Hartree potential times the volume element, and 2 v_sigma grad rho
            w = torch.zeros(ld, dtype=torch.float32, device="cuda")
            w[:N] = (torch.rand(N, generator=gen, device="cuda") - 0.6) * 0.129 ** 3
            u = torch.zeros(3, ld, dtype=torch.float32, device="cuda")
            u[:, :N] = torch.randn(3, N, generator=gen, device="cuda") * 0.02
            s.update(w=w, u=u, dV=0.129 ** 3)
        return s
    n, rs = case["n"], case["rs"]
    L = _box(n)
    if kind == "scf":
        s.update(solver=hqc.make_solver(n, L, rs, case["basis"], **_method(case)),
                 xp=torch.tensor(_protons(n, rng), device="cuda"))
    elif kind == "forces":
        s.update(pes=hqc.make_pes(n, L, rs, case["basis"], forces=True, **_method(case)),
                 xp=torch.tensor(_protons(n, rng), device="cuda"))
    elif kind == "mixed":
        B = case["batch"]
        s.update(pes=hqc.make_pes(n, L, rs, case["basis"], forces=True, precision="mixed", concurrency=B,
                                  **_method(case)),
                 xp=torch.tensor(_protons(n, rng, B if B > 1 else None), dtype=torch.float32, device="cuda",
                                 requires_grad=True))
    elif kind == "kpt":
        s.update(solver=hqc.make_solver(n, L, rs, case["basis"], gamma=False, **_method(case)),
                 xp=torch.tensor(_protons(n, rng), device="cuda"),
                 # points of the 2x2x2 Monkhorst-Pack mesh, one of each pair k, -k
                 kpts=np.pi / (2 * L * rs) * np.array([[1, 1, 1], [1, 1, -1], [1, -1, 1], [-1, 1, 1]])[
                     rng.permutation(4)[:case["batch"]]])
    elif kind == "slater":
        xp = _protons(n, rng)
        nao = n * NAO[case["basis"]]
        mo = np.linalg.qr(rng.normal(size=(nao, nao)))[0]
        if case["kpoint"]:
            mo = np.linalg.qr(rng.normal(size=(nao, nao)) + 1j * rng.normal(size=(nao, nao)))[0]
        s.update(slater=hqc.make_slater(n, L, rs, case["basis"], gamma=not case["kpoint"]),
                 xp=torch.tensor(xp, device="cuda"), mo=torch.tensor(mo, device="cuda"),
                 xe=torch.tensor(_electrons(xp, L, case["walkers"], rng), device="cuda"),
                 kpt=rng.uniform(-np.pi / (L * rs), np.pi / (L * rs), 3))
    elif kind == "coulomb":
        xp = _protons(n, rng)
        xe = _electrons(xp, L, case["walkers"], rng)
        x = np.concatenate([np.broadcast_to(xp, xe.shape), xe], axis=1)
        s.update(x=torch.tensor(x, device="cuda"), G=hqc.kpoints(3, case["gmax"]), L=L, kappa=10.0)
    elif kind == "overlap":
        s.update(overlap=hqc.make_overlap(n, L, rs, case["basis"], gamma=not case["kpoint"]),
                 xp=torch.tensor(_protons(n, rng, case["batch"]), device="cuda"),
                 kpts=rng.uniform(-np.pi / (L * rs), np.pi / (L * rs), (case["batch"], 3)))
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "scf":
        _, dm, bands, E, Ki, Vep, Vee, Se, conv = s["solver"](s["xp"])
        return dict(dm=dm, bands=bands, E=E, Ki=Ki, Vep=Vep, Vee=Vee, Se=Se, converged=conv)
    if kind == "forces":
        F, g = s["pes"].value_and_grad(s["xp"])
        return dict(F=F, grad=g)
    if kind == "mixed":
        E = hqc.pes_energy(s["xp"], s["pes"])
        (g,) = torch.autograd.grad(E.sum(), s["xp"])
        return dict(F=E, grad=g)
    if kind == "kpt":
        _, dm, bands, E, Ki, Vep, Vee, Se, conv = s["solver"](s["xp"], s["kpts"])
        return dict(dm=dm, bands=bands, E=E, Ki=Ki, Vep=Vep, Vee=Vee, Se=Se, converged=conv)
    if kind == "slater":
        args = (s["xp"], s["xe"], s["mo"]) + ((s["kpt"],) if case["kpoint"] else ())
        up, dn = s["slater"](*args)
        return dict(up=up, dn=dn)
    if kind == "coulomb":
        vpp, vep, vee = hqc.potential_energy(s["x"], s["kappa"], s["G"], s["L"], case["rs"])
        return dict(vpp=vpp, vep=vep, vee=vee)
    if kind == "overlap":
        S, T = s["overlap"].with_kinetic(*((s["xp"], s["kpts"]) if case["kpoint"] else (s["xp"],)))
        return dict(S=S, T=T)
    if kind == "density":
        rho, grad = _lib.tc_orbital_density(s["phi"], s["C"], s["occ"], s["N"], case["occ"], s["dphi"], drain=2)
        return dict(rho=rho, grad=grad)
    return dict(M=_lib.tc_quadrature_gga(s["phi"], s["dphi"], s["w"], s["u"], s["dV"], s["N"], drain=4))


def work(case):
    kind = case["kind"]
    if kind in ("density", "quadrature"):
        nao, N = case["nao"], case["grid"] ** 3
        if kind == "density":  # four fields of the orbitals from the four AO fields
            return dict(bytes=4 * nao * N * 4 + 4 * N * 8, flops=2.0 * 4 * nao * case["occ"] * N)
        return dict(bytes=4 * nao * N * 4 + 4 * N * 4 + nao * nao * 8, flops=2.0 * nao * nao * N)
    n = case["n"]
    if kind == "slater":
        W, nao, c = case["walkers"], n * NAO[case["basis"]], 2 if case["kpoint"] else 1
        return dict(bytes=8.0 * (W * n * 3 + c * nao * n + c * W * n * n / 2),
                    flops=W * n * (2.0 * c * c * nao * n / 2 + n * 3 * 5 * 20 * c))
    if kind == "coulomb":
        # half of the sphere of G vectors, one complex multiply-add a particle and vector
        W, nG = case["walkers"], 4.0 / 3.0 * np.pi * case["gmax"] ** 3 / 2
        return dict(bytes=8.0 * W * (2 * n * 3 + 3), flops=W * (8.0 * 2 * n * nG + 40.0 * (2 * n) ** 2 / 2))
    if kind == "overlap":
        nao, c = n * NAO[case["basis"]], 2 if case["kpoint"] else 1
        # each pair of primitives of each pair of atoms (a triangle of them) over the lattice terms that matter
        return dict(bytes=8.0 * case["batch"] * (3 * n + 2 * c * nao * nao),
                    flops=case["batch"] * n * n / 2 * 15 * 30 * 60.0 * c)
    # an SCF: per iteration the occupied orbitals and half of the Fock matrix on the grid, at least
    nao, N = n * NAO[case["basis"]], case["grid"] ** 3
    fields = 4 if case["xc"] == "pbe" else 1
    c = 4 if kind == "kpt" else 1
    occ = n // 2 if not case["kelvin"] else min(nao, n)
    flops = c * (2.0 * fields * nao * occ + 1.0 * nao * nao * (2 if fields == 4 else 1)) * N * TYPICAL_CYCLES
    if not case["dft"]:  # one transform a pair of an AO and an orbital
        flops += c * nao * occ * N * 2.5 * np.log2(N) * TYPICAL_CYCLES
    B = case.get("batch", 1)
    out = 3 * n + 1 if kind in ("forces", "mixed") else 2 * nao * nao
    return dict(bytes=B * 8.0 * (3 * n + out), flops=float(B * flops))


# ---------------------------------------------------------------------------
# what the outputs are, in 64 bits (where they are sums: an SCF's fixed point has no plain formula)
# ---------------------------------------------------------------------------
def _lattice(L, rcut=24.0):
    t = np.arange(-(rcut // L), rcut // L + 1) * L
    T = np.stack(np.meshgrid(t, t, t, indexing="ij"), -1).reshape(-1, 3)
    return t, T[(T ** 2).sum(1) <= rcut ** 2]


def _exact_slater(s):
    case = s["case"]
    n, rs = case["n"], case["rs"]
    alpha, coef, ls, carts = [torch.tensor(np.asarray(v), device="cuda") for v in basis_tables(case["basis"])]
    t = torch.tensor(_lattice(_box(n) * rs)[0], device="cuda")
    xp, xe = s["xp"] * rs, s["xe"] * rs
    ups, dns = [], []
    for chunk in xe.split(max(1, 400_000 // (n * n))):
        u = chunk[:, :, None, :, None] - xp[None, None, :, :, None] - t  # walker, electron, atom, axis, image
        phase = torch.exp(1j * torch.tensor(s["kpt"], device="cuda")[:, None] * t) if case["kpoint"] else 1.0
        f = []
        for l in (0, 1):
            cols = []
            for a in alpha:
                cols.append((u ** l * torch.exp(-a * u * u) * phase).sum(-1))
            f.append(torch.stack(cols, -1))  # walker, electron, atom, axis, primitive
        ao = []
        for k in range(len(ls)):
            prod = 1.0
            for d in range(3):
                prod = prod * f[1 if int(ls[k]) == 1 and int(carts[k]) == d else 0][..., d, :]
            ao.append((prod * coef[k]).sum(-1))
        ao = torch.stack(ao, -1).flatten(2)
        ups.append(ao[:, :n // 2] @ s["mo"][:, :n // 2])
        dns.append(ao[:, n // 2:] @ s["mo"][:, :n // 2])
    return dict(up=torch.cat(ups), dn=torch.cat(dns))


def _exact_coulomb(s):
    x, L, kappa = s["x"] / s["L"], s["L"], s["kappa"]
    G = torch.tensor(np.asarray(s["G"]), dtype=torch.float64, device="cuda")
    G = G[(G[:, 0] > 0) | ((G[:, 0] == 0) & ((G[:, 1] > 0) | ((G[:, 1] == 0) & (G[:, 2] > 0))))]  # one of G, -G
    G2 = (G ** 2).sum(1)
    gk = 2 * torch.exp(-np.pi ** 2 * G2 / kappa ** 2) / (np.pi * G2)
    n = x.shape[1] // 2
    g0 = -np.pi / kappa ** 2
    out = []
    for c in x.split(32):
        r = c[:, :, None] - c[:, None, :]
        r = r - torch.round(r)
        d = r.norm(dim=-1) + torch.eye(2 * n, device=c.device, dtype=c.dtype)
        v = torch.special.erfc(kappa * d) / d
        tri = torch.triu(torch.ones(n, n, device=c.device, dtype=c.dtype), 1)
        ph = 2 * np.pi * torch.remainder(c @ G.T, 1.0)
        ph = torch.polar(torch.ones_like(ph), ph)
        sp, se = ph[:, :n].sum(1), ph[:, n:].sum(1)
        pp = (v[:, :n, :n] * tri).sum((1, 2)) + (gk * 0.5 * (sp.abs() ** 2 - n)).sum(1) + 0.5 * n * (n - 1) * g0
        ee = (v[:, n:, n:] * tri).sum((1, 2)) + (gk * 0.5 * (se.abs() ** 2 - n)).sum(1) + 0.5 * n * (n - 1) * g0
        pe = v[:, :n, n:].sum((1, 2)) + (gk * (sp * se.conj()).real).sum(1) + n * n * g0
        out.append(torch.stack([pp, -pe, ee]))
    out = torch.cat(out, 1) * (2 * s["case"]["rs"] / L)
    return dict(vpp=out[0], vep=out[1], vee=out[2])


def _exact_overlap(s):
    case = s["case"]
    n, rs = case["n"], case["rs"]
    alpha, coef, ls, carts = [np.asarray(v) for v in basis_tables(case["basis"])]
    T = torch.tensor(_lattice(_box(n) * rs)[1], device="cuda")
    nb = len(ls)
    Ss, Ts = [], []
    for b in range(case["batch"]):
        xp = s["xp"][b] * rs
        ty = torch.complex128 if case["kpoint"] else torch.float64
        S = torch.zeros(n, nb, n, nb, dtype=ty, device="cuda")
        K = torch.zeros_like(S)
        u = xp[:, None, None, :] - xp[None, :, None, :] + T  # R_i - R_j + t
        phase = torch.exp(-1j * (T @ torch.tensor(s["kpts"][b], device="cuda"))) if case["kpoint"] else 1.0
        for ia, a in enumerate(alpha):
            for ib, c in enumerate(alpha):
                p = a + c
                pa, pb = -c / p * u, a / p * u  # product centre minus either centre
                one = torch.exp(-a * c / p * u * u) * np.sqrt(np.pi / p)
                I = {(0, 0): one, (1, 0): pa * one}
                for j in range(3):
                    for i in (0, 1):
                        v = pb * I[i, j]
                        if j:
                            v = v + j / (2 * p) * I[i, j - 1]
                        if i:
                            v = v + i / (2 * p) * I[0, j]
                        I[i, j + 1] = v
                for k in range(nb):
                    for q in range(nb):
                        w = coef[k, ia] * coef[q, ib]
                        if w == 0.0:
                            continue
                        lk = [int(ls[k] == 1 and carts[k] == d) for d in range(3)]
                        lq = [int(ls[q] == 1 and carts[q] == d) for d in range(3)]
                        o = [I[lk[d], lq[d]][..., d] for d in range(3)]
                        # -1/2 d2/dx2 of x^l exp(-c x^2)
                        t = [((3 if lq[d] else 1) * c * I[lk[d], lq[d]] - 2 * c * c * I[lk[d], lq[d] + 2])[..., d]
                             for d in range(3)]
                        S[:, k, :, q] += w * (o[0] * o[1] * o[2] * phase).sum(-1)
                        K[:, k, :, q] += w * ((t[0] * o[1] * o[2] + o[0] * t[1] * o[2] + o[0] * o[1] * t[2])
                                              * phase).sum(-1)
        Ss.append(S.reshape(n * nb, n * nb))
        Ts.append(K.reshape(n * nb, n * nb))
    return dict(S=torch.stack(Ss), T=torch.stack(Ts))


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("slater", "coulomb", "overlap", "density", "quadrature"):
        return None
    s = prepare(case, seed)
    if kind == "slater":
        return _exact_slater(s)
    if kind == "coulomb":
        return _exact_coulomb(s)
    if kind == "overlap":
        return _exact_overlap(s)
    nao, N = case["nao"], s["N"]
    phi = s["phi"][:, :N].double()
    if kind == "density":
        Y = s["C"][:, :case["occ"]] * s["occ"][:case["occ"]].sqrt()
        psi = Y.T @ phi
        grad = [2 * (psi * (Y.T @ s["dphi"][d * nao:(d + 1) * nao, :N].double())).sum(0) for d in range(3)]
        return dict(rho=(psi ** 2).sum(0), grad=torch.stack(grad))
    Z = 0.5 * s["w"][:N].double() * phi
    for d in range(3):
        Z += s["dV"] * s["u"][d, :N].double() * s["dphi"][d * nao:(d + 1) * nao, :N].double()
    M = Z @ phi.T
    return dict(M=M + M.T)
