"""Performance cases of the RGF library: the calls its users make, over the
sizes they make them at.

Kinds of case (``kind``):

* ``dropin``   one ``green_RGF_RS`` call on host arrays, as a Fortran energy
  loop makes it: one energy, the reference's output set;
* ``solve``    one batched ``Context.solve_energies`` over the energies of a
  device, ballistic, with scattering self-energies, or with overlap blocks
  (``green_RGF_CMS``), for the output set the caller asks for;
* ``w``        the screened interaction of one q-point (``w_solve_energies``);
* ``gw``       polarization and self-energy of the GW loop, direct sums;
* ``gwfft``    the same by FFT on one rank's slice of (i, j) elements;
* ``adjoint``  transmission and its potential derivatives (``adjoint_energies``).

Devices are nearly periodic chains, as the nanowires and nanotubes of the
reference's drivers are: one Hermitian block and one coupling block repeated
(``uniform coupling``), a linear potential drop between the contacts and weak
on-site disorder.  The broadening is 5 meV in the device and the leads, 10 meV
where derivatives are taken: Sancho-Rubio decimation amplifies rounding by the
inverse square of it, and at these values FP64 results are determined to
better than 1e-9 whatever the order of the sums.
"""
import math

import numpy as np
import torch

from liteqt_b200 import rgf

BOLTZ = rgf.BOLTZ_RGF_RS
MU = (0.2, -0.2)                       # contact chemical potentials, eV
TEMP = (0.025 / BOLTZ, 0.025 / BOLTZ)  # kT = 25 meV
PI = 3.14159265359                     # the reference's constant (green_rgf.f90:23)
ETA = 5e-3                             # broadening, eV
ETA_ADJOINT = 1e-2

# Output sets: the density loop's, the one with the hole density that the GW
# loop reads, and the reference routine's own.
OUTPUTS = {
    "density": ("ldos", "ndens"),
    "gw": ("ldos", "ndens", "pdens"),
    "full": ("ldos", "ndens", "pdens", "GRi1", "cur"),
}


def listed():
    return [
        # a Fortran loop's single call on a small nanotube cell (32 orbitals)
        dict(name="dropin_one_energy", kind="dropin", nm=32, nx=20),
        # the plain FP64 chain: 1000 energies of a small device
        dict(name="solve_nm32_nx50", kind="solve", nm=32, nx=50, nen=1000, outputs="density", scattering=False,
             overlap=False),
        # G of a GW iteration: scattering self-energies in, G^R, G^<, G^> out
        dict(name="solve_nm64_scattering", kind="solve", nm=64, nx=40, nen=256, outputs="gw", scattering=True,
             overlap=False),
        # the benchmark's workload: one wave of energies of a large device
        dict(name="solve_nm128_nx100", kind="solve", nm=128, nx=100, nen=296, outputs="density", scattering=False,
             overlap=False),
        # a few energies of a large device: one rank's share of a wide run, or
        # the points that an adaptive grid adds
        dict(name="solve_nm128_few", kind="solve", nm=128, nx=40, nen=12, outputs="full", scattering=False,
             overlap=False),
        # a block size that is no power of two
        dict(name="solve_nm104_nx30", kind="solve", nm=104, nx=30, nen=200, outputs="full", scattering=False,
             overlap=False),
        # a non-orthogonal basis with scattering
        dict(name="solve_nm72_overlap", kind="solve", nm=72, nx=30, nen=150, outputs="gw", scattering=True,
             overlap=True),
        # the largest block size
        dict(name="solve_nm256_nx30", kind="solve", nm=256, nx=30, nen=148, outputs="density", scattering=False,
             overlap=False),
        # W of a GW iteration, one q-point
        dict(name="w_nm64_nx40", kind="w", nm=64, nx=40, nen=256),
        # the GW loop's direct convolutions
        dict(name="gw_direct_nen512", kind="gw", nm=16, nx=10, nen=512, nky=2, nkz=2, ndiag=3, imag_only=True),
        # the production loop's FFT convolutions on one rank's slice
        dict(name="gw_fft_nen4096", kind="gwfft", nm=64, nx=10, nen=4096, nky=4, nkz=4, ndiag=3, nij=128,
             first_ij=1025),
        # the Jacobian of a Newton-Poisson step
        dict(name="adjoint_nm64_nx100", kind="adjoint", nm=64, nx=100, nen=296),
    ]


def _log_int(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["dropin", "solve", "solve", "solve", "solve", "solve", "w", "gw", "gwfft", "adjoint"])
    if kind == "dropin":
        return dict(kind=kind, nm=_log_int(rng, 16, 128, 8), nx=_log_int(rng, 3, 40))
    if kind == "gw":
        nky, nkz = rng.choice([(1, 1), (1, 3), (2, 2), (4, 1)])
        return dict(kind=kind, nm=rng.randint(5, 20), nx=rng.randint(3, 10), nen=_log_int(rng, 60, 512), nky=nky,
                    nkz=nkz, ndiag=rng.randint(0, 4), imag_only=rng.random() < 0.7)
    if kind == "gwfft":
        nky, nkz = rng.choice([(1, 1), (1, 4), (2, 2), (3, 2), (4, 4)])
        nm = rng.choice([16, 24, 64])
        return dict(kind=kind, nm=nm, nx=rng.randint(2, 10), nen=2 * _log_int(rng, 50, 2048), nky=nky, nkz=nkz,
                    ndiag=rng.randint(0, 4), nij=rng.randint(nm, 2 * nm), first_ij=nm * rng.randint(0, 7) + 1)
    nm = _log_int(rng, 16, 256, 8)
    nx = _log_int(rng, 4, 100)
    # no more work than the largest listed case
    most = 256 ** 3 * (30 * 30 + 400) * 148 / (float(nm) ** 3 * (30 * nx + 400))
    most = min(most, 24e9 / (16.0 * nm * nm * nx * 6))
    nen = _log_int(rng, 1, max(1, min(1000, int(most))))
    if kind == "w":
        return dict(kind=kind, nm=min(nm, 128), nx=nx, nen=min(nen, 256))
    if kind == "adjoint":
        return dict(kind=kind, nm=min(nm, 128), nx=nx, nen=max(2, min(nen, 296)))
    scattering = rng.random() < 0.4
    return dict(kind=kind, nm=nm, nx=nx, nen=nen, outputs=rng.choice(["density", "gw", "full"]), scattering=scattering,
                overlap=scattering and rng.random() < 0.4)


# ---------------------------------------------------------------------------
# inputs

_contexts = {}


def _context(**opts):
    """A program keeps one context for its solves."""
    key = tuple(sorted(opts.items()))
    if key not in _contexts:
        _contexts[key] = rgf.Context(rgf.Options(**opts))
    return _contexts[key]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _cnormal(g, *shape):
    return torch.complex(_normal(g, *shape), _normal(g, *shape))


def _energies(nen):
    """Mid-points of a grid over the bias window (few energies) or the band."""
    half = 0.3 if nen < 32 else 1.0
    return (np.arange(nen) + 0.5) / nen * 2 * half - half


def _device(g, nm, nx):
    """(Hii, H1i) in the Fortran block layout (nx, nm, nm), last axes (column, row)."""
    off = _cnormal(g, nm, nm) * (0.8 / math.sqrt(nm))
    H0 = torch.triu(off, 1)
    H0 = H0 + H0.mH
    onsite = torch.rand(nx, nm, generator=g, device="cuda", dtype=torch.float64) * 0.02
    onsite = onsite + torch.rand(nm, generator=g, device="cuda", dtype=torch.float64) - 0.5
    onsite = onsite + torch.linspace(0.1, -0.1, nx, device="cuda", dtype=torch.float64)[:, None]
    Hii = H0.expand(nx, nm, nm) + torch.diag_embed(onsite.to(torch.complex128))
    T = -2.7 * (torch.eye(nm, device="cuda", dtype=torch.float64) + _normal(g, nm, nm) * (0.3 / math.sqrt(nm)))
    H1i = T.to(torch.complex128).expand(nx, nm, nm)
    return Hii.mT.contiguous(), H1i.mT.contiguous()


def _overlap(g, nm, nx):
    X = torch.triu(_cnormal(g, nm, nm) * (0.05 / math.sqrt(nm)), 1)
    S = torch.eye(nm, device="cuda", dtype=torch.complex128) + X + X.mH
    return S.expand(nx, nm, nm).mT.contiguous()


def _self_energies(g, nm, nx, nen):
    """Scattering Sigma^< = i f B and Sigma^R = A - i B / 2 with B Hermitian
    positive and A Hermitian, per energy and block (a product of two small
    factors keeps the draw quick)."""
    r = 4
    U = _cnormal(g, nen, nx, nm, r) * math.sqrt(0.02 / nm)
    B = U @ U.mH + 0.002 * torch.eye(nm, device="cuda", dtype=torch.complex128)
    V = _cnormal(g, nx, nm, nm) * (0.02 / math.sqrt(nm))
    A = (V + V.mH).expand(nen, nx, nm, nm)
    f = torch.rand(nen, 1, 1, 1, generator=g, device="cuda", dtype=torch.float64)
    sl = (1j * f) * B
    sr = A - 0.5j * B
    return sl.mT.contiguous(), sr.mT.contiguous()


def _coulomb(g, nm, nx):
    """Bare Coulomb blocks of random orbital positions, 1.44 / (r + 0.3) eV."""
    pos = torch.rand(nx, nm, 3, generator=g, device="cuda", dtype=torch.float64)
    pos[:, :, 0] = (pos[:, :, 0] + torch.arange(nx, device="cuda")[:, None]) * 0.5
    pos[:, :, 1:] *= 2.0
    V = 1.44 / (torch.cdist(pos, pos) + 0.3)
    V1 = torch.zeros_like(V)
    V1[:-1] = 1.44 / (torch.cdist(pos[1:], pos[:-1]) + 0.3)   # V_{l+1,l}
    c = torch.complex128
    return V.to(c).mT.contiguous(), V1.to(c).mT.contiguous()


def _polarization(g, nm, nx, nen):
    """P^R complex symmetric, P^< and P^> i times real symmetric."""
    s = 0.02
    Y = _normal(g, nen, nx, nm, 4) / math.sqrt(nm)
    B = Y @ Y.mT
    X = _normal(g, nx, nm, nm) / math.sqrt(2 * nm)
    A = (X + X.mT).expand(nen, nx, nm, nm)
    f = torch.rand(nen, 1, 1, 1, generator=g, device="cuda", dtype=torch.float64)
    PR = torch.complex(s * A, -s * B)
    z = torch.zeros_like(B)
    return torch.complex(z, 2 * s * f * B), torch.complex(z, -2 * s * (1 - f) * B), PR


def _empty(*shape, dtype=torch.complex128):
    return torch.zeros(*shape, dtype=dtype, device="cuda")


def prepare(case, seed):
    g = _gen(seed)
    kind, nm, nx = case["kind"], case["nm"], case["nx"]
    s = dict(case=case)
    if kind == "dropin":
        s["ctx"] = _context(eta_dev=ETA, eta_lead=ETA)
        Hii, H1i = _device(g, nm, nx)
        s["E"] = float(np.random.default_rng(seed).uniform(-0.1, 0.1))
        s["Hii"], s["H1i"] = Hii.cpu().numpy(), H1i.cpu().numpy()
        z = np.zeros((nx, nm, nm), np.complex128)
        s["zero"] = z
        s["out"] = {k: np.zeros_like(z) for k in ("ndens", "pdens", "ldos", "GRi1")}
        s["out"]["cur"] = np.zeros((nx, nm, nm))
        s["out"]["tr"], s["out"]["tre"] = np.zeros(1), np.zeros(1)
        return s
    if kind == "solve":
        nen = case["nen"]
        s["ctx"] = _context(eta_dev=ETA, eta_lead=ETA)
        s["E"] = _energies(nen)
        s["Hii"], s["H1i"] = _device(g, nm, nx)
        s["Sii"] = _overlap(g, nm, nx) if case["overlap"] else None
        s["sl"], s["sr"] = _self_energies(g, nm, nx, nen) if case["scattering"] else (None, None)
        out = {}
        for k in OUTPUTS[case["outputs"]]:
            out[k] = _empty(nen, nx, nm, nm, dtype=torch.float64 if k == "cur" else torch.complex128)
        for k in ("T", "tr", "tre"):
            out[k] = _empty(nen, dtype=torch.float64)
        s["out"] = out
        return s
    if kind == "w":
        nen = case["nen"]
        s["ctx"] = _context(eta_dev=ETA, eta_lead=ETA)
        s["V"] = _coulomb(g, nm, nx)
        s["P"] = _polarization(g, nm, nx, nen)
        s["out"] = {k: _empty(nen, nx, nm, nm) for k in ("WL", "WG", "WR")}
        return s
    if kind == "adjoint":
        nen = case["nen"]
        s["ctx"] = _context(eta_dev=ETA_ADJOINT, eta_lead=ETA_ADJOINT)
        s["E"] = _energies(nen)
        s["Hii"], s["H1i"] = _device(g, nm, nx)
        s["out"] = dict(T=_empty(nen, dtype=torch.float64), dTdV=_empty(nen, nx, dtype=torch.float64),
                        dTds=_empty(nen, dtype=torch.float64))
        return s
    nen, nk = case["nen"], case["nky"] * case["nkz"]
    s["ctx"] = _context(eta_dev=ETA, eta_lead=ETA)
    if kind == "gw":
        shape = (nk, nen, nx, nm, nm)
        s["G"] = [_cnormal(g, *shape) * 0.1 for _ in range(3)]
        s["W"] = [_cnormal(g, *shape) * 0.1 for _ in range(3)]
        s["S"] = [_cnormal(g, *shape) * 0.01 for _ in range(3)]
        s["P"] = [_empty(*shape) for _ in range(3)]
    else:
        shape = (case["nij"], nx, nk, nen)
        s["G"] = [_cnormal(g, *shape) * 0.1 for _ in range(5)]
        s["W"] = [_cnormal(g, *shape) * 0.1 for _ in range(3)]
        s["P"] = [_empty(*shape) for _ in range(3)]
        s["S"] = [_empty(*shape) for _ in range(3)]
    return s


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "dropin":
        o, z = s["out"], s["zero"]
        rgf.green_RGF_RS(np.array(TEMP), case["nm"], case["nx"], s["E"], np.array(MU), s["Hii"], s["H1i"], z, z, z,
                         o["ndens"], o["pdens"], o["ldos"], o["tr"], o["tre"], o["cur"], GRi1=o["GRi1"], ctx=s["ctx"])
        return o
    ctx = s["ctx"]
    if kind == "solve":
        ctx.solve_energies(s["Hii"], s["H1i"], s["E"], MU, TEMP, sigma_lesser=s["sl"], sigma_r=s["sr"], Sii=s["Sii"],
                           **s["out"])
        return s["out"]
    if kind == "w":
        o = s["out"]
        ctx.w_solve_energies(*s["V"], *s["P"], WL=o["WL"], WG=o["WG"], WR=o["WR"])
        return o
    if kind == "adjoint":
        o = s["out"]
        dIdV, dIds = ctx.adjoint_energies(s["Hii"], s["H1i"], s["E"], MU, TEMP, T=o["T"], dTdV=o["dTdV"],
                                          dTds=o["dTds"])
        return dict(o, dIdV=dIdV, dIds=np.array([dIds]))
    P, S = s["P"], s["S"]
    grid = dict(nky=case["nky"], nkz=case["nkz"], ndiag=case["ndiag"])
    if kind == "gw":
        ctx.gw_polarization(*s["G"], PL=P[0], PG=P[1], PR=P[2], dE=0.01, spindeg=2.0, imag_only=case["imag_only"],
                            **grid)
        # the running self-energies are updated in place, as in the GW loop
        ctx.gw_self_energy(*s["G"], *s["W"], SL=S[0], SG=S[1], SR=S[2], dE=0.01, alpha_mix=0.5,
                           imag_only=case["imag_only"], **grid)
    else:
        grid.update(nm=case["nm"], first_ij=case["first_ij"], dEn=0.01)
        ctx.gw_polarization_fft(*s["G"], PL=P[0], PG=P[1], PR=P[2], spindeg=2.0, **grid)
        ctx.gw_self_energy_fft(*s["G"][:3], *s["W"], SL=S[0], SG=S[1], SR=S[2], **grid)
    return dict(PL=P[0], PG=P[1], PR=P[2], SL=S[0], SG=S[1], SR=S[2])


# ---------------------------------------------------------------------------
# the work a pass cannot do without

SANCHO = 19   # Sancho-Rubio iterations per lead at a broadening of 5 meV


def _band(case):
    """Banded (row, column) elements of the direct form."""
    nm, nd = case["nm"], case["ndiag"]
    return sum(min(nm - 1, i + nd) - max(0, i - nd) + 1 for i in range(nm))


def _banded_ij(case):
    nm, nd = case["nm"], case["ndiag"]
    return [i for i in range(case["nij"])
            if abs((i + case["first_ij"] - 1) // nm - (i + case["first_ij"] - 1) % nm) <= nd
            and (i + case["first_ij"] - 1) // nm < nm]


def work(case):
    kind, nm, nx = case["kind"], case["nm"], case["nx"]
    blk = 16.0 * nm * nm * nx
    if kind in ("dropin", "solve", "adjoint"):
        nen = case.get("nen", 1)
        outs = OUTPUTS["full" if kind == "dropin" else case["outputs"]] if kind != "adjoint" else ()
        # Sancho: 6 products and an inverse an iteration, both leads; forward
        # and backward sweep: the products of the recursion and one inverse
        per = 7.0 * 2 * SANCHO
        scattering = case.get("scattering", False)
        if kind == "adjoint":
            per += nx * (2 * 5 + 7)
        else:
            per += nx * (7 if scattering else 6) + nx * (7 if not scattering else 8)
            if "cur" in outs:
                per += nx * 6
            if case.get("overlap"):
                per += nx * 4
        bytes_ = 2 * blk + nen * blk * (len(outs) - (0.5 if "cur" in outs else 0.0))
        if scattering:
            bytes_ += 2 * nen * blk
        if case.get("overlap"):
            bytes_ += blk
        return dict(bytes=bytes_, flops=8.0 * nm ** 3 * per * nen)
    if kind == "w":
        return dict(bytes=2 * blk + 6 * case["nen"] * blk, flops=8.0 * nm ** 3 * 24 * nx * case["nen"])
    nen, nk = case["nen"], case["nky"] * case["nkz"]
    if kind == "gw":
        lines = _band(case) * nx
        # pairs of (energy, offset) of both windows; products of imaginary G
        # are one real multiply-add (P) or two (Sigma)
        m = max(nen // 2 - 10, 0)
        pairs = sum(nen - abs(v) for v in range(-m, m + 1)) * nk * nk
        fl = lines * pairs * ((2.0 * 4 + 2.0 * 10) if case["imag_only"] else (8.0 * 4 + 8.0 * 5))
        arr = 16.0 * nm * nm * nx * nen * nk
        return dict(bytes=6 * 16.0 * lines * nen * nk + 9 * arr, flops=fl)
    lines = len(_banded_ij(case)) * nx
    N = 2.0 * nen * nk
    io = 16.0 * nen * nk
    return dict(bytes=(5 + 6) * lines * io + 6 * case["nij"] * nx * io,
                flops=lines * (9 + 9) * 5.0 * N * math.log2(N) if lines else 1.0)


# ---------------------------------------------------------------------------
# the same results by torch in 64 bits


def _fermi(x):
    return 1.0 / (1.0 + torch.exp(x))


def _sancho(z, S, H, h10):
    """Surface Green's function of a semi-infinite lead (Sancho-Rubio)."""
    bb, ss, a, b = H, H, h10, h10.mH
    a, b = a.expand_as(bb), b.expand_as(bb)
    for _ in range(100):
        A = torch.linalg.inv(z * S - bb)
        Aa, Ab = A @ a, A @ b
        c = b @ Aa
        ss, bb = ss + c, bb + c + a @ Ab
        a, b = a @ Aa, b @ Ab
        if float(b.detach().abs().sum(dim=(-1, -2)).max()) < 1e-100:
            break
    return torch.linalg.inv(z * S - ss)


def _z(E, eta):
    return torch.complex(E, torch.full_like(E, eta))[:, None, None]


def _chain(E, Hii, H1i, Sii, sl, sr, outs, o):
    """green_RGF_RS / green_RGF_CMS for a batch of energies; outputs into o."""
    c = torch.complex128
    nx, nm = Hii.shape[0], Hii.shape[1]
    H, T = Hii.mT, H1i.mT
    eye = torch.eye(nm, device="cuda", dtype=c)
    S = Sii.mT if Sii is not None else eye.expand(nx, nm, nm)
    z = _z(E, ETA)

    def sig_r(l):
        if sr is None:
            return 0.0
        s = sr[:, l].mT
        return s @ S[l] if Sii is not None else s

    def sig_l(l):
        if sl is None:
            return 0.0
        s = sl[:, l].mT
        return s @ S[l] if Sii is not None else s

    def fermi(mu, temp):
        return _fermi((E - mu) / (BOLTZ * temp)).to(c)[:, None, None]

    batch = (E.shape[0], nm, nm)
    H0 = (H[0] + sig_r(0)).expand(batch)
    sigL = T[0] @ _sancho(z, S[0], H0, T[0].mH) @ T[0].mH
    g = [torch.linalg.inv(z * S[0] - H0 - sigL)]
    gl = [g[0] @ (-(sigL - sigL.mH) * fermi(MU[0], TEMP[0]) + sig_l(0)) @ g[0].mH]
    col = g[0]
    for l in range(1, nx - 1):
        g.append(torch.linalg.inv(z * S[l] - H[l] - sig_r(l) - T[l] @ g[-1] @ T[l].mH))
        gl.append(g[-1] @ (T[l] @ gl[-1] @ T[l].mH + sig_l(l)) @ g[-1].mH)
        col = g[-1] @ (T[l] @ col)
    n = nx - 1
    HN = (H[n] + sig_r(n)).expand(batch)
    sigR = T[n].mH @ _sancho(z, S[n], HN, T[n]) @ T[n]
    G = torch.linalg.inv(z * S[n] - HN - sigR - T[n] @ g[-1] @ T[n].mH)
    fR = fermi(MU[1], TEMP[0])
    Gn = G @ (-(sigR - sigR.mH) * fR + T[n] @ gl[-1] @ T[n].mH + sig_l(n)) @ G.mH

    def trace(A, B):
        return (A * B.mT).sum(dim=(-1, -2)).real

    def current(sig, f):
        """Re Tr[Sigma^<(contact) G^> - Sigma^>(contact) G^<]."""
        gam = -(sig - sig.mH)
        return trace(gam * f, Gn + G - G.mH) - trace(gam * (f - 1.0), Gn)

    o["tr"][:] = -current(sigR, fR)
    X = G @ (T[n] @ col)
    o["T"][:] = trace(1j * (sigR - sigR.mH), X @ (1j * (sigL - sigL.mH)) @ X.mH)

    def put(l, GR=None, cur=None, Gp=None):
        if "ldos" in outs:
            o["ldos"][:, l] = G.mT
        if "ndens" in outs:
            o["ndens"][:, l] = Gn.mT
        if "pdens" in outs:
            o["pdens"][:, l] = (Gn + G - G.mH if Gp is None else Gp).mT
        if GR is not None and "GRi1" in outs:
            o["GRi1"][:, l] = GR.mT
        if cur is not None and "cur" in outs:
            o["cur"][:, l] = cur.mT

    Gp = Gn + G - G.mH
    put(n)
    for l in range(nx - 2, -1, -1):
        Hb, gr, gn = T[l], g[l], gl[l]
        Q = gr @ Hb.mH
        GN0 = Q @ G
        cur = None
        if "cur" in outs:
            low = Hb.mH @ (Gn @ Q.mH + G @ (Hb @ gn))
            up = Hb @ (Q @ Gn + gn @ Hb.mH @ G.mH)
            cur = low.real - up.real
        R = GN0 @ Hb
        Gn = gn + Q @ Gn @ Q.mH + R @ gn + gn @ R.mH
        G = gr + R @ gr
        if Sii is not None:
            Gp = Q @ Gp @ Q.mH
        put(l, GN0, cur, Gp if Sii is not None else None)
        g[l] = gl[l] = None
    o["tre"][:] = current(sigL, fermi(MU[0], TEMP[1]))


def _exact_solve(s, outs):
    o = {}
    nx, nm = s["Hii"].shape[0], s["Hii"].shape[1]
    nen = len(s["E"])
    for k in outs:
        o[k] = _empty(nen, nx, nm, nm, dtype=torch.float64 if k == "cur" else torch.complex128)
    for k in ("T", "tr", "tre"):
        o[k] = _empty(nen, dtype=torch.float64)
    E = torch.from_numpy(s["E"]).cuda()
    step = max(1, int(20e9 / (16.0 * nm * nm * nx * 4)))
    for a in range(0, nen, step):
        part = slice(a, a + step)
        pick = lambda v: None if v is None else v[part]  # noqa: E731
        _chain(E[part], s["Hii"], s["H1i"], s["Sii"], pick(s["sl"]), pick(s["sr"]), outs,
               {k: v[part] for k, v in o.items()})
    return o


def _exact_w(s):
    """green_rgf_calc_w by its own recursions."""
    V, V1 = s["V"][0].mT, s["V"][1].mT
    PL, PG, PR = (p.mT for p in s["P"])
    nen, nx, nm = PL.shape[0], PL.shape[1], PL.shape[2]
    eye = torch.eye(nm, device="cuda", dtype=torch.complex128)
    out = {k: _empty(nen, nx, nm, nm) for k in ("WL", "WG", "WR")}
    x, wlr = [None] * nx, [None] * nx
    x[-1] = torch.linalg.inv(eye - V[-1] @ PR[:, -1])
    wlr[-1] = x[-1] @ V[-1]
    for l in range(nx - 2, -1, -1):
        up = -(V1[l].mH @ PR[:, l + 1])          # M_{l,l+1}
        low = -(V1[l] @ PR[:, l])                # M_{l+1,l}
        B = up @ x[l + 1]
        x[l] = torch.linalg.inv(eye - V[l] @ PR[:, l] - B @ low)
        wlr[l] = x[l] @ (V[l] - B @ V1[l])
    wo = wi_prev = low_prev = None
    for l in range(nx):
        W = wlr[l] if l == 0 else wlr[l] - x[l] @ low_prev @ wo
        wi = None
        if l < nx - 1:
            low = -(V1[l] @ PR[:, l])
            wo = (V1[l].mT - W @ low.mT) @ x[l + 1].mT
            low_prev = low
            wi = 1j * wo.imag
        wj = wi if l < nx - 1 else wi_prev
        wm = wi if l == 0 else wi_prev
        j, m = (l + 1 if l < nx - 1 else l), max(l - 1, 0)
        out["WR"][:, l] = W.mT
        for k, P in (("WL", PL), ("WG", PG)):
            out[k][:, l] = (W @ P[:, l] @ W.mH - wj @ P[:, j] @ wj.mT - wm.mT @ P[:, m] @ wm).mT
        wi_prev = wi
    return out


def _exact_adjoint(s):
    """T(E) of the chain, differentiated by autograd."""
    c = torch.complex128
    Hii, H1i = s["Hii"], s["H1i"]
    nx, nm = Hii.shape[0], Hii.shape[1]
    H, Tc = Hii.mT, H1i.mT
    nen = len(s["E"])
    eye = torch.eye(nm, device="cuda", dtype=c)
    T, dV, ds = (torch.zeros(n, device="cuda", dtype=torch.float64) for n in ((nen,), (nen, nx), (nen,)))
    step = max(1, int(60e9 / (16.0 * nm * nm * (10 * nx + 800))))
    for a in range(0, nen, step):
        E = torch.from_numpy(s["E"][a:a + step]).cuda()
        v = torch.zeros(len(E), nx, device="cuda", dtype=torch.float64, requires_grad=True)
        sc = torch.ones(len(E), device="cuda", dtype=torch.float64, requires_grad=True)
        z = _z(E, ETA_ADJOINT)

        def block(l):
            return H[l] + v[:, l, None, None] * eye

        def coupling(l):
            return Tc[l] * sc[:, None, None] if 1 <= l <= nx - 2 else Tc[l]

        n = nx - 1
        sigL = Tc[0] @ _sancho(z, eye, block(0), Tc[0].mH) @ Tc[0].mH
        g = torch.linalg.inv(z * eye - block(0) - sigL)
        col = g
        for l in range(1, nx - 1):
            h = coupling(l)
            g = torch.linalg.inv(z * eye - block(l) - h @ g @ h.mH)
            col = g @ (h @ col)
        sigR = Tc[n].mH @ _sancho(z, eye, block(n), Tc[n]) @ Tc[n]
        G = torch.linalg.inv(z * eye - block(n) - sigR - Tc[n] @ g @ Tc[n].mH)
        X = G @ (Tc[n] @ col)
        t = ((1j * (sigR - sigR.mH)) @ X @ (1j * (sigL - sigL.mH)) * X.conj()).sum(dim=(-1, -2)).real
        gv, gs = torch.autograd.grad(t.sum(), (v, sc))
        T[a:a + step], dV[a:a + step], ds[a:a + step] = t.detach(), gv, gs
    E = s["E"]
    f = [1.0 / (1.0 + np.exp((E - MU[i]) / (BOLTZ * TEMP[i]))) for i in (0, 1)]
    w = (f[0] - f[1]) * (E[1] - E[0]) * 1.6022e-19 / (PI * 2.0) / 1.0546e-34 * 1.6022e-19
    w = torch.from_numpy(w).cuda()
    return dict(T=T, dTdV=dV, dTds=ds, dIdV=(w @ dV).cpu().numpy(), dIds=(w @ ds).reshape(1).cpu().numpy())


def _k_sum(X, Y, nky, nkz, correlate):
    """Sum over k of X(k) with Y(k - q) (correlate) or of X(k - q) with Y(q),
    as circular transforms over the k-grid; X, Y spectra (..., nk, N)."""
    sh = X.shape
    X, Y = (torch.fft.fft2(a.reshape(*sh[:-2], nky, nkz, sh[-1]), dim=(-3, -2)) for a in (X, Y))
    if correlate:
        Y = torch.roll(torch.flip(Y, (-3, -2)), (1, 1), (-3, -2))
    R = torch.fft.ifft2(X * Y, dim=(-3, -2))
    # the reference's k - q index carries a shift of nk/2 - 1 per axis
    sy = (nky // 2 - 1) % nky if nky > 1 else 0
    sz = (nkz // 2 - 1) % nkz if nkz > 1 else 0
    sign = 1 if correlate else -1
    return torch.roll(R, (sign * sy, sign * sz), (-3, -2)).reshape(sh)


def _correlate(X, Y, nky, nkz, offsets, N):
    """sum_k sum_e X(e, k) Y(e - b, k - q) for each b of offsets; (..., nk, nen)."""
    fx = torch.fft.fft(X, N)
    fy = torch.fft.fft(Y, N)
    fy = torch.roll(torch.flip(fy, (-1,)), 1, -1)
    return torch.fft.ifft(_k_sum(fx, fy, nky, nkz, True))[..., offsets % N]


def _convolve(G, W, nky, nkz, offsets, N):
    """sum_q sum_b G(e - b, k - q) W(b, q), W given at each b of offsets."""
    placed = torch.zeros(*W.shape[:-1], N, dtype=W.dtype, device=W.device)
    placed[..., offsets % N] = W
    R = _k_sum(torch.fft.fft(G, N), torch.fft.fft(placed), nky, nkz, False)
    return torch.fft.ifft(R)[..., :G.shape[-1]]


def _exact_gwfft(s):
    case = s["case"]
    nen, nky, nkz = case["nen"], case["nky"], case["nkz"]
    nk, N, h = nky * nkz, 2 * nen, nen // 2
    shape = (case["nij"], case["nx"], nk, nen)
    out = {k: _empty(*shape) for k in ("PL", "PG", "PR", "SL", "SG", "SR")}
    fP = -1j * 0.01 / 2.0 / PI * 2.0 / nk
    fS = 1j * 0.01 / 2.0 / PI / nk
    shift = torch.arange(nen, device="cuda") - h
    place = torch.arange(-(h - 1), h, device="cuda")
    for i in _banded_ij(case):
        GL, GG, GR, GLt, GGt = (a[i] for a in s["G"])
        WL, WG, WR = (a[i][..., :nen - 1] for a in s["W"])
        P = lambda x, y: _correlate(x, y, nky, nkz, shift, N)  # noqa: E731
        C = lambda x, y: _convolve(x, y, nky, nkz, place, N)  # noqa: E731
        out["PL"][i] = P(GL, GGt) * fP
        out["PG"][i] = P(GG, GLt) * fP
        out["PR"][i] = (P(GL, GR.conj()) + P(GR, GLt)) * fP
        SL, SG = C(GL, WL) * fS, C(GG, WG) * fS
        SR = (C(GL, WR) + C(GR, WL) + C(GR, WR)) * fS
        out["SL"][i], out["SG"][i] = SL, SG
        out["SR"][i] = torch.complex(SR.real, (SG - SL).imag / 2.0)
    return out


def _exact_gw(s):
    case = s["case"]
    nm, nx, nen, nky, nkz, nd = (case[k] for k in ("nm", "nx", "nen", "nky", "nkz", "ndiag"))
    nk, N, m = nky * nkz, 2 * nen, nen // 2 - 10
    out = {k: torch.zeros_like(s["G"][0]) for k in ("PL", "PG", "PR")}
    new = [torch.zeros_like(a) for a in s["S"]]
    if m >= 0:
        fP = -1j * 0.01 / 2.0 / PI * 2.0 / nk
        fS = 1j * 0.01 / 2.0 / PI / nk
        off = torch.arange(-m, m + 1, device="cuda")
        at = off + nen // 2 - 1
        idx = torch.arange(nm, device="cuda")
        ii, jj = torch.meshgrid(idx, idx, indexing="ij")
        keep = (ii - jj).abs() <= nd
        ii, jj = ii[keep], jj[keep]

        def line(A, i, j):
            """(elements, nx, nk, nen) of A(i, j); the last axes of A are (column, row)."""
            return A[:, :, :, j, i].permute(3, 2, 0, 1)

        def back(dst, v, i, j, where):
            dst[:, where[:, None], :, j, i] = v.permute(0, 3, 2, 1)

        im = (lambda a: 1j * a.imag) if case["imag_only"] else (lambda a: a)
        G = [im(a) for a in s["G"]]
        for i, j in zip(ii.tolist(), jj.tolist()):
            i1, j1 = torch.tensor([i], device="cuda"), torch.tensor([j], device="cuda")
            GL, GG, GR = (line(a, i1, j1)[0] for a in G)
            GLt, GGt = (line(a, j1, i1)[0] for a in G[:2])
            WL, WG, WR = (line(a, i1, j1)[0][..., at] for a in s["W"])
            P = lambda x, y: _correlate(x, y, nky, nkz, off, N) * fP  # noqa: E731
            for k, v in (("PL", P(GL, GGt)), ("PG", P(GG, GLt)), ("PR", P(GL, GR.conj()) + P(GR, GLt))):
                out[k][:, at, :, j, i] = v.permute(1, 2, 0)
            # the sum leaves out G's last energy and the first output energy
            gl, gg, gr = (torch.cat([a[..., :-1], torch.zeros_like(a[..., -1:])], -1) for a in (GL, GG, GR))
            C = lambda x, y: _convolve(x, y, nky, nkz, off, N) * fS  # noqa: E731
            for k, v in enumerate((C(gl, WL), C(gg, WG), C(gl, WR) + C(gr, WL) + C(gr, WR))):
                v[..., 0] = 0
                new[k][:, :, :, j, i] = v.permute(1, 2, 0)
    NL, NG, NR = new
    NR = torch.complex(NR.real, (NG.imag - NL.imag) / 2.0)
    for k, v, old in (("SL", NL, s["S"][0]), ("SG", NG, s["S"][1]), ("SR", NR, s["S"][2])):
        r = old + 0.5 * ((v + v.mT) / 2.0 - old)
        for dst, src in ((0, 2), (1, 2), (nx - 1, nx - 3), (nx - 2, nx - 3)):
            r[:, :, dst] = r[:, :, src]
        out[k] = r
    return out


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    if kind == "dropin":
        t = dict(E=np.array([s["E"]]), Hii=torch.from_numpy(s["Hii"]).cuda(), H1i=torch.from_numpy(s["H1i"]).cuda(),
                 Sii=None, sl=None, sr=None)
        o = _exact_solve(t, OUTPUTS["full"])
        o.pop("T")
        return {k: (v if k in ("tr", "tre") else v[0]).cpu().numpy() for k, v in o.items()}
    if kind == "solve":
        return _exact_solve(s, OUTPUTS[case["outputs"]])
    if kind == "w":
        return _exact_w(s)
    if kind == "adjoint":
        return _exact_adjoint(s)
    if kind == "gw":
        return _exact_gw(s)
    return _exact_gwfft(s)
