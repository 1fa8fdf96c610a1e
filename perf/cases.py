"""The calls whose time this repository is judged by, with their inputs and checks.

Every case is one pass of a user's program through ``salmon_b200.rt.GpuSystem``:

  rt      one real-time step as ``drive.rt_propagate`` runs it (scf: Hartree + PZ
          potential rebuilt on the device; etrs: two half steps around the extrapolated
          potential) or, with a potential from the host, as ``bench.py``'s end-to-end
          leg runs it
  energy  kinetic and nonlocal energies of the resident orbitals, taken every few steps
  cg      the CG half of a ground-state iteration (``drive.ground_state``): Gram-Schmidt,
          CG, Gram-Schmidt, then the occupied bands and their density
  diag    its other half: Gram-Schmidt, subspace diagonalisation, the density.  The two are
          apart because eigenvectors are defined up to a phase, on which the reference's CG
          (real overlaps with the lower bands) depends
  hpsi    H applied to one orbital through host arrays, the smallest call of the library

The systems are diamond-Si cells (8 atoms per 10.26 bohr cube, s and p projectors), the
shapes of the testsuites, of ``system.BATCHED_SYSTEMS``, of ``tile_table.json`` and of
``bench.py``.  Orbitals and potentials are smooth random fields made from the seed.
``exact`` restates every pass with plain torch in 64 bits.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from salmon_b200 import system as S
from salmon_b200.rt import GpuSystem

CELL = 10.26          # bohr
RPS = 2.0             # projector sphere radius, bohr
DEV = "cuda"


# ------------------------------------------------------------------ the cases --
def _rt(name, cells, grid, nk, nb, prec, mode):
    return dict(name=name, kind="rt", cx=cells[0], cy=cells[1], cz=cells[2], nx=grid[0], ny=grid[1], nz=grid[2],
                nk=nk, nb=nb, nocc=nb, prec=prec, mode=mode)


def listed():
    one = (1, 1, 1)
    return [
        # H on one orbital between host arrays (hpsi_omp_KB_RT), as a host code calls it band by band
        dict(_rt("hpsi_16cubed_c128", one, (16, 16, 16), 8, 4, "c128", "-"), kind="hpsi"),
        # the bulk-Si testsuite's real-time step: 8^3 grid, 4^3 k-points, 16 occupied bands
        _rt("rt_8cubed_c128_scf", one, (8, 8, 8), 64, 16, "c128", "scf"),
        # the Si8 production step at the usual spacing
        _rt("rt_16cubed_c64_scf", one, (16, 16, 16), 64, 16, "c64", "scf"),
        # Si16, a non-cubic cell, with the other propagator
        _rt("rt_16x16x32_c64_etrs", (1, 1, 2), (16, 16, 32), 32, 32, "c64", "etrs"),
        # odd and ragged sizes: odd z rows, few k-points, a band count that fills no tile
        _rt("rt_18x24x27_c64_scf", one, (18, 24, 27), 5, 13, "c64", "scf"),
        # the benchmark's microbench shape, both precisions, potential from the host
        _rt("rt_32cubed_c64", one, (32, 32, 32), 64, 32, "c64", "host"),
        _rt("rt_32cubed_c128", one, (32, 32, 32), 64, 32, "c128", "host"),
        # the Si216 supercell step, the largest configuration
        _rt("rt_48cubed_c64_scf", (3, 3, 3), (48, 48, 48), 4, 432, "c64", "scf"),
        # the energies on a grid of no simple FFT size
        dict(_rt("energy_20cubed_c128", one, (20, 20, 20), 64, 32, "c128", "-"), kind="energy"),
        # the testsuite's ground state: 32 bands of which 16 occupied, CG as the reference has it
        dict(_rt("cg_8cubed", one, (8, 8, 8), 64, 32, "c128", "plain"), kind="cg", nocc=16, ncg=5),
        # Si64 on a rank's block of two k-points, 128 + 16 bands, TPA-preconditioned
        dict(_rt("cg_32cubed_tpa", (2, 2, 2), (32, 32, 32), 2, 144, "c128", "tpa"), kind="cg", nocc=128, ncg=4),
        # Si16's subspace diagonalisation, 32 + 8 bands
        dict(_rt("diag_16x16x32", (1, 1, 2), (16, 16, 32), 32, 40, "c128", "-"), kind="diag", nocc=32),
    ]


def _fft_ok(n):
    for p in (2, 3):
        while n % p == 0:
            n //= p
    return n == 1


def draw(rng):
    kind = rng.choices(["rt", "cg", "diag", "energy", "hpsi"], [6, 2, 1, 1, 1])[0]
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))  # noqa: E731
    cells = [rng.choice([1, 1, 1, 2, 2, 3]) for _ in range(3)]
    smooth = rng.random() < 0.6 or kind == "cg"  # sizes that the potential update and TPA take
    sizes = [n for n in range(8, 49) if _fft_ok(n) or not smooth]
    grid = []
    for c in cells:
        near = [n for n in sizes if 8 * c <= n <= min(48, 32 * c)]
        grid.append(min(near, key=lambda n, t=log(8 * c, min(48, 32 * c)): abs(n - t)))
    NL = grid[0] * grid[1] * grid[2]
    prec = "c128" if kind in ("cg", "diag") else rng.choice(["c64", "c64", "c128"])
    shape = dict(kind=kind, cx=cells[0], cy=cells[1], cz=cells[2], nx=grid[0], ny=grid[1], nz=grid[2], prec=prec)
    if kind in ("cg", "diag"):
        nb = log(6, 96 if kind == "cg" else 64)
        nk = max(1, min(log(1, 64), int(4e9 / (NL * nb * nb))))
        gs = dict(shape, nk=nk, nb=nb, nocc=max(1, nb - rng.randint(0, nb // 3)), mode="-")
        return dict(gs, mode=rng.choice(["plain", "tpa"]), ncg=rng.choice([2, 3, 4, 5])) if kind == "cg" else gs
    nb = log(1, 256)
    most = 8e7 if prec == "c64" else 4e7
    nb = max(1, min(nb, int(most / NL)))
    nk = max(1, min(log(1, 64), int(most / (NL * nb))))
    mode = rng.choice(["scf", "scf", "etrs"]) if all(_fft_ok(n) for n in grid) else "host"
    return dict(shape, nk=nk, nb=nb, nocc=nb, mode=mode if kind == "rt" else "-")


# --------------------------------------------------------------------- inputs --
_GEO = ("cx", "cy", "cz", "nx", "ny", "nz", "nk", "nb", "nocc")


@functools.lru_cache(maxsize=None)
def _geometry(cx, cy, cz, nx, ny, nz, nk, nb, nocc):
    aL = CELL * np.array([cx, cy, cz], dtype=np.float64)
    Rion = np.concatenate([(S.DIAMOND_RED + [i, j, k]) * CELL for i in range(cx) for j in range(cy) for k in range(cz)])
    Mps, Jxyz, Jxx, Jyy, Jzz, dist = S.calc_jxyz(nx, ny, nz, aL, Rion, RPS)
    uV, iuV, a_tbl = S.gaussian_projectors(Mps, dist, float(np.prod(aL / [nx, ny, nz])))
    nkx = max(d for d in (1, 2, 3, 4) if nk % d == 0)
    nky = max(d for d in (1, 2, 3, 4) if (nk // nkx) % d == 0)
    kAc0 = S.uniform_k_grid(nkx, nky, nk // nkx // nky, 2 * np.pi / aL)
    occ = np.zeros((nk, nb))
    occ[:, :nocc] = 2.0 / nk
    return S.System(NLx=nx, NLy=ny, NLz=nz, aL=aL, kAc0=kAc0, NB=nb, NBoccmax=nocc, occ=occ, Rion=Rion, Rps=RPS,
                    Mps=Mps, Jxyz=Jxyz, Jxx=Jxx, Jyy=Jyy, Jzz=Jzz, uV=uV, iuV=iuV, a_tbl=a_tbl)


def _sys(case):
    return _geometry(*(case[k] for k in _GEO))


def _filter(s, gc):
    """exp(-|G|^2 / 2 gc^2) on the grid's reciprocal lattice."""
    g = [2 * np.pi / a * n * torch.fft.fftfreq(n, dtype=torch.float64, device=DEV)
         for n, a in zip((s.NLx, s.NLy, s.NLz), s.aL)]
    return torch.exp(-(g[0][:, None, None] ** 2 + g[1][None, :, None] ** 2 + g[2][None, None, :] ** 2) / (2 * gc * gc))


def _potential(s, gen, scale=0.4):
    z = torch.randn((s.NLx, s.NLy, s.NLz), generator=gen, dtype=torch.float64, device=DEV)
    v = torch.fft.ifftn(torch.fft.fftn(z) * _filter(s, 1.0)).real
    return (scale * v / v.std() - scale).reshape(-1)


def _inputs(case, seed):
    """(orbitals (nk, bands, NL) complex128 on the GPU, potentials, k at the step's middle and end)."""
    s = _sys(case)
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    rng = np.random.default_rng(int(seed))
    nb = s.NB if case["kind"] in ("cg", "diag") else s.NBoccmax
    if case["kind"] == "hpsi":
        zu = torch.empty((1, 1, s.NL), dtype=torch.complex128, device=DEV)
    else:
        zu = torch.empty((s.NK, nb, s.NL), dtype=torch.complex128, device=DEV)
    # ground-state runs start from random orbitals, real-time runs from smooth ones
    f = None if case["kind"] in ("cg", "diag") else _filter(s, 1.0)
    for k in range(zu.shape[0]):
        z = torch.randn((zu.shape[1], s.NLx, s.NLy, s.NLz), generator=gen, dtype=torch.complex128, device=DEV)
        if f is not None:
            z = torch.fft.ifftn(z * f, dim=(1, 2, 3))
        z = z.reshape(zu.shape[1], -1)
        zu[k] = z / (z.abs().square().sum(dim=1, keepdim=True) * s.Hxyz).sqrt()
    if case["prec"] == "c64":
        zu = zu.to(torch.complex64).to(torch.complex128)  # inputs that complex(4) holds exactly
    v = [_potential(s, gen) for _ in range(2)]
    A = rng.uniform(-0.05, 0.05, (3, 3, 1))
    k = [np.ascontiguousarray(s.kAc0 + a) for a in A]
    return zu, v, k


def _dt(s):
    """A time step inside the Taylor step's stability range for this spacing."""
    return min(0.1, 1.8 / (3.25 * float((1.0 / s.H ** 2).sum())))


class _View:
    """A handle's device memory as torch takes it; the tensor keeps the view, and the view the handle."""

    def __init__(self, g, ptr, shape, typestr):
        self.g = g
        self.__cuda_array_interface__ = dict(shape=shape, typestr=typestr, data=(ptr, False), version=3)


def _state_view(g, st):
    p = g.state_ptr()
    if st.get("ptr") != p:
        s = g.sysm
        st["ptr"] = p
        st["zu"] = torch.as_tensor(_View(g, p, (s.NK, s.NBoccmax, s.NL), "<c16" if g.precision == "c128" else "<c8"),
                                   device=DEV)
    return st["zu"]


def prepare(case, seed):
    s = _sys(case)
    zu, v, k = _inputs(case, seed)
    torch.cuda.synchronize()  # the library has a stream of its own
    g = GpuSystem(s, case["prec"])
    st = dict(g=g, case=case, k=k, dt=_dt(s), v=[x.cpu().numpy() for x in v], n=0)
    if case["kind"] in ("cg", "diag"):
        g.gs_set_state(zu.cpu().numpy())
        g.set_vloc(st["v"][1])
        g.update_projector(k[0])
        if case["kind"] == "cg":
            g.set_cg_preconditioner(case["mode"])
    elif case["kind"] == "hpsi":
        st["psi"] = zu.reshape(-1).cpu().numpy()
        g.set_vloc(st["v"][0])
        g.update_projector(k[0])
    else:
        g.set_state_dev(zu.data_ptr())
        if case["mode"] in ("scf", "etrs"):
            g.set_vpsl(st["v"][0])
            g.update_vloc()
        else:
            g.set_vloc(st["v"][0])
        if case["mode"] == "etrs":
            g.vloc_history_reset()
        g.update_projector(k[0])
    return st


# ------------------------------------------------------------------- one pass --
def run(st):
    g, case, k, dt = st["g"], st["case"], st["k"], st["dt"]
    if case["kind"] == "hpsi":
        return g.hpsi_omp_KB_RT(1, st["psi"])
    if case["kind"] == "energy":
        return np.array(g.energy_terms(k[0]))
    if case["kind"] in ("cg", "diag"):
        # the potential moves between iterations, as in an SCF loop (two potentials in turn)
        g.set_vloc(st["v"][st["n"] % 2])
        st["n"] += 1
        g.gram_schmidt()
        if case["kind"] == "diag":
            out = {"esp": g.subspace_diag()}
            g.gs_to_rt()
        else:
            out = {"esp_var": g.cg(case["ncg"])[0]}
            g.gram_schmidt()
            g.gs_to_rt()
            out["zu"] = _state_view(g, st)
        out["rho"] = g.psi_rho_RT()
        return out
    if case["mode"] == "etrs":
        g.update_projector(k[0])
        g.hamiltonian(0.5 * dt)
        g.vloc_extrapolate()
        g.update_projector(k[2])
        g.hamiltonian(0.5 * dt, flag_current=True)
    else:
        g.update_projector(k[1])
        if case["mode"] == "host":
            g.set_vloc(st["v"][0])
        g.hamiltonian(dt, flag_current=True)
    out = {"energies": np.array(g.update_vloc())} if case["mode"] != "host" else {"rho": g.psi_rho_RT()}
    out["jav"] = g.current_RT(k[2])
    out["zu"] = _state_view(g, st)
    return out


# ------------------------------------------------------------- what it must do --
def work(case):
    s = _sys(case)
    S_ = 8 if case["prec"] == "c64" else 16
    sph = 4 * int(s.Mps.sum())                          # (projector, point) pairs of an orbital
    h = 158 * s.NL + 16 * sph                           # one H application of an orbital
    norb = s.NK * s.NBoccmax
    if case["kind"] == "hpsi":
        return {"bytes": 40 * s.NL + 8 * sph, "flops": h}
    if case["kind"] == "energy":
        return {"bytes": S_ * norb * s.NL, "flops": norb * (h + 8 * s.NL)}
    if case["kind"] in ("cg", "diag"):
        nb = s.NB
        orth = 8 * nb * nb * s.NL                       # Gram-Schmidt, or the lower bands' projections of all bands
        flops = orth + nb * (h + 8 * nb * s.NL * 1.5) + 30 * nb ** 3
        if case["kind"] == "cg":
            tpa = case["mode"] == "tpa"
            fft = 2 * 5 * s.NL * math.log2(s.NL) if tpa else 0
            flops = 2.5 * orth + case["ncg"] * ((2 if tpa else 1) * orth + nb * (h + 80 * s.NL + fft)) + 2 * nb * h
        return {"bytes": 2 * 16 * s.NK * nb * s.NL, "flops": s.NK * flops}
    steps = 2 if case["mode"] == "etrs" else 1
    flops = norb * (steps * 4 * (h + 8 * s.NL) + 3 * s.NL + 60 * s.NL + 20 * sph)
    return {"bytes": steps * 2 * S_ * norb * s.NL + 24 * s.NL, "flops": flops}


def tolerance(case):
    # measured against exact(): FP64 passes 1e-15 to 1e-14 (a sum in another order moves them as much),
    # complex(4) steps 0.8e-7 to 1.1e-7; one complex(4) H cancels 3.25 / h^2 per axis against values of order 1
    if case["kind"] in ("cg", "diag"):
        return {"rel": 1e-11}
    if case["prec"] == "c128":
        return {"rel": 1e-13}
    return {"rel": {"hpsi": 2e-5, "energy": 1e-7}.get(case["kind"], 5e-7)}


# -------------------------------------------------------------- in 64 bits --
class _H:
    """H of a system at the k-points ``k`` (3, NK), for batches (NK, nb, NL) on the GPU."""

    def __init__(self, s, k):
        self.s, self.shape, self.k = s, (s.NLx, s.NLy, s.NLz), torch.tensor(k.T.copy(), device=DEV)
        lap, nab = S.fd_coef()
        self.lap = [lap[S.ND:] / h ** 2 for h in s.H]
        self.nab = [nab[S.ND:] / h for h in s.H]
        m = torch.arange(s.Nps)[None, :] < torch.tensor(s.Mps)[:, None]
        self.idx = torch.tensor(np.where(m.numpy(), s.Jxyz - 1, 0)[s.a_tbl - 1].astype(np.int64), device=DEV)
        self.uV = torch.tensor(s.uV * m.numpy()[s.a_tbl - 1], device=DEV)
        self.pos = torch.tensor(s.sphere_positions()[s.a_tbl - 1], device=DEV)
        self.iuV = torch.tensor(s.iuV.astype(np.float64), device=DEV)

    def zproj(self, ik):
        return torch.exp(-1j * (self.pos @ self.k[ik])) * self.uV

    def local(self, x, ik, v=None):
        """((k - i grad)^2 / 2 + v) x for x (nb, NL); ik None: vector b of x at k-point b."""
        k = (self.k if ik is None else self.k[ik:ik + 1]).reshape(-1, 3, 1, 1, 1)
        x = x.reshape((-1,) + self.shape)
        out = x * (0.5 * (k.square().sum(dim=1) - sum(float(c[0]) for c in self.lap)))
        for d in range(3):
            kd = 1j * k[:, d]
            for n in range(1, 5):
                p, m = torch.roll(x, -n, d + 1), torch.roll(x, n, d + 1)
                out -= (0.5 * float(self.lap[d][n])) * (p + m) + (kd * float(self.nab[d][n])) * (p - m)
        out = out.reshape(out.shape[0], -1)
        return out if v is None else out + v * x.reshape(out.shape)

    def nonlocal_(self, x, z):
        """The projector term for x (nb, NL); z: zproj of one k-point, or of one per vector."""
        zb = z if z.dim() == 3 else z[None]
        u = (zb.conj() * x[:, self.idx]).sum(dim=2) * (self.s.Hxyz * self.iuV)
        out = torch.zeros_like(x)
        out.index_add_(1, self.idx.reshape(-1), (u[:, :, None] * zb).reshape(x.shape[0], -1))
        return out

    def __call__(self, x, ik, v):
        return self.local(x, ik, v) + self.nonlocal_(x, self.zproj(ik))


def _chunks(s, nb):
    c = max(1, int(3e7 // (s.NL + 4 * s.Nlma * s.Nps // max(1, s.NI) + s.Nlma * s.Nps)))
    return [(b, min(nb, b + c)) for b in range(0, nb, c)]


def _taylor(s, zu, k, v, dt):
    H = _H(s, k)
    for ik in range(zu.shape[0]):
        for b, e in _chunks(s, zu.shape[1]):
            t = zu[ik, b:e].clone()
            acc = t.clone()
            for n in range(1, 5):
                t = H(t, ik, v) * (-1j * dt / n)
                acc += t
            zu[ik, b:e] = acc


def _rho(s, zu):
    occ = torch.tensor(s.occ, device=DEV)
    rho = torch.zeros(s.NL, dtype=torch.float64, device=DEV)
    for ik in range(zu.shape[0]):
        for b in range(s.NBoccmax):
            rho += occ[ik, b] * zu[ik, b].abs().square()
    return rho


def _vloc(s, rho, vpsl):
    """(Hartree + PZ + vpsl, Eh, Exc)."""
    shape = (s.NLx, s.NLy, s.NLz)
    g = [2 * np.pi / a * n * torch.fft.fftfreq(n, dtype=torch.float64, device=DEV) for n, a in zip(shape, s.aL)]
    G2 = g[0][:, None, None] ** 2 + g[1][None, :, None] ** 2 + g[2][None, None, :] ** 2
    G2[0, 0, 0] = 1.0
    R = torch.fft.fftn(rho.reshape(shape)) * (4 * np.pi) / G2
    R[0, 0, 0] = 0.0
    vh = torch.fft.ifftn(R).real.reshape(-1)
    tr = rho + 1e-10
    rs = (3.0 / (4 * np.pi * tr)) ** (1.0 / 3.0)
    e = -0.75 * (3.0 / (2.0 * np.pi)) ** (2.0 / 3.0) / rs
    de = e / (3 * tr)
    den = 1.0 + 1.0529 * rs.sqrt() + 0.3334 * rs
    ln = rs.log()
    hi = rs > 1.0
    e = e + torch.where(hi, -0.1423 / den, 0.0311 * ln - 0.048 + 0.002 * rs * ln - 0.0116 * rs)
    de = de + torch.where(hi, -0.1423 * (0.5 * 1.0529 * rs.sqrt() + 0.3334 * rs) / (3 * tr) / den ** 2,
                          -rs / (3 * tr) * (0.0311 / rs + 0.002 * (ln + 1) - 0.0116))
    return vh + vpsl + e + rho * de, float(0.5 * (vh * rho).sum() * s.Hxyz), float((e * rho).sum() * s.Hxyz)


def _current(s, zu, k):
    H = _H(s, k)
    jav = torch.zeros(3, dtype=torch.float64, device=DEV)
    occ = torch.tensor(s.occ, device=DEV)
    vol = float(np.prod(s.aL))
    for ik in range(zu.shape[0]):
        z = H.zproj(ik)
        for b, e in _chunks(s, s.NBoccmax):
            x = zu[ik, b:e]
            o = occ[ik, b:e]
            g = x.reshape((-1,) + H.shape)
            nrm = x.abs().square().sum(dim=1)
            t = torch.einsum("lj,blj->blj", z.conj(), x[:, H.idx]) * s.Hxyz
            u = t.sum(dim=2) * H.iuV
            for d in range(3):
                f = sum(float(H.nab[d][n]) * (g.conj() * torch.roll(g, -n, d + 1)).imag.sum(dim=(1, 2, 3))
                        for n in range(1, 5))
                nl = ((t * H.pos[None, :, :, d]).sum(dim=2).conj() * u).imag.sum(dim=1)
                jav[d] += (o * (float(H.k[ik, d]) * nrm + 2 * f)).sum() * s.Hxyz / vol + (o * 2 * nl).sum() / vol
    return jav.cpu().numpy()


def _energies(s, zu, k):
    H = _H(s, k)
    occ = torch.tensor(s.occ, device=DEV)
    ek = en = 0.0
    for ik in range(zu.shape[0]):
        z = H.zproj(ik)
        k2 = 0.5 * float(H.k[ik].square().sum())
        for b, e in _chunks(s, s.NBoccmax):
            x, o = zu[ik, b:e], occ[ik, b:e]
            t = (x.conj() * H.local(x, ik)).sum(dim=1).real - k2 * x.abs().square().sum(dim=1)
            ek += float((o * (t * s.Hxyz + k2)).sum())
            u = torch.einsum("lj,blj->bl", z.conj(), x[:, H.idx]) * s.Hxyz
            en += float((o[:, None] * u.abs().square() * H.iuV).sum())
    return ek, en


def _orthonormal(zu, Hxyz):
    """Gram-Schmidt's result: the QR factorisation with a positive diagonal."""
    for k in range(zu.shape[0]):
        q, r = torch.linalg.qr(zu[k].T)
        d = torch.diagonal(r)
        zu[k] = (q * (d / d.abs())).T / math.sqrt(Hxyz)


def _cg(s, H, zu, v, ncg, tpa):
    """CG_ompk band by band, all k-points of a band together; returns the residuals times occ."""
    nk, NB, h = zu.shape[0], zu.shape[1], s.Hxyz
    dot = lambda a, b: (a.conj() * b).sum(dim=1, keepdim=True) * h  # noqa: E731
    nrm = lambda a: a.abs().square().sum(dim=1, keepdim=True) * h  # noqa: E731

    z = torch.stack([H.zproj(ik) for ik in range(nk)])

    def apply(x):
        t = H.local(x, None)
        return t + v * x + H.nonlocal_(x, z), t

    # the lower bands are not orthogonal to each other (their overlaps' imaginary parts stay), so the order of
    # the one-by-one projections counts: c_j = <u_j|x> - sum_{i<j} <u_j|u_i> c_i, a unit triangular system
    gram = torch.zeros((nk, NB, NB), dtype=zu.dtype, device=DEV)

    def lower(x, ib, part=lambda a: a):
        if ib == 0:
            return x
        d = part(torch.einsum("kbi,ki->kb", zu[:, :ib].conj(), x) * h)
        c = torch.linalg.solve_triangular(part(gram[:, :ib, :ib]), d[:, :, None], upper=False, unitriangular=True)
        return x - torch.einsum("kbi,kb->ki", zu[:, :ib], c[:, :, 0].to(x.dtype))

    if tpa:
        T = torch.zeros((nk,) + H.shape, dtype=torch.float64, device=DEV)
        for d, n in enumerate(H.shape):
            th = 2 * np.pi * torch.fft.fftfreq(n, dtype=torch.float64, device=DEV)
            t = sum(-float(H.lap[d][m]) * torch.cos(m * th) for m in range(1, 5)) - 0.5 * float(H.lap[d][0])
            q = sum(2 * float(H.nab[d][m]) * torch.sin(m * th) for m in range(1, 5))
            T += (t[None] + H.k[:, d:d + 1] * q[None]).reshape([nk] + [n if e == d else 1 for e in range(3)])
        T += 0.5 * H.k.square().sum(dim=1).reshape(nk, 1, 1, 1)
    var = torch.empty((nk, NB), dtype=torch.float64, device=DEV)
    occ = torch.tensor(s.occ, device=DEV)
    for ib in range(NB):
        u = lower(zu[:, ib], ib, part=lambda a: a.real)
        x = u / nrm(u).sqrt()
        hx, tx = apply(x)
        e = dot(x, hx).real
        pk = gg = None
        for it in range(ncg):
            gk = lower(hx - e * x, ib)
            if tpa:
                tb = dot(x, tx).real.clamp_min(1e-6).reshape(nk, 1, 1, 1)
                r = T.clamp_min(0) / tb
                p = 27 + r * (18 + r * (12 + 8 * r))
                hk = torch.fft.ifftn(torch.fft.fftn(gk.reshape((nk,) + H.shape), dim=(1, 2, 3)) * (p / (p + 16 * r ** 4)),
                                     dim=(1, 2, 3)).reshape(nk, -1)
                hk = lower(hk, ib)
                hk = hk - x * dot(x, hk)
                new = dot(gk, hk).real
            else:
                hk, new = gk, nrm(gk)
            pk = hk if it == 0 else hk + (new / gg) * pk
            gg = new
            po = pk - x * dot(x, pk)
            po = po / nrm(po).sqrt()
            hp, tp = apply(po)
            xp, pp = dot(x, hp), dot(po, hp).real
            ev = 0.5 * ((e + pp) - ((e - pp) ** 2 + 4 * xp.abs() ** 2).sqrt())
            cx = xp / (ev - e)
            cp = 1 / (1 + cx.abs() ** 2).sqrt()
            cx = cx * cp
            x, hx, tx = cx * x + cp * po, cx * hx + cp * hp, cx * tx + cp * tp
            e = dot(x, hx).real
        x = x / nrm(x).sqrt()
        zu[:, ib] = x
        gram[:, ib, :ib] = torch.einsum("kbi,ki->kb", zu[:, :ib], x.conj()) * h
        hx = apply(x)[0]
        var[:, ib] = nrm(hx - dot(x, hx).real * x).sqrt()[:, 0] * occ[:, ib]
    return var.cpu().numpy()


def exact(case, seed):
    s = _sys(case)
    zu, v, k = _inputs(case, seed)
    if case["kind"] == "hpsi":
        return _H(s, k[0])(zu[0], 0, v[0])[0].cpu().numpy()
    if case["kind"] == "energy":
        return np.array(_energies(s, zu, k[0]))
    if case["kind"] in ("cg", "diag"):
        H = _H(s, k[0])
        _orthonormal(zu, s.Hxyz)
        if case["kind"] == "diag":
            out = {"esp": np.empty((s.NK, s.NB))}
            for ik in range(s.NK):
                a = torch.einsum("bi,ci->bc", zu[ik].conj(), H(zu[ik], ik, v[0])) * s.Hxyz
                w, z = torch.linalg.eigh((a + a.conj().T) / 2)
                out["esp"][ik] = w.cpu().numpy()
                zu[ik] = torch.einsum("bi,bc->ci", zu[ik], z)
        else:
            out = {"esp_var": _cg(s, H, zu, v[0], case["ncg"], case["mode"] == "tpa")}
            _orthonormal(zu, s.Hxyz)
            out["zu"] = zu[:, :s.NBoccmax]
        out["rho"] = _rho(s, zu).cpu().numpy()
        return out
    dt = _dt(s)
    if case["mode"] == "host":
        _taylor(s, zu, k[1], v[0], dt)
        out = {"rho": _rho(s, zu).cpu().numpy()}
    else:
        v0 = _vloc(s, _rho(s, zu), v[0])[0]
        if case["mode"] == "etrs":
            _taylor(s, zu, k[0], v0, 0.5 * dt)
            # the first extrapolation: 3 V - 3 V + V with all three the starting potential
            _taylor(s, zu, k[2], v0, 0.5 * dt)
        else:
            _taylor(s, zu, k[1], v0, dt)
        out = {"energies": np.array(_vloc(s, _rho(s, zu), v[0])[1:])}
    out["jav"] = _current(s, zu, k[2])
    out["zu"] = zu
    return out
