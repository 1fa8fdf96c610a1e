"""The blocked forms of the ground-state routines at the sizes where they change shape:
32-band panels of the Gram-Schmidt, 256-band blocks and the whole-GPU form of CG's
projections, the shared- and global-memory eigensolver.

Tolerances: FP64 sums of N terms in another order differ by a few eps times the
condition of what they feed: 1e-12 for well-conditioned Gram-Schmidt, eps * kappa for
a nearly dependent band, 1e-9 for CG (a few iterations amplify the rounding)."""
import numpy as np
import pytest

from _helpers import rel
from oracle import oracle as O
from salmon_b200 import system as S

pytestmark = pytest.mark.gpu


def raw_system(grid, nk, nb, seed=5):
    sysm, kAc, vloc, _ = S.small_system(*grid, nk=nk, nb=nb, seed=seed)
    rng = np.random.default_rng(seed + 1)
    z = rng.standard_normal((nk, nb, sysm.NL)) + 1j * rng.standard_normal((nk, nb, sysm.NL))
    return sysm, kAc, vloc, z


def handle(sysm, kAc, vloc, z):
    from salmon_b200.rt import GpuSystem
    g = GpuSystem(sysm)
    g.set_vloc(vloc)
    g.update_projector(kAc)
    g.gs_set_state(z)
    return g


def gram_schmidt(sysm, kAc, vloc, z):
    with handle(sysm, kAc, vloc, z) as g:
        g.gram_schmidt()
        return g.gs_get_state()


@pytest.mark.parametrize("nb", [1, 31, 32, 33, 70])
def test_gram_schmidt_panels(cuda_lib, nb):
    case = raw_system((7, 9, 11), 2, nb)
    out = gram_schmidt(*case)
    assert rel(out, O.gram_schmidt(case[0], case[3])) < 1e-12


def test_gram_schmidt_dependent_and_zero_bands(cuda_lib):
    sysm, kAc, vloc, z = raw_system((7, 9, 11), 3, 40)
    z[0, 5] = z[0, 3] + 1e-7 * z[0, 5]      # refused by the Cholesky of the first panel
    z[1, 36] = z[1, 34] + 1e-7 * z[1, 36]   # of the second
    ref = O.gram_schmidt(sysm, z)
    out = gram_schmidt(sysm, kAc, vloc, z)
    # kappa ~ 1e7: the dependent band itself moves by eps * kappa ~ 2e-9, and later ones with it
    assert rel(out, ref) < 1e-7
    assert rel(out[2], ref[2]) < 1e-12
    ov = np.einsum("kbi,kci->kbc", out.conj(), out) * sysm.Hxyz
    assert np.abs(ov - np.eye(40)).max() < 1e-7
    z[2, 4] = 0.0                           # NaN from there on, as one by one
    with np.errstate(all="ignore"):
        ref = O.gram_schmidt(sysm, z)
    out = gram_schmidt(sysm, kAc, vloc, z)
    np.testing.assert_array_equal(np.isnan(out[2]).any(axis=1), np.isnan(ref[2]).any(axis=1))
    assert rel(out[2, :4], ref[2, :4]) < 1e-12


def orthonormality(sysm, out):
    ov = np.einsum("kbi,kci->kbc", out.conj(), out) * sysm.Hxyz
    return np.abs(ov - np.eye(out.shape[1])).max()


@pytest.mark.parametrize("nb,sine", [(32, 0.51), (32, 0.55), (24, 0.51), (32, 0.6), (33, 0.6), (32, 0.8), (32, 0.99)])
def test_gram_schmidt_correlated_bands(cuda_lib, nb, sine):
    """Bands that each overlap with the one before: the distance to the earlier bands stays
    `sine` while the condition number grows like ((1 + cosine) / sine)^nb at worst.  Not worse
    than the one-by-one form, whose loss of orthogonality is a few eps * kappa."""
    sysm, kAc, vloc, z = raw_system((7, 9, 11), 2, nb)
    for k in range(2):
        q = np.linalg.qr(z[k].T)[0].T
        z[k, 0] = q[0]
        z[k, 1:] = np.sqrt(1 - sine**2) * q[:-1] + sine * q[1:]
    kappa = max(np.linalg.cond(z[k]) for k in range(2))
    out = gram_schmidt(sysm, kAc, vloc, z)
    eps = np.finfo(float).eps
    assert orthonormality(sysm, out) < 4 * eps * kappa + 1e-14
    assert rel(out, O.gram_schmidt(sysm, z)) < 20 * eps * kappa + 1e-13


@pytest.mark.parametrize("eps", [1e-1, 1e-2, 1e-3, 1e-4])
def test_gram_schmidt_second_round(cuda_lib, eps):
    """One close pair: a condition number of about 1 / eps, which the second round takes out
    within a panel; what is left of the first panel in the second one's bands is rounding
    over eps, as one by one."""
    sysm, kAc, vloc, z = raw_system((7, 9, 11), 2, 40)
    z[0, 5] = z[0, 3] + eps * z[0, 5]
    z[1, 36] = z[1, 34] + eps * z[1, 36]
    out = gram_schmidt(sysm, kAc, vloc, z)
    assert orthonormality(sysm, out[:1]) < 1e-14
    assert orthonormality(sysm, out) < 1e-15 / eps + 1e-14
    assert rel(out, O.gram_schmidt(sysm, z)) < 1e-14 / eps + 1e-13


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("band", [0, 17, 38])
def test_gram_schmidt_non_finite_band(cuda_lib, band, value):
    """The bands below a non-finite one stay what they are without it, as one by one."""
    sysm, kAc, vloc, z = raw_system((7, 9, 11), 2, 40)
    z[1, band, 100] = value
    with np.errstate(all="ignore"):
        ref = O.gram_schmidt(sysm, z)
    out = gram_schmidt(sysm, kAc, vloc, z)
    assert rel(out[0], ref[0]) < 1e-12
    assert np.isnan(out[1, band:]).any(axis=1).all()
    if band:
        assert rel(out[1, :band], ref[1, :band]) < 1e-12


@pytest.mark.parametrize("grid,nk,nb,orthonormal", [
    ((7, 9, 11), 2, 9, False),      # bands not orthogonal: the order of the projections counts
    ((8, 8, 8), 1, 260, True),      # two blocks of lower bands
    ((16, 16, 16), 1, 128, True),   # one k-point: projections over the whole GPU
    ((16, 16, 16), 1, 128, False),
])
def test_cg_projections(cuda_lib, grid, nk, nb, orthonormal):
    sysm, kAc, vloc, z = raw_system(grid, nk, nb)
    z = S.orthonormalise(z, sysm.Hxyz) if orthonormal else z / np.sqrt((np.abs(z) ** 2).sum(-1, keepdims=True) * sysm.Hxyz)
    with handle(sysm, kAc, vloc, z) as g:
        esp, its = g.cg(2)
        out = g.gs_get_state()
    ref, esp_ref, its_ref = O.cg(sysm, kAc, vloc, z, 2)
    np.testing.assert_array_equal(its, its_ref)
    assert rel(out, ref) < 1e-9
    assert rel(esp, esp_ref) < 1e-9


def test_gram_schmidt_many_k_points(cuda_lib):
    """More k-points than the second and third dimension of a grid can count."""
    from _helpers import grid_system
    from salmon_b200.rt import GpuSystem
    sysm = grid_system((3, 3, 3), nk=65600, nb=3)
    rng = np.random.default_rng(8)
    z = rng.standard_normal((65600, 3, sysm.NL)) + 1j * rng.standard_normal((65600, 3, sysm.NL))
    with GpuSystem(sysm) as g:
        g.gs_set_state(z)
        g.gram_schmidt()
        out = g.gs_get_state()
    assert rel(out, O.gram_schmidt(sysm, z)) < 1e-12


def tpa_cg(sysm, kAc, vloc, z, ncg):
    """CG with the Teter-Payne-Allan factor as it is defined, projection by projection."""
    from oracle import net_oracle as N
    d = sysm.desc()
    lap3, nab3 = (np.array([list(getattr(d, p + c)) for c in "xyz"]) for p in ("lap", "nab"))
    shape, w = (sysm.NLx, sysm.NLy, sysm.NLz), sysm.Hxyz
    _, zproj = O.update_projector(sysm, kAc)
    z = z.copy()
    for k in range(sysm.nk_local):
        H = lambda x: O.hpsi(sysm, kAc, vloc, zproj, k + 1, x, want_tt=True)  # noqa: E731
        dot = lambda a, b: np.vdot(a, b) * w  # noqa: E731

        def project(x, lower):
            for u in lower:
                x = x - u * dot(u, x)
            return x

        for b in range(sysm.NB):
            x, lower = z[k, b], z[k, :b]
            for u in lower:
                x = x - u * dot(u, x).real
            x = x / np.sqrt(dot(x, x).real)
            hx, tx = H(x)
            for it in range(ncg):
                e, t = dot(x, hx).real, dot(x, tx).real
                g = project(hx - e * x, lower)
                h = project(N.tpa_apply(g, shape, kAc[:, k], max(t, 1e-6), lap3, nab3), lower)
                h = h - x * dot(x, h)
                s = dot(g, h).real
                p = h if it == 0 else h + s / s_old * p
                s_old = s
                q = p - x * dot(x, p)
                q = q / np.sqrt(dot(q, q).real)
                hq, tq = H(q)
                c, f = dot(x, hq), dot(q, hq).real
                ev = 0.5 * (e + f - np.sqrt((e - f) ** 2 + 4 * abs(c) ** 2))
                cx = c / (ev - e)
                cp = 1 / np.sqrt(1 + abs(cx) ** 2)
                x, hx, tx = (cp * (cx * a + y) for a, y in ((x, q), (hx, hq), (tx, tq)))
            z[k, b] = x / np.sqrt(dot(x, x).real)
    return z


@pytest.mark.parametrize("grid,nk,nb", [((8, 9, 12), 2, 9), ((16, 16, 16), 1, 128)])  # clusters, the whole GPU
def test_cg_projections_preconditioned(cuda_lib, grid, nk, nb):
    sysm, kAc, vloc, z = raw_system(grid, nk, nb)
    z = S.orthonormalise(z, sysm.Hxyz)
    with handle(sysm, kAc, vloc, z) as g:
        g.set_cg_preconditioner("tpa")
        g.cg(3)
        out = g.gs_get_state()
    assert rel(out, tpa_cg(sysm, kAc, vloc, z, 3)) < 1e-9


@pytest.mark.parametrize("nb", [7, 82, 84, 128])  # A and V in shared memory up to 82 bands
def test_subspace_diag_sizes(cuda_lib, nb):
    sysm, kAc, vloc, z = raw_system((8, 9, 10), 2, nb)
    z = S.orthonormalise(z, sysm.Hxyz)
    with handle(sysm, kAc, vloc, z) as g:
        esp = g.subspace_diag()
        out = g.gs_get_state()
    _, esp_ref = O.diag(sysm, kAc, vloc, z)
    assert rel(esp, esp_ref) < 1e-11
    ov = np.einsum("kbi,kci->kbc", out.conj(), out) * sysm.Hxyz
    assert np.abs(ov - np.eye(nb)).max() < 1e-11
    for k in range(2):
        assert rel(out[k].T @ out[k].conj(), z[k].T @ z[k].conj()) < 1e-10


def plane_wave_bands(shape, nb, mix):
    """Plane waves on a grid without projectors, whose H is diagonal with known values, the
    bands b and b + nb/2 mixed by a rotation for every b in mix."""
    from _helpers import grid_system
    sysm = grid_system(shape, nk=1, nb=nb)
    ln = sysm.lap_nab()
    e, waves = [], []
    for d, n in enumerate(shape):
        lap = ln["lap" + "xyz"[d]]
        m = np.arange(n)
        e.append(-0.5 * (lap[0] + 2 * sum(lap[j] * np.cos(2 * np.pi * m * j / n) for j in range(1, 5))))
        waves.append(np.exp(2j * np.pi * np.outer(m, np.arange(n)) / n))
    e = (e[0][:, None, None] + e[1][:, None] + e[2]).ravel()
    z = np.einsum("ax,by,cz->abcxyz", *waves).reshape(sysm.NL, sysm.NL)[:nb] / np.sqrt(sysm.NL * sysm.Hxyz)
    for b in mix:
        z[b], z[b + nb // 2] = 0.8 * z[b] + 0.6j * z[b + nb // 2], 0.6j * z[b] + 0.8 * z[b + nb // 2]
    return sysm, z[None], np.sort(e[:nb])


def test_subspace_diag_many_bands(cuda_lib):
    """More than 2048 bands: more rotations in a step than a CTA has threads."""
    from salmon_b200.rt import GpuSystem
    nb = 2080
    sysm, z, e = plane_wave_bands((13, 13, 13), nb, [3, 520, 1035])
    with GpuSystem(sysm) as g:
        g.set_vloc(np.zeros(sysm.NL))
        g.update_projector(np.zeros((3, 1)))
        g.gs_set_state(z)
        esp = g.subspace_diag()
        out = g.gs_get_state()[0]
    assert np.abs(esp[0] - e).max() < 1e-11 * np.abs(e).max()
    assert np.abs(out.conj() @ out.T * sysm.Hxyz - np.eye(nb)).max() < 1e-11
