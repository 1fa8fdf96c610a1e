"""The forms for small batches and grids against the general ones and the oracle: the
point-parallel H application (rows of odd length, grids below the stencil's width, points
in several spheres), the fused transforms of the potential (every radix, one axis of
length 1, planes beyond shared memory) and the density with few orbitals.

Tolerances: complex(8) 1e-12 (FP64 sums in another order); complex(4) 2e-6, the bound of
the complex(4) step against the FP64 oracle."""
import numpy as np
import pytest

from _helpers import grid_system, rel
from oracle import oracle as O, scf_oracle as X
from salmon_b200 import system as S

pytestmark = pytest.mark.gpu
TOL = {"c128": 1e-12, "c64": 2e-6}


@pytest.mark.parametrize("precision", ["c128", "c64"])
@pytest.mark.parametrize("shape,nat,rps", [((8, 10, 12), 2, 1.6), ((3, 5, 7), 1, 0.9), ((9, 7, 11), 6, 3.0)])
def test_point_form(cuda_lib, precision, shape, nat, rps):
    from salmon_b200.rt import GpuSystem
    sysm, kAc, vloc, zu = S.small_system(*shape, nk=2, nb=3, nat=nat, Rps=rps, seed=11)
    _, zproj = O.update_projector(sysm, kAc)
    z_in = zu if precision == "c128" else zu.astype(np.complex64).astype(np.complex128)
    ref = O.hamiltonian(sysm, kAc, vloc, zproj, 0.01, z_in)
    h_ref, tt_ref = O.hpsi(sysm, kAc, vloc, zproj, 2, z_in[1, 1], want_tt=True)
    out = {}
    for kernel in (0, 1):  # 0: small batches take the point form; 1: the stencil passes
        with GpuSystem(sysm, precision) as g:
            g.set_param("taylor_kernel", kernel)
            g.set_state(zu)
            g.set_vloc(vloc)
            g.update_projector(kAc)
            g.hamiltonian(0.01)
            assert rel(g.get_state(), ref) < TOL[precision]
            g.hamiltonian(0.01)  # projects from the sphere values that the first step exported
            out[kernel] = g.get_state()
            h, tt = g.hpsi_omp_KB_GS(2, z_in[1, 1])
            assert rel(h, h_ref) < TOL[precision] and rel(tt, tt_ref) < TOL[precision]
    assert rel(out[0], out[1]) < TOL[precision]


@pytest.mark.parametrize("shape", [(8, 9, 12), (1, 6, 8), (16, 2, 27), (6, 81, 64), (4, 96, 96)])
def test_fused_potential(cuda_lib, shape):
    from salmon_b200.rt import GpuSystem
    sysm = grid_system(shape)
    rng = np.random.default_rng(3)
    rho = rng.uniform(0.0, 0.5, sysm.NL)
    vpsl = rng.standard_normal(sysm.NL)
    v_ref, e_ref = X.vloc(rho, vpsl, shape, sysm.aL, sysm.Hxyz)
    with GpuSystem(sysm) as g:
        g.set_vpsl(vpsl)
        for _ in range(2):  # the energies' counter is back at zero
            e = g.update_vloc(rho)
            assert rel(g.get_vloc(), v_ref) < 1e-12
            assert rel(e, e_ref) < 1e-12


@pytest.mark.parametrize("nk,nb", [(1, 1), (1, 15), (1, 17), (3, 33)])
def test_density_chunks(cuda_lib, nk, nb):
    from salmon_b200.rt import GpuSystem
    sysm, _, _, zu = S.small_system(5, 6, 7, nk=nk, nb=nb)
    with GpuSystem(sysm) as g:
        g.set_state(zu)
        assert rel(g.psi_rho_RT(), O.psi_rho(sysm, zu)) < 1e-12


@pytest.mark.parametrize("precision", ["c128", "c64"])
@pytest.mark.parametrize("shape", [(9, 33, 20), (6, 5, 40), (4, 3, 7), (7, 1, 9), (3, 2, 130)])
def test_current_and_energy_march(cuda_lib, precision, shape):
    """Blocks of rows with an odd last one, a single row, fewer planes than the queue."""
    from salmon_b200.rt import GpuSystem
    sysm, kAc, vloc, zu = S.small_system(*shape, nk=2, nb=2, seed=5)
    z = zu if precision == "c128" else zu.astype(np.complex64).astype(np.complex128)
    with GpuSystem(sysm, precision) as g:
        g.set_state(zu)
        g.set_vloc(vloc)
        jav, e = g.current_RT(kAc), g.energy_terms(kAc)
    assert rel(jav, O.current(sysm, kAc, z)) < 1e-11  # FP64 sums in both precisions
    assert rel(e, O.energy_terms(sysm, kAc, z)) < 1e-11


@pytest.mark.parametrize("precision", ["c128", "c64"])
@pytest.mark.parametrize("shape,nb", [((22, 9, 11), 1), ((13, 34, 16), 3), ((10, 8, 8), 80), ((31, 36, 30), 2)])
def test_march_slabs(cuda_lib, precision, shape, nb):
    """Few orbitals: the march in slabs of at least four planes, the last one shorter."""
    from salmon_b200.rt import GpuSystem
    sysm, kAc, vloc, zu = S.small_system(*shape, nk=1, nb=nb, seed=5)
    z = zu if precision == "c128" else zu.astype(np.complex64).astype(np.complex128)
    with GpuSystem(sysm, precision) as g:
        g.set_state(zu)
        g.set_vloc(vloc)
        assert rel(g.current_RT(kAc), O.current(sysm, kAc, z)) < 1e-11
        assert rel(g.energy_terms(kAc), O.energy_terms(sysm, kAc, z)) < 1e-11
        g.update_projector(kAc)
        g.hamiltonian(0.004, flag_current=True)
        z1 = np.asarray(g.get_state(), np.complex128)
        assert rel(g.current_RT(kAc), O.current(sysm, kAc, z1)) < 1e-11


@pytest.mark.parametrize("precision", ["c128", "c64"])
@pytest.mark.parametrize("cur_fixed", [1, 2])
@pytest.mark.parametrize("shape", [(1, 32, 32), (3, 32, 32), (4, 48, 48), (5, 32, 32), (6, 48, 48)])
def test_current_of_few_planes(cuda_lib, precision, cur_fixed, shape):
    """Planes with a fixed form of the current: around the length of its queue (five planes),
    as a call of its own and out of a step that computes the sums beside the update."""
    from salmon_b200.rt import GpuSystem
    sysm, kAc, vloc, zu = S.small_system(*shape, nk=1, nb=3, a=(shape[0] * 0.5, 9.0, 9.5), seed=5)
    z = zu if precision == "c128" else zu.astype(np.complex64).astype(np.complex128)
    with GpuSystem(sysm, precision) as g:
        g.set_param("cur_fixed", cur_fixed)
        g.set_state(zu)
        g.set_vloc(vloc)
        assert rel(g.current_RT(kAc), O.current(sysm, kAc, z)) < 1e-11
        g.update_projector(kAc)
        g.hamiltonian(0.004, flag_current=True)
        z1 = np.asarray(g.get_state(), np.complex128)
        assert rel(g.current_RT(kAc), O.current(sysm, kAc, z1)) < 1e-11


@pytest.mark.parametrize("precision", ["c128", "c64"])
@pytest.mark.parametrize("shape,nslab", [((3, 32, 32), 1), ((10, 32, 32), 3), ((7, 48, 48), 2), ((5, 16, 32), 1),
                                         ((4, 16, 16), 1)])
def test_two_row_pass(cuda_lib, precision, shape, nslab):
    """Planes with a two-row form: fewer planes than the queue, x-slabs, the H application too."""
    from salmon_b200.rt import GpuSystem
    sysm, kAc, vloc, zu = S.small_system(*shape, nk=1, nb=3, a=(shape[0] * 0.5, 9.0, 9.5), seed=3)
    _, zproj = O.update_projector(sysm, kAc)
    z_in = zu if precision == "c128" else zu.astype(np.complex64).astype(np.complex128)
    with GpuSystem(sysm, precision) as g:
        g.set_param("taylor_kernel", 1)
        g.set_param("nslab", nslab)
        g.set_state(zu)
        g.set_vloc(vloc)
        g.update_projector(kAc)
        g.hamiltonian(0.004)
        assert rel(g.get_state(), O.hamiltonian(sysm, kAc, vloc, zproj, 0.004, z_in)) < TOL[precision]
        h, tt = g.hpsi_omp_KB_GS(1, z_in[0, 2])
    h_ref, tt_ref = O.hpsi(sysm, kAc, vloc, zproj, 1, z_in[0, 2], want_tt=True)
    assert rel(h, h_ref) < TOL[precision] and rel(tt, tt_ref) < TOL[precision]


@pytest.mark.parametrize("precision", ["c128", "c64"])
@pytest.mark.parametrize("nb,rps", [(1, 0.7), (5, 1.6), (35, 1.6), (33, 2.4)])
def test_whole_atom_projections(cuda_lib, precision, nb, rps):
    """Atoms staged whole: ragged band groups, points in two spheres, atoms of few points."""
    from salmon_b200.rt import GpuSystem
    sysm, kAc, vloc, zu = S.small_system(8, 10, 12, nk=2, nb=nb, Rps=rps, seed=9)
    _, zproj = O.update_projector(sysm, kAc)
    z_in = zu if precision == "c128" else zu.astype(np.complex64).astype(np.complex128)
    with GpuSystem(sysm, precision) as g:
        g.set_param("taylor_kernel", 1)
        g.set_state(zu)
        g.set_vloc(vloc)
        g.update_projector(kAc)
        g.hamiltonian(0.02)
        assert rel(g.get_state(), O.hamiltonian(sysm, kAc, vloc, zproj, 0.02, z_in)) < TOL[precision]


@pytest.mark.parametrize("precision", ["c128", "c64"])
def test_projector_tables_wider_than_the_atoms(cuda_lib, precision):
    """Atoms of few points in tables with room for 30000: the tile kernels do not fit in shared
    memory, the whole-atom form does; a single step and a captured one."""
    from salmon_b200.rt import GpuBatch, GpuSystem
    sysm, kAc, vloc, zu = S.small_system(8, 10, 12, nk=2, nb=5, seed=9)
    _, zproj = O.update_projector(sysm, kAc)
    z_in = zu if precision == "c128" else zu.astype(np.complex64).astype(np.complex128)
    ref = O.hamiltonian(sysm, kAc, vloc, zproj, 0.02, z_in)
    n = sysm.uV.shape[1]
    for name in ("Jxyz", "Jxx", "Jyy", "Jzz", "uV"):
        t = getattr(sysm, name)
        wide = np.zeros((t.shape[0], 30000), t.dtype)
        wide[:, :n] = t
        setattr(sysm, name, wide)
    with GpuSystem(sysm, precision) as g:
        g.set_param("taylor_kernel", 1)
        g.set_vloc(vloc)
        g.update_projector(kAc)
        g.set_state(zu)
        g.hamiltonian(0.02)
        assert rel(g.get_state(), ref) < TOL[precision]
        g.set_state(zu)
        b = GpuBatch([g])
        b.step([0.02])
        assert rel(g.get_state(), ref) < TOL[precision]
        b.close()
