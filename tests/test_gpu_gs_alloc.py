"""The ground state's buffers: a call that runs out of memory leaves the handle as it was, and
the next one does not take half of the buffers for all of them."""
import numpy as np
import pytest

from _helpers import rel
from oracle import oracle as O
from salmon_b200 import system as S
from salmon_b200._lib import SalmonGPUError

pytestmark = pytest.mark.gpu


def test_out_of_memory(cuda_lib):
    """200000 bands of 64 points: the orbitals take 205 MB, one subspace matrix 640 GB."""
    from salmon_b200.rt import GpuSystem
    sysm, kAc, vloc, zu = S.small_system(4, 4, 4, nk=1, nb=3, nat=1, Rps=2.0, seed=2)
    nb = 200000
    sysm.NB = nb
    sysm.occ = np.concatenate([sysm.occ, np.zeros((1, nb - sysm.occ.shape[1]))], axis=1)
    _, zproj = O.update_projector(sysm, kAc)
    ref = O.hamiltonian(sysm, kAc, vloc, zproj, 0.02, zu)
    with GpuSystem(sysm) as g:
        g.set_vloc(vloc)
        g.update_projector(kAc)
        for _ in range(2):
            with pytest.raises(SalmonGPUError):
                g.gs_set_state(np.ones((1, nb, sysm.NL), complex))
        g.set_state(zu)
        g.hamiltonian(0.02)
        assert rel(g.get_state(), ref) < 1e-12


@pytest.mark.parametrize("grid", [(8, 10, 12), (16, 16, 16)])
def test_captured_step_after_growth(cuda_lib, grid):
    """More bands in the ground state than in real time: the projections' buffers grow, and a
    batch that captured a step before is captured anew."""
    from salmon_b200.rt import GpuBatch, GpuSystem
    sysm, kAc, vloc, zu = S.small_system(*grid, nk=2, nb=40, seed=2)
    sysm.NBoccmax = 3
    zu = np.ascontiguousarray(zu[:, :3])
    _, zproj = O.update_projector(sysm, kAc)
    one = O.hamiltonian(sysm, kAc, vloc, zproj, 0.02, zu)
    two = O.hamiltonian(sysm, kAc, vloc, zproj, 0.02, one)
    with GpuSystem(sysm) as g:
        g.set_vloc(vloc)
        g.update_projector(kAc)
        g.set_state(zu)
        with GpuBatch([g]) as b:
            b.step(0.02)
            assert rel(g.get_state(), one) < 1e-12
            g.gs_set_state(np.ones((2, 40, sysm.NL), complex))
            b.step(0.02)
            assert rel(g.get_state(), two) < 1e-12
