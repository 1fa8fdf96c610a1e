"""Sizes whose dynamic shared memory alone stays below the default limit of 48 KB and passes
it together with the kernel's static part.  A limit raised by an earlier, larger grid would
hide a missing one, so each case runs in its own process.  So does the first use of one kernel
by several threads at once.

Tolerances: FP64 sums in another order, 1e-12 (potential), 1e-11 (current, energies,
eigenvalues), as for the other sizes."""
import os
import subprocess
import sys

import numpy as np
import pytest

from _helpers import grid_system, rel
from oracle import oracle as O, scf_oracle as X
from salmon_b200 import system as S

pytestmark = pytest.mark.gpu


def potential(*shape):
    """27x54 and 18x81 planes: 48816 dynamic bytes and 528 static ones."""
    from salmon_b200.rt import GpuSystem
    sysm = grid_system(shape)
    rng = np.random.default_rng(3)
    rho, vpsl = rng.uniform(0.0, 0.5, sysm.NL), rng.standard_normal(sysm.NL)
    v_ref, e_ref = X.vloc(rho, vpsl, shape, sysm.aL, sysm.Hxyz)
    with GpuSystem(sysm) as g:
        g.set_vpsl(vpsl)
        e = g.update_vloc(rho)
        assert rel(g.get_vloc(), v_ref) < 1e-12 and rel(e, e_ref) < 1e-12


def march(*shape):
    """Rows of 252 to 256 points: 48384 to 49152 dynamic bytes and 1024 static ones."""
    from salmon_b200.rt import GpuSystem
    sysm, kAc, vloc, zu = S.small_system(*shape, nk=1, nb=2, seed=5)
    with GpuSystem(sysm) as g:
        g.set_state(zu)
        g.set_vloc(vloc)
        assert rel(g.current_RT(kAc), O.current(sysm, kAc, zu)) < 1e-11
        assert rel(g.energy_terms(kAc), O.energy_terms(sysm, kAc, zu)) < 1e-11


def eigensolver(*shape):
    """812 bands: 48736 dynamic bytes and 512 static ones."""
    from salmon_b200.rt import GpuSystem
    sysm, kAc, vloc, _ = S.small_system(*shape, nk=1, nb=812, seed=5)
    rng = np.random.default_rng(6)
    z = rng.standard_normal((1, 812, sysm.NL)) + 1j * rng.standard_normal((1, 812, sysm.NL))
    z = S.orthonormalise(z, sysm.Hxyz)
    with GpuSystem(sysm) as g:
        g.set_vloc(vloc)
        g.update_projector(kAc)
        g.gs_set_state(z)
        esp = g.subspace_diag()
    assert rel(esp, O.diag(sysm, kAc, vloc, z)[1]) < 1e-11


def threads(*rows):
    """Handles whose planes differ in size, first used at the same moment by a thread each."""
    from concurrent.futures import ThreadPoolExecutor
    from threading import Barrier
    from salmon_b200.rt import GpuSystem
    start = Barrier(len(rows))

    def one(n):
        sysm = grid_system((2, n, 96))
        with GpuSystem(sysm) as g:
            g.set_vpsl(np.zeros(sysm.NL))
            start.wait()
            for _ in range(20):
                g.update_vloc(np.ones(sysm.NL))

    with ThreadPoolExecutor(len(rows)) as ex:
        list(ex.map(one, rows))


@pytest.mark.parametrize("what,shape", [("threads", (16, 24, 27, 32, 36, 48, 54, 64)),
                                        ("potential", (2, 27, 54)), ("potential", (3, 18, 81)), ("march", (3, 2, 252)),
                                        ("march", (6, 4, 256)), ("eigensolver", (9, 10, 10))])
def test_default_limit_edge(cuda_lib, what, shape):
    here = os.path.dirname(os.path.abspath(__file__))
    code = f"import sys; sys.path[:0] = {[os.path.dirname(here), here]!r}; import {__name__} as t; t.{what}(*{shape!r})"
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
