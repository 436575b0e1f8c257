"""The banded LU of the coarsest matrix, and its solves, at the edges of their kernels.

Solves whose coarsest grids have the narrowest bands, bands at both sides of the
one-block kernel's limit (kl = 20) and of the panel kernel's block sizes (kl = 32, 96 and
224), the last panel full, of one column and in between; above 2048 unknowns also the
substitution's block sizes (kl = 240 and 496) and a band within one block of rows.  Cycle
counts equal the oracle's and the stream function agrees within the bound of
test_gpu_parity.py (1e-9 of its largest value).
"""
import numpy as np
import pytest

from oracle.pyoracle import Oracle
from tracer_code_gb300 import Simulation
from tests.cases import case_1024_like, fresh_state

pytestmark = pytest.mark.gpu


# n = (nx / 2^(grids-1) + 1) (nz / 2^(grids-1) + 1), kl = 2 nz / 2^(grids-1) + 2
@pytest.mark.parametrize("nx,nz,grids,kl", [(64, 16, 3, 10), (48, 18, 2, 20), (48, 20, 2, 22), (44, 22, 2, 24),
                                            (42, 30, 2, 32), (46, 32, 2, 34), (20, 94, 2, 96), (16, 96, 2, 98),
                                            (14, 222, 2, 224), (16, 224, 2, 226),
                                            (2000, 16, 3, 10), (92, 92, 2, 94), (36, 238, 2, 240), (34, 240, 2, 242),
                                            (16, 494, 2, 496), (16, 496, 2, 498)])
def test_solve_equals_oracle(gpu_lib, nx, nz, grids, kl):
    p = case_1024_like(nx=nx, nz=nz, tpc=4, grids=grids)
    p.aspect, p.max_cycles = nx / nz, 200
    st = fresh_state(p, seed=nx)
    g, o = Simulation(p), Oracle(p)
    for s in (g, o):
        s.upload(st)
        s.compute_velocities()
    assert (g.info.kl, g.info.ku, g.info.grids) == (kl, kl, grids)
    assert g.multigrid() == o.multigrid()
    a, b = g.download()["SF"], o.download()["SF"]
    assert np.abs(b).max() > 0 and np.abs(a - b).max() <= 1e-9 * np.abs(b).max()
    g.close()
