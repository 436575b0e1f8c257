"""Default shapes of the FP64 smoother against 32x8 blocks, one launch per sweep.

Grids whose levels have one CTA of 128 points, a few, sixteen of more than 128, columns
beyond 128, and both block shapes of the per-sweep kernel: the solve ends in the same
state bit for bit.
"""
import numpy as np
import pytest

from tracer_code_gb300 import Simulation
from tests.cases import case_1024_like, fresh_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz,grids,Vbc", [(128, 64, 4, 0), (64, 64, 4, 1), (48, 128, 3, 0), (528, 32, 3, 1),
                                             (368, 184, 3, 0)])
def test_default_shapes_match(gpu_lib, nx, nz, grids, Vbc):
    p = case_1024_like(nx=nx, nz=nz, tpc=2, grids=grids)
    p.aspect, p.Vbc, p.max_cycles = nx / nz, Vbc, 200
    st = fresh_state(p, seed=nz)
    out = []
    for default in (True, False):
        g = Simulation(p)
        g.upload(st)
        if not default:
            g.set_launch_shapes([(32, 8, 0)] * (g.info.grids - 1))
        out.append((g.multigrid(), g.download()["SF"]))
        g.close()
    assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1])
