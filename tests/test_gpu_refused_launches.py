"""Devices that refuse a cluster or a cooperative grid: the kernels without them take over.

tc_debug_refuse_clusters makes the launchers of the viscosity filter (in place and on a
copy), of the LU by panels, of the banded substitution and of the tile visits behave as if
the device had refused them.  Whole steps, eager and as one graph, then give the results of
a handle that was refused nothing, bit for bit: FP64 and mixed, an explicit inverse and a
banded coarse solve (n > 2048), and a handle refused only after its first step.
"""
import numpy as np
import pytest

from tracer_code_gb300 import Simulation
from tests.cases import case_1024_like, case_128_like, fresh_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mk,prec,nx,nz,grids", [(case_1024_like, 0, 128, 96, 3), (case_1024_like, 1, 496, 128, 5),
                                                 (case_1024_like, 1, 96, 96, 2), (case_128_like, 0, 92, 92, 2)])
def test_steps_are_the_same(gpu_lib, mk, prec, nx, nz, grids):
    p = mk(nx=nx, nz=nz, tpc=3, grids=grids)
    p.aspect, p.max_cycles = nx / nz, 200
    p.mg_zero_coarse, p.solver_precision = 1, prec
    p.cycle_correction = 3 if prec else 0
    st = fresh_state(p, seed=nx)
    out = []
    for when in (-1, 0, 1):  # refused: never, from the start, after the first step
        with Simulation(p) as g:
            g.set_step_graph(True)
            g.upload(st)
            res = []
            for n in range(3):
                if n == when:
                    g.debug_refuse_clusters(True)
                res.append(g.step())
            d = g.download()
            out.append((res, d["SF"], d["T"], d["rtr"], g.get("vis_grid", 2)))
    for o in out[1:]:
        assert o[0] == out[0][0]
        for a, b in zip(o[1:], out[0][1:]):
            assert np.array_equal(a, b)
