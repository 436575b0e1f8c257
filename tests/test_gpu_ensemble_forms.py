"""What an ensemble step changes for a handle ends with the call.

Handles that step side by side use no visit over the whole grid (k_tile.cu).  A handle
that is stepped alone again, or that is the only one of an ensemble, takes the forms of a
handle that never was in an ensemble: as many kernels in each step, and the same bits
throughout.  512x128 cells: level 1 runs over the grid when it can.
"""
import numpy as np
import pytest

from tracer_code_gb300 import Simulation, load_library, state
from tests.cases import case_1024_like

pytestmark = pytest.mark.gpu


def _case():
    p = case_1024_like(nx=512, nz=128, grids=5, tpc=3, Ra=1.0e5, visT=100.0)
    p.mg_zero_coarse, p.mg_coarse_matrix, p.solver_precision, p.cycle_correction = 1, 1, 1, 3
    return p


def _launches(f):
    lib = load_library()
    lib.tc_kernel_launches.restype = __import__("ctypes").c_int64
    n = lib.tc_kernel_launches()
    r = f()
    return r, lib.tc_kernel_launches() - n


@pytest.mark.parametrize("graph,own_graph", [(False, False), (True, False), (True, True)])
def test_handle_alone_again_is_as_before(gpu_lib, graph, own_graph):
    from tracer_code_gb300.ensemble import Ensemble
    p = _case()
    with Simulation(p) as ref:
        ref.set_step_graph(own_graph)
        ref.upload(state.initial_state(p, seed=5))
        steps = [_launches(ref.step) for _ in range(6)]
        sf = ref.download()["SF"]
    ens = Ensemble([p, p], seeds=[5, 6], autotune=False, graph=graph)
    a = ens.sims[0]
    a.set_step_graph(own_graph)
    out = []
    for n in range(6):
        if n in (1, 3):
            rows, cyc, dts = ens.step()
            assert (rows[0], cyc[0], dts[0]) == steps[n][0]
        else:
            r, launches = _launches(a.step)
            assert r == steps[n][0]
            if n in (2, 4, 5):
                assert launches == steps[n][1], n
    assert np.array_equal(a.download()["SF"], sf)
    ens.close()


@pytest.mark.parametrize("graph", [False, True])
def test_ensemble_of_one_is_as_a_handle_alone(gpu_lib, graph):
    from tracer_code_gb300.ensemble import Ensemble
    p = _case()
    with Simulation(p) as ref:
        ref.set_step_graph(graph)
        ref.upload(state.initial_state(p, seed=5))
        steps = [_launches(ref.step) for _ in range(3)]
    ens = Ensemble([p], seeds=[5], autotune=False, graph=graph)
    for n in range(3):
        (rows, cyc, dts), launches = _launches(ens.step)
        assert (rows[0], cyc[0], dts[0]) == steps[n][0]
        if n > 0:
            assert launches == steps[n][1]
    ens.close()
