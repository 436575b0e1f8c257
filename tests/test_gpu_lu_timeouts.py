"""The bounded waits of the coarse LU by panels (k_lu_panel): a wait that runs out is
reported by the solve it happened in, and the factors it left are not used again.

The debug switch of test_gpu_timeouts.py makes every wait of the factorisation give up
at once, after a short bounded poll of a word that nothing sets.  On coarse grids whose
bands take the panels' block sizes of 64, 128, 256 and 512 rows the solve returns
TC_ERR_DEVICE_TIMEOUT; with the switch off the same handle then solves as a fresh one
does.  The isoviscous case starts at a time after zero, where a solve takes factors that
an earlier one left: those of the timed-out solve must not be among them.
"""
import numpy as np
import pytest

from tracer_code_gb300 import Simulation, TracerError
from tests.cases import case_1024_like, case_128_like, fresh_state

pytestmark = pytest.mark.gpu

TIMEOUT = 13  # TC_ERR_DEVICE_TIMEOUT


# kl = 2 nz / 2^(grids-1) + 2
@pytest.mark.parametrize("mk,prec,nx,nz,kl", [(case_1024_like, 0, 44, 22, 24), (case_1024_like, 1, 46, 60, 62),
                                              (case_1024_like, 0, 16, 224, 226), (case_1024_like, 0, 16, 300, 302),
                                              (case_128_like, 0, 46, 60, 62), (case_128_like, 1, 92, 92, 94)])
def test_lu_wait_runs_out_then_handle_solves(gpu_lib, mk, prec, nx, nz, kl):
    p = mk(nx=nx, nz=nz, tpc=2, grids=2)
    p.aspect, p.max_cycles = nx / nz, 200
    p.mg_zero_coarse, p.solver_precision = 1, prec
    st = fresh_state(p, seed=nx)

    def make():
        g = Simulation(p)
        g.upload(st)
        g.set_clock(3, 0.01)
        return g

    with make() as f:
        assert f.info.kl == kl
        c_ref = f.multigrid()
        sf_ref = f.download()["SF"]
    with make() as g:
        g.debug_wait_test(True)
        with pytest.raises(TracerError) as e:
            g.multigrid()
        assert e.value.status == TIMEOUT and "LU" in str(e.value)
        g.debug_wait_test(False)
        assert g.multigrid() == c_ref
        assert np.array_equal(g.download()["SF"], sf_ref)
