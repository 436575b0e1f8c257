"""The FP32 build of the bottom matrix at the shapes of its two forms.

Levels of 63x15, 55x17 and 31x31 points take two points a thread (the last strip of a
column shares one with the strip before), 93x11 one.  As test_gpu_subcycle.py requires of
the mixed solve: the W-cycles with the matrix within 15% of those with the sweeps, and the
oracle's convergence test met.
"""
import pytest

from tracer_code_gb300 import Simulation
from tests.cases import fresh_state
from tests.test_gpu_subcycle import _case, _oracle_ratio

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz", [(256, 64), (224, 72), (128, 128), (376, 48)])
def test_mixed_solve_with_matrix(gpu_lib, nx, nz):
    def case(matrix):
        p = _case(1, matrix, nx, nz, 4)
        p.aspect = nx / nz
        return p

    st = fresh_state(case(0), seed=nz)
    res = {}
    for m in (0, 1):
        g = Simulation(case(m))
        g.upload(st)
        res[m] = (g.multigrid(), g.download()["SF"])
        g.close()
    assert abs(res[1][0] - res[0][0]) <= 0.15 * res[0][0] + 1, (res[0][0], res[1][0])
    assert _oracle_ratio(case(1), st, res[1][1]) <= case(1).tolerance
