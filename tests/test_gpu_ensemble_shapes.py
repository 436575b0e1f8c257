"""Launch shapes of levels whose visits run over the whole grid only when the handle is
stepped alone: the shape for ensembles is tuned, returned, applied and used beside it.

Counted in kernel launches (a visit in one launch, in several sweeps per launch, in one
launch per sweep), which depend on the shapes alone as the results do not.
"""
import pytest

from tracer_code_gb300 import Simulation, TracerError, state
from tests.cases import case_1024_like

pytestmark = pytest.mark.gpu

GRID = 10000


def _case(prec=1, nx=512, nz=128):
    p = case_1024_like(nx=nx, nz=nz, grids=5, tpc=3, Ra=1.0e5, visT=100.0)
    p.mg_zero_coarse, p.mg_coarse_matrix, p.solver_precision, p.cycle_correction = 1, 1, prec, 3
    return p


def _step_launches(p, shapes, n):
    """Results and kernel launches of the second step of n equal cases."""
    from tracer_code_gb300.ensemble import Ensemble
    ens = Ensemble([p] * n, seeds=[5] * n, autotune=shapes is None, graph=False)
    if shapes is not None:
        for s in ens.sims:
            s.set_launch_shapes(shapes)
    ens.step()
    before = Simulation.kernel_launches()
    res = ens.step(nthreads=1)
    count = Simulation.kernel_launches() - before
    tuning = ens.tuning
    ens.close()
    return res, count, tuning


def test_the_shape_beside_the_grid_is_used_in_ensembles_only(gpu_lib):
    p = _case()
    rest = [(32, 8, 1)] * 3

    def run(v, n):
        res, count, _ = _step_launches(p, [(32, 8, v)] + rest, n)
        return res[0][0], res[1][0], count

    alone, pair = {}, {}
    for v in (1, 0, 1003, GRID, GRID + 1003):
        row, cyc, alone[v] = run(v, 1)
        row2, cyc2, pair[v] = run(v, 2)
        assert (row, cyc) == (row2, cyc2)
    assert alone[GRID + 1003] == alone[GRID] == alone[1] < alone[1003] < alone[0]
    assert pair[GRID + 1003] == pair[1003] < pair[0]
    assert pair[GRID] == pair[0] == 2 * alone[0]
    assert pair[1003] == 2 * alone[1003]


def test_copied_shapes_are_the_tuned_ones(gpu_lib):
    p = _case()
    res, tuned, tuning = _step_launches(p, None, 2)
    assert tuning[0] == tuning[1]
    res2, copied, _ = _step_launches(p, tuning[0], 2)
    assert res[0] == res2[0] and tuned == copied


@pytest.mark.parametrize("prec,level", [(0, 1), (1, 2)])
def test_levels_without_such_visits_refuse_the_shape(gpu_lib, prec, level):
    p = _case(prec, 256, 64)
    with Simulation(p) as g:
        shapes = [[32, 8, 1] for _ in range(g.info.grids - 1)]
        shapes[level - 1][2] = GRID + 1
        with pytest.raises(TracerError) as e:
            g.set_launch_shapes(shapes)
        assert e.value.status == 1
