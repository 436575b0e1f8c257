"""The running sums of stats at the edges of their chunks.

Sums of 128 trapezoids a chunk, one chunk less and more, single chunks and remainders:
every entry of the row that no transcendental function precedes equals the oracle's.
"""
import numpy as np
import pytest

from oracle.pyoracle import Oracle
from tracer_code_gb300 import Simulation
from tests.cases import case_1024_like, fresh_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz", [(32, 128), (128, 32), (136, 120), (248, 136), (264, 40), (40, 264)])
def test_rows_equal_oracle(gpu_lib, nx, nz):
    p = case_1024_like(nx=nx, nz=nz, tpc=5, grids=3)
    p.aspect = nx / nz
    st = fresh_state(p, seed=nx + nz)
    st["SF"] = np.random.default_rng(nz).standard_normal(st["T"].shape)
    g, o = Simulation(p), Oracle(p)
    rows = []
    for s in (g, o):
        s.upload(st)
        s.compute_velocities()
        rows.append(s.stats())
    assert (g.nx, g.nz) == (nx, nz)
    for name in ("vrms", "mobility", "Tavg", "Nu", "Nu_bot", "q1", "q2", "q3", "q4", "tracer_min", "tracer_max"):
        assert rows[0][name] == rows[1][name], name
    assert list(rows[0]["Cavg"]) == list(rows[1]["Cavg"]) and list(rows[0]["ent"]) == list(rows[1]["ent"])
    g.close()
