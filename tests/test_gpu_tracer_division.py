"""Tracer stages on grids whose spacings are no powers of two.

The stages divide by ds through quot_round (k_tracer.cu: Newton corrections of the
product with the rounded reciprocal); on a power-of-two ds they multiply.  Given
identical velocities, positions, counts, composition and temperature must equal the
oracle's bit for bit, as test_gpu_parity.py requires on power-of-two grids.
"""
import numpy as np
import pytest

from oracle.pyoracle import Oracle
from tracer_code_gb300 import Simulation
from tests.cases import case_1024_like, fresh_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz,aspect,tracer", [(72, 24, 3.0, 0), (40, 56, 0.7, 0), (88, 40, 2.2, 1), (64, 96, 1.0, 0)])
def test_stages_equal_oracle(gpu_lib, nx, nz, aspect, tracer):
    p = case_1024_like(nx=nx, nz=nz, tpc=9, grids=3)
    p.aspect, p.RK_update, p.tracer = aspect, 0, tracer
    st = fresh_state(p, seed=nz)
    x = np.arange(-2, nx + 3) / nx
    z = np.arange(-2, nz + 3) / nz
    # cells with a wide range of velocities, 1e-9 of the largest among them
    st["SF"] = np.ascontiguousarray(30.0 * np.sin(np.pi * z)[:, None] ** 3 *
                                    (np.sin(3 * np.pi * x) * np.exp(-18.0 * x))[None, :])
    g, o = Simulation(p), Oracle(p)
    for s in (g, o):
        s.upload(st)
        s.compute_velocities()
    for _ in range(3):
        assert g.energy_time() == o.energy_time()
    a, b = g.download(), o.download()
    for key in a:
        assert np.array_equal(a[key], b[key]), key
    g.close()
