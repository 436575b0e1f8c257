"""Give-up exits that no other test reaches: the banded coarse substitution
(k_coarse_solve) and the network's weight gradients (k_wgrad).

The switches of test_gpu_timeouts.py make their waits give up after a short bounded poll.
Two-level FP64 solves on 1000x8 and 1000x10 cells have no fused visit and a coarse band that
one CTA factors (kl = 10 and 12), so the substitution's is the only wait in them; its other
row count, kl > 240, comes after a factorisation that gives up as well.  A backward pass
reports the wait; with the switch off its gradients are those of a fresh network.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from tracer_code_gb300 import Simulation, TracerError
from tests.cases import case_1024_like, fresh_state
from tests.test_gpu_nn import make_batch

pytestmark = pytest.mark.gpu

TIMEOUT = 13  # TC_ERR_DEVICE_TIMEOUT


@pytest.mark.parametrize("prec,nx,nz", [(0, 1000, 8), (1, 1000, 10), (0, 36, 242)])
def test_coarse_solve_gives_up_then_handle_solves(gpu_lib, prec, nx, nz):
    p = case_1024_like(nx=nx, nz=nz, grids=2, tpc=1, Ra=1.0e4, visT=10.0)
    p.solver_precision, p.aspect, p.max_cycles = prec, nx / nz, 200
    st = fresh_state(p, seed=nx)
    with Simulation(p) as f:
        f.upload(st)
        c_ref, sf_ref = f.multigrid(), f.download()["SF"]
    with Simulation(p) as g:
        g.upload(st)
        g.debug_wait_test(True)
        with pytest.raises(TracerError) as e:
            g.multigrid()
        assert e.value.status == TIMEOUT
        g.debug_wait_test(False)
        assert g.multigrid() == c_ref
        assert np.array_equal(g.download()["SF"], sf_ref)


def test_backward_gives_up_then_gradients_are_right(gpu_lib):
    from tracer_code_gb300.learned import Net
    nb, H, W = 2, 64, 128
    raw, sf = make_batch(5, nb, H, W)
    rd, sd = torch.from_numpy(raw).cuda(), torch.from_numpy(sf).cuda()
    ref, net = Net(nb, H, W, seed=4), Net(nb, H, W, seed=4)
    loss_ref = ref.loss_backward(rd.data_ptr(), sd.data_ptr(), nb)
    net.debug_wait_test(True)
    with pytest.raises(TracerError) as e:
        net.loss_backward(rd.data_ptr(), sd.data_ptr(), nb)
    assert e.value.status == TIMEOUT
    net.debug_wait_test(False)
    assert net.loss_backward(rd.data_ptr(), sd.data_ptr(), nb) == loss_ref
    assert np.array_equal(net.get_grads(), ref.get_grads())
    net.close()
    ref.close()
