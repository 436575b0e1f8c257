"""Weight gradients on the tensor cores (k_wgrad.cu) at the sizes where its tiles
change: the narrowest images (16-pixel rows at the coarsest level, four rows a
tile), one split and several, image rows of one and of many tiles, odd batches.

The whole network's gradient is compared with the oracle's, which rounds every
stored activation to BF16 as the GPU does and sums in float64: the bounds are those
of test_gpu_nn.py (BF16 roundings that fall the other way dominate), per layer and
in all.  The bias gradients, summed in another kernel, are held to the same.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import nn_oracle as nno
from tests.test_gpu_nn import make_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,H,W", [(1, 64, 128), (3, 64, 128), (1, 32, 256), (1, 16, 512), (1, 16, 1024), (5, 32, 256)])
def test_gradients_match_oracle(gpu_lib, nb, H, W):
    from tracer_code_gb300.learned import Net
    raw, sf_new = make_batch(H + W + nb, nb, H, W)
    net = Net(nb, H, W, seed=4)
    params = net.get_params()
    rd, sd = torch.from_numpy(raw).cuda(), torch.from_numpy(sf_new).cuda()
    loss = net.loss_backward(rd.data_ptr(), sd.data_ptr(), nb)
    g = net.get_grads().astype(np.float64)
    # a second pass gives the same bits (fixed summation order)
    net.loss_backward(rd.data_ptr(), sd.data_ptr(), nb)
    assert np.array_equal(net.get_grads().astype(np.float64), g)
    lo, go, _ = nno.loss_and_grads(params, raw, sf_new)
    assert abs(loss - lo) <= 1e-3 * lo
    assert np.linalg.norm(g - go) <= 3e-2 * np.linalg.norm(go)
    for l, (w, b, cout, cin) in enumerate(nno.param_layout()[0]):
        for lo_, hi_ in ((w, b), (b, b + cout)):
            assert np.linalg.norm(g[lo_:hi_] - go[lo_:hi_]) <= 0.1 * np.linalg.norm(go[lo_:hi_]) + 1e-12, (l, lo_)
    net.close()
