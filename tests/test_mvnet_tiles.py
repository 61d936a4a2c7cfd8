"""The gradient kernels at the edges of their tiles: fewer rows than one K step,
row counts that leave ragged last steps and ragged splits, one MB (every crop
and window mostly outside the map) and one pair against several.  Oracle and
tolerances as in test_mvnet.py: normwise 2% per tensor, loss within 0.1%."""
import numpy as np
import pytest

from oracle import mvnet_ref as M
from rusty_h264_b200 import mvnet
from test_mvnet import acc, small_batch  # noqa: F401  (acc is the fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,cw,ch", [(1, 16, 16), (3, 16, 48), (1, 304, 272), (4, 208, 112)])
def test_gradient_tiles(acc, P, cw, ch):  # noqa: F811
    net = mvnet.MvNet(acc, seed=21 + P)
    b = small_batch(acc, P, cw, ch, seed=11 + P)
    g, loss = net.grads(b["pairs"].data_ptr(), P, cw, ch, b["d_nmv"].data_ptr(), b["d_lab"].data_ptr())
    g = g.cpu().numpy().astype(np.float64)
    wl, wg, _ = M.loss_and_grads(net.params(), b["x0"], b["nmv"].astype(np.int64), b["lab"].astype(np.int64))
    assert abs(float(loss.item()) - wl) <= 1e-3 * abs(wl)
    o = 0
    for name, shp in M.SHAPES:
        k = int(np.prod(shp))
        assert np.linalg.norm(g[o:o + k] - wg[o:o + k]) <= 2e-2 * np.linalg.norm(wg[o:o + k]), name
        o += k
    net.close()
