"""The SATD grid's argmin where the rate is no bound on the cost."""
import numpy as np
import pytest

from rusty_h264_b200 import accel as A
from test_gpu_edges import dev
from test_gpu_presets import acc  # noqa: F401  (acc is the fixture)

pytestmark = pytest.mark.gpu


def test_first_of_equal_costs_at_infinite_lambda(acc):  # noqa: F811
    """Every cost is the saturated rate (it wraps below the distortion) and the
    picture repeats every three rows, so rows 1, 4, 7, ... of a column tie: the
    first in raster order wins."""
    R, pad, n = 32, 64, 65
    rng = np.random.default_rng(1)
    rows = rng.integers(0, 256, (3, 48)).astype(np.uint8)
    ref = rows[np.arange(48) % 3]
    src = np.zeros_like(ref)
    x0, y0 = 16, 16
    src[y0:y0 + 16, x0:x0 + 16] = rows[(y0 + 1 + np.arange(16)) % 3][:, x0:x0 + 16]  # matches rows dy = 1 (mod 3)
    d_ref = acc.hpel_build(dev(acc, ref[None]), pad)[0]
    d_src = dev(acc, src)
    zero = acc.zeros((9, 2), acc.torch.int32)
    _, satd, best = acc.fullpel_grid(A.Picture(d_src.data_ptr(), d_ref.data_ptr(), 48, 48, pad), R, zero, zero, 1, 0,
                                     None, float("inf"))
    acc.sync()
    g = satd.cpu().numpy()[4].reshape(n, n)
    first = int(np.flatnonzero(g.ravel() == g.min())[0])
    assert g.min() == 0 and (g == 0).sum() > 1
    want = [(first % n - R) * 4, (first // n - R) * 4]
    assert best.cpu().numpy()[4, :2].tolist() == want
