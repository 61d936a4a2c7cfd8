"""Picks whose MVs do not fit 16 bits: the proposals of the learned calls are the
caller's, and one far outside the picture wins where a block is as flat as the
picture's corner.  Its neighbours predict from the whole MV."""
import numpy as np
import pytest

from oracle import oracle as O
from rusty_h264_b200 import accel as A
from test_gpu_edges import dev, texture
from test_gpu_parity import _closed_buffers, _closed_result, _compare_closed
from test_gpu_presets import O_half, acc  # noqa: F401  (acc is the fixture)

pytestmark = pytest.mark.gpu

W, H, NMB, QP, LAM = 160, 96, 60, 28, 2.0
GATE = A.split_gate_for_qp(QP)
CORNERS = {(-1, -1): 40, (1, -1): 90, (-1, 1): 150, (1, 1): 215}


def scene(rng, n):
    """Textures with four corner values; a third of the MBs of frames 1.. flat at one of them."""
    clip = np.stack([texture(rng, H, W) for _ in range(n)])
    for f in clip:
        f[:32, :32], f[:32, -32:], f[-32:, :32], f[-32:, -32:] = (CORNERS[k] for k in ((-1, -1), (1, -1), (-1, 1), (1, 1)))
    props = rng.integers(-8, 9, (n, NMB, 16)).astype(np.int32) * 4
    for f in range(1, n):
        for m in rng.permutation(NMB)[:20]:
            sx, sy = rng.choice([-1, 1], 2)
            y, x = 16 * (m // 10), 16 * (m % 10)
            clip[f, y:y + 16, x:x + 16] = CORNERS[(sx, sy)]
            k = rng.integers(0, 8)
            props[f, m, 2 * k] = sx * int(rng.choice([32764, 32767, 32768, 32769, 40001, 65534, 131074]))
            props[f, m, 2 * k + 1] = sy * int(rng.choice([600, 32768, 50003, 70000]))
    return clip, props


@pytest.mark.parametrize("frames", [1, 4])
def test_learned_frames(acc, frames):  # noqa: F811
    clip, props = scene(np.random.default_rng(frames), frames + 1)
    d, d_props = dev(acc, clip), dev(acc, props)
    planes = acc.hpel_build(d[:-1], 32)
    pk, co = acc.zeros((frames, NMB, 6), acc.torch.int32), acc.zeros((frames, NMB, 2), acc.torch.int64)
    acc.me_frames_learned([A.MeLearnedFrame(
        A.MeFrame(A.Picture(d[f + 1].data_ptr(), planes[f].data_ptr(), W, H, 32), LAM, GATE, pk[f].data_ptr(),
                  co[f].data_ptr()), d_props[f + 1].data_ptr(), 1 << 30, None) for f in range(frames)],
        A.default_me_params())
    acc.sync()
    far = 0
    for f in range(frames):
        wp, wc, _ = O.me_frame_learned(clip[f + 1], clip[f], O.build_planes4(clip[f], 32), O.balanced_params(), LAM,
                                       props[f + 1], 1 << 30, GATE)
        assert np.array_equal(pk[f].cpu().numpy()[:, :5], wp[:, :5]), f
        assert np.array_equal(co[f].cpu().numpy(), wc), f
        far += int((np.abs(wp[:, 1:5]) > 32767).any(1).sum())
    assert far >= 5 * frames


def test_learned_step(acc):  # noqa: F811
    """The step's predictors and edge strengths."""
    Y, props = scene(np.random.default_rng(9), 4)
    U, V = O_half(255 - Y), O_half(Y)
    want = O.closed_loop_clip(Y, U, V, O.balanced_params(), LAM, GATE, QP, props=props, prop_t=1 << 30)
    assert (np.abs(want["picks"][..., 1:5]) > 32767).any(2).sum() >= 15
    b, d_props = _closed_buffers(acc, Y, U, V), dev(acc, props)
    for f in range(1, 4):
        acc._check(acc.L.h264a_hpel_build(acc.ctx, b["ry"][f - 1].data_ptr(), W, H, 32, 1, W * H,
                                          b["planes"].data_ptr(), acc._stream()))
        me = A.MeFrame(A.Picture(b["y"][f].data_ptr(), b["planes"].data_ptr(), W, H, 32), LAM, GATE,
                       b["picks"][f].data_ptr(), b["costs"][f].data_ptr())
        acc.closed_step(A.ClosedStep(me, b["u"][f].data_ptr(), b["v"][f].data_ptr(), b["ru"][f - 1].data_ptr(),
                                     b["rv"][f - 1].data_ptr(), b["ry"][f].data_ptr(), b["ru"][f].data_ptr(),
                                     b["rv"][f].data_ptr(), b["coeffs"][f].data_ptr(), b["ccoeffs"][f].data_ptr(),
                                     QP, 6, d_props[f].data_ptr(), None, 1 << 30), A.default_me_params())
    acc.sync()
    _compare_closed(_closed_result(b), want)
