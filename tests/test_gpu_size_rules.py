"""The rules that choose a path by the size of a call, each side of each rule
against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from rusty_h264_b200 import accel as A
from test_gpu_edges import dev, texture
from test_gpu_parity import _compare_closed
from test_gpu_presets import O_half, acc, panning  # noqa: F401  (acc is the fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cw,ch,n,rows", [(352, 288, 1, 6), (640, 352, 12, 12), (1920, 1072, 13, 24)])
def test_hpel_bands(acc, cw, ch, n, rows):  # noqa: F811
    """Bands of 6, 12 and 24 rows, the last one short of its rows."""
    pad = 32
    pw, ph = cw + 2 * pad, ch + 2 * pad
    cells = (pw + 119) // 120 * ph * n
    assert rows == (6 if cells < 25000 else (12 if cells < 250000 else 24)) and ph % rows
    frames = np.random.default_rng(rows).integers(0, 256, (n, ch, cw)).astype(np.uint8)
    got = acc.hpel_build(dev(acc, frames), pad=pad)
    acc.sync()
    for i in {0, n // 2, n - 1}:
        assert np.array_equal(got[i].cpu().numpy(), O.build_planes4(frames[i], pad)), i


@pytest.mark.parametrize("mb_w,segw", [(23, 1), (53, 2), (80, 3), (97, 4), (123, 5), (145, 6), (169, 7)])
def test_closed_loop_segment_widths(acc, mb_w, segw):  # noqa: F811
    """Column segments of one to seven MBs, the last one narrower."""
    assert segw == min(max(mb_w // 24, 1), 7) and (segw == 1 or mb_w % segw)
    cw, ch, qp, lam = 16 * mb_w, 48, 28, 8.0
    Y = panning(4, ch + 32, cw, mb_w)[:, 16:16 + ch]
    Y = np.ascontiguousarray(Y)
    U, V = O_half(255 - Y), O_half(Y)
    gate = A.split_gate_for_qp(qp)
    got = acc.pixel_path_closed(Y, U, V, A.default_me_params(), lam, gate, qp)
    _compare_closed(got, O.closed_loop_clip(Y, U, V, O.balanced_params(), lam, gate, qp))


@pytest.mark.parametrize("cw,ch", [(272, 112), (720, 64), (1360, 48), (96, 80), (80, 96), (112, 80)])
def test_lookahead_odd_widths(acc, cw, ch):  # noqa: F811
    """HalfRes pictures an odd number of MBs wide, and pictures about as large as a window."""
    clip = panning(4, ch + 48, cw, cw, 9, 4)[:, 24:24 + ch]
    clip = np.ascontiguousarray(clip)
    full = dev(acc, clip)
    half = acc.downsample2x(full)
    got = acc.lookahead_costs(full, half, 2)
    acc.sync()
    for g, w in zip(got, O.lookahead_clip(clip, 2)):
        assert np.array_equal(g.cpu().numpy(), w)
