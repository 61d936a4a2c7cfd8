"""Every preset knob through the frame searches (which run all but the Balanced
preset in an instance of their own), and some presets each through the step, the closed
loop, the learned and the multi-reference calls.  Bit-exact with the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from rusty_h264_b200 import accel as A
from test_gpu_edges import dev, texture
from test_gpu_parity import _closed_buffers, _closed_result, _compare_closed, me_variants, oracle_params

pytestmark = pytest.mark.gpu

VARIANTS = me_variants()
KNOBS = {name: (ov, tab) for name, ov, tab in VARIANTS}
LAM, QP = 9.0, 29
GATE = A.split_gate_for_qp(QP)


@pytest.fixture(scope="module")
def acc():
    a = A.Accel(0)
    yield a
    a.close()


def preset(acc, name):
    ov, tab = KNOBS[name]
    tab = O.mv_cost_table() if tab is None else tab
    params = A.default_me_params(**ov)
    d_tab = dev(acc, tab)
    params.d_mv_cost_tab = d_tab.data_ptr()
    return params, oracle_params(ov), tab, d_tab


def panning(n, ch, cw, seed, vx=5, vy=-3):
    """A texture panning by (vx, vy), a patch that moves against it, noise."""
    rng = np.random.default_rng(seed)
    my, mx = n * abs(vy), n * abs(vx)
    tex, patch = texture(rng, ch + 2 * my, cw + 2 * mx), texture(rng, 40, 56)
    out = []
    for k in range(n):
        f = tex[my + k * vy:my + k * vy + ch, mx + k * vx:mx + k * vx + cw].astype(np.int32)
        f[20 + 2 * k:20 + 2 * k + 40, 30 + 3 * k:30 + 3 * k + 56] = patch[:min(40, ch - 20 - 2 * k), :min(56, cw - 30 - 3 * k)]
        out.append(np.clip(f + rng.integers(-3, 4, f.shape), 0, 255).astype(np.uint8))
    return np.stack(out)


@pytest.mark.parametrize("frames", [1, 3])
@pytest.mark.parametrize("name", list(KNOBS))
def test_frame_searches(acc, name, frames):
    params, op, tab, keep = preset(acc, name)
    clip = panning(frames + 1, 112, 176, 3 + frames)
    d = dev(acc, clip)
    planes = acc.hpel_build(d[:-1], 32)
    nmb = 7 * 11
    pk, co = acc.zeros((frames, nmb, 6), acc.torch.int32), acc.zeros((frames, nmb, 2), acc.torch.int64)
    acc.me_frames([A.MeFrame(A.Picture(d[f + 1].data_ptr(), planes[f].data_ptr(), 176, 112, 32), LAM, GATE,
                             pk[f].data_ptr(), co[f].data_ptr()) for f in range(frames)], params)
    acc.sync()
    for f in range(frames):
        wp, wc = O.me_frame(clip[f + 1], clip[f], O.build_planes4(clip[f], 32), op, LAM, GATE, tab=tab)
        assert np.array_equal(pk[f].cpu().numpy()[:, :5], wp[:, :5]), f
        assert np.array_equal(co[f].cpu().numpy(), wc), f


@pytest.mark.parametrize("name", ["sadfp_smooth", "fast_satd", "sp_fc_walk"])
@pytest.mark.parametrize("prop_t", [200, 1 << 30])
def test_learned_search(acc, name, prop_t):
    params, op, tab, keep = preset(acc, name)
    clip = panning(4, 96, 160, 21)
    d = dev(acc, clip)
    planes = acc.hpel_build(d[:-1], 32)
    nmb = 60
    props = np.random.default_rng(5).integers(-8, 9, (3, nmb, 16)).astype(np.int32) * 4
    props[:, :, 4:6] = (20, -12)  # the pan
    d_props = dev(acc, props)
    pk, co = acc.zeros((3, nmb, 6), acc.torch.int32), acc.zeros((3, nmb, 2), acc.torch.int64)
    fb = acc.zeros((3, nmb), acc.torch.int32)
    acc.me_frames_learned([A.MeLearnedFrame(
        A.MeFrame(A.Picture(d[f + 1].data_ptr(), planes[f].data_ptr(), 160, 96, 32), LAM, GATE, pk[f].data_ptr(),
                  co[f].data_ptr()), d_props[f].data_ptr(), prop_t, fb[f].data_ptr()) for f in range(3)], params)
    acc.sync()
    for f in range(3):
        wp, wc, wf = O.me_frame_learned(clip[f + 1], clip[f], O.build_planes4(clip[f], 32), op, LAM, props[f], prop_t,
                                        GATE, tab=tab)
        assert np.array_equal(fb[f].cpu().numpy(), wf), f
        assert np.array_equal(pk[f].cpu().numpy()[:, :5], wp[:, :5]), f
        assert np.array_equal(co[f].cpu().numpy(), wc), f


@pytest.mark.parametrize("name", ["sadfp_smooth", "fast_satd", "walk_to_convergence"])
def test_multi_reference_search(acc, name):
    params, op, tab, keep = preset(acc, name)
    clip = panning(5, 96, 160, 33)
    d = dev(acc, clip)
    planes = acc.hpel_build(d, 32)
    pn = np.stack([O.build_planes4(f, 32) for f in clip])
    nmb, jobs = 60, [(4, [3, 2, 1]), (3, [2, 1]), (2, [0])]
    pk, co = acc.zeros((3, nmb, 8), acc.torch.int32), acc.zeros((3, nmb, 2), acc.torch.int64)
    fr = []
    for i, (s, refs) in enumerate(jobs):
        m = A.MeMrFrame()
        m.d_src, m.nref, m.cw, m.ch, m.pad = d[s].data_ptr(), len(refs), 160, 96, 32
        for k, r in enumerate(refs):
            m.d_planes[k] = planes[r].data_ptr()
        m.lambda_me, m.split_gate, m.d_picks, m.d_costs = LAM, GATE, pk[i].data_ptr(), co[i].data_ptr()
        fr.append(m)
    acc.me_frames_multiref(fr, params)
    acc.sync()
    for i, (s, refs) in enumerate(jobs):
        wp, wc = O.me_frame_multiref(clip[s], clip[refs], pn[refs], op, LAM, GATE, tab=tab)
        assert np.array_equal(pk[i].cpu().numpy()[:, :7], wp[:, :7]), i
        assert np.array_equal(co[i].cpu().numpy(), wc), i


def yuv(n, ch, cw, seed):
    y = panning(n, ch, cw, seed)
    return y, O_half(255 - y), O_half(y)


def O_half(y):
    return np.stack([O.downsample2x(np.ascontiguousarray(f)) for f in y])


@pytest.mark.parametrize("name", ["sadfp_smooth", "fast_satd", "sp_fc_walk"])
def test_closed_loop_and_step(acc, name):
    params, op, tab, keep = preset(acc, name)
    Y, U, V = yuv(5, 96, 176, 41)
    want = O.closed_loop_clip(Y, U, V, op, LAM, GATE, QP, tab=tab)
    _compare_closed(acc.pixel_path_closed(Y, U, V, params, LAM, GATE, QP, tab=tab), want)
    b = _closed_buffers(acc, Y, U, V)
    for f in range(1, 5):
        acc._check(acc.L.h264a_hpel_build(acc.ctx, b["ry"][f - 1].data_ptr(), 176, 96, 32, 1, 176 * 96,
                                          b["planes"].data_ptr(), acc._stream()))
        me = A.MeFrame(A.Picture(b["y"][f].data_ptr(), b["planes"].data_ptr(), 176, 96, 32), LAM, GATE,
                       b["picks"][f].data_ptr(), b["costs"][f].data_ptr())
        acc.closed_step(A.ClosedStep(me, b["u"][f].data_ptr(), b["v"][f].data_ptr(), b["ru"][f - 1].data_ptr(),
                                     b["rv"][f - 1].data_ptr(), b["ry"][f].data_ptr(), b["ru"][f].data_ptr(),
                                     b["rv"][f].data_ptr(), b["coeffs"][f].data_ptr(), b["ccoeffs"][f].data_ptr(),
                                     QP, 6, None, None, 0), params)
    acc.sync()
    _compare_closed(_closed_result(b), want)


def test_learned_closed_loop(acc):
    from rusty_h264_b200 import mvnet

    params, op, tab, keep = preset(acc, "sadfp_smooth")
    Y, U, V = yuv(5, 96, 176, 43)
    net = mvnet.MvNet(acc, seed=3)
    got = acc.pixel_path_closed(Y, U, V, params, LAM, GATE, QP, net=net, fallback_t=100, tab=tab)
    want = O.closed_loop_clip(Y, U, V, op, LAM, GATE, QP, props=got["props"], prop_t=100, tab=tab)
    _compare_closed(got, want)
    assert np.array_equal(got["fallback"], want["fallback"])
    net.close()


@pytest.mark.parametrize("learned", [False, True])
def test_frames_alone_and_together(acc, learned):
    """A frame alone (its own work queue, the fewest CTAs) and the same frames
    in one call, interleaved: every frame of both as the oracle has it."""
    clip = panning(5, 128, 208, 51)
    d = dev(acc, clip)
    planes = acc.hpel_build(d[:-1], 32)
    nmb, params = 104, A.default_me_params()
    props = np.random.default_rng(7).integers(-8, 9, (4, nmb, 16)).astype(np.int32) * 4
    d_props = dev(acc, props)
    for together in (True, False):
        pk, co = acc.zeros((4, nmb, 6), acc.torch.int32), acc.zeros((4, nmb, 2), acc.torch.int64)
        fb = acc.zeros((4, nmb), acc.torch.int32)
        fr = [A.MeLearnedFrame(A.MeFrame(A.Picture(d[f + 1].data_ptr(), planes[f].data_ptr(), 208, 128, 32), LAM, GATE,
                                         pk[f].data_ptr(), co[f].data_ptr()), d_props[f].data_ptr(), 200,
                               fb[f].data_ptr()) for f in range(4)]
        for call in [fr] if together else [[x] for x in fr]:
            if learned:
                acc.me_frames_learned(call, params)
            else:
                acc.me_frames([x.me for x in call], params)
        acc.sync()
        for f in range(4):
            pl = O.build_planes4(clip[f], 32)
            if learned:
                wp, wc, wf = O.me_frame_learned(clip[f + 1], clip[f], pl, O.balanced_params(), LAM, props[f], 200, GATE)
                assert np.array_equal(fb[f].cpu().numpy(), wf), (together, f)
            else:
                wp, wc = O.me_frame(clip[f + 1], clip[f], pl, O.balanced_params(), LAM, GATE)
            assert np.array_equal(pk[f].cpu().numpy()[:, :5], wp[:, :5]), (together, f)
            assert np.array_equal(co[f].cpu().numpy(), wc), (together, f)
