"""The searches, planes, grids, lookahead and deblocking at the sizes where
their kernels change path: motion past the search window and off the planes,
unaligned sources, rates beyond the rate table, band lengths, tile remainders,
one-column and one-row pictures.  Integer work, bit-exact with the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from rusty_h264_b200 import accel as A

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def acc():
    a = A.Accel(0)
    yield a
    a.close()


def dev(acc, a):
    return acc.to_dev(np.ascontiguousarray(a))


def texture(rng, h, w):
    t = rng.random((h, w))
    for _ in range(4):  # smooth, so that a search can follow the motion
        t = (t + np.roll(t, 1, 0) + np.roll(t, 1, 1) + np.roll(t, (1, 1), (0, 1))) / 4
    return (255 * (t - t.min()) / (t.max() - t.min())).astype(np.uint8)


def synthetic_picks(rng, nmb):
    picks = np.zeros((nmb, 6), np.int32)
    picks[:, 0] = rng.integers(0, 3, nmb)
    picks[:, 1:3] = rng.integers(-9, 10, (nmb, 2))
    picks[:, 3:5] = np.where(picks[:, :1] == 0, picks[:, 1:3], picks[:, 1:3] + rng.integers(-4, 5, (nmb, 2)))
    return picks


@pytest.mark.parametrize("pan,pad,off,lam,frames", [
    ((0, 0), 32, 1, 12.0, 1),  # a source that is not word-aligned, the few-frames launch
    ((9, -6), 32, 2, 9.0, 4),
    ((38, -29), 32, 0, 10.0, 3),  # past the window
    ((38, 31), 3, 0, 10.0, 1),  # past the window and off the planes' narrow padding
    ((-70, 52), 12, 3, 4.0, 3),
    ((9, -6), 32, 0, 8388607.0, 2),  # the largest lambda of the integer rate table
    ((9, -6), 32, 0, 8388608.0, 3),  # and the first beyond it
])
def test_search_leaves_the_window(acc, pan, pad, off, lam, frames):
    """The seed chain follows a pan per frame; the outer MBs' candidates leave
    the planes.  16-pel ladder and partitions, every shape allowed."""
    rng = np.random.default_rng(abs(pan[0]) + pad + off)
    ch, cw = 96, 176
    my, mx = frames * abs(pan[1]), frames * abs(pan[0])
    tex = texture(rng, ch + 2 * my, cw + 2 * mx)
    clip = [np.ascontiguousarray(tex[my + k * pan[1]:my + k * pan[1] + ch, mx + k * pan[0]:mx + k * pan[0] + cw])
            for k in range(frames + 1)]
    fs, keep, outs = [], [], []
    nmb = (cw // 16) * (ch // 16)
    for k in range(1, frames + 1):
        buf = dev(acc, np.concatenate([np.zeros(off, np.uint8), clip[k].ravel()]))
        pl = acc.hpel_build(dev(acc, clip[k - 1][None]), pad)[0]
        picks, costs = acc.zeros((nmb, 6), acc.torch.int32), acc.zeros((nmb, 2), acc.torch.int64)
        keep += [buf, pl]
        outs.append((picks, costs))
        fs.append(A.MeFrame(A.Picture(buf.data_ptr() + off, pl.data_ptr(), cw, ch, pad), lam, A.split_gate_for_qp(26),
                            picks.data_ptr(), costs.data_ptr()))
    acc.me_frames(fs, A.default_me_params())
    acc.sync()
    for k in range(1, frames + 1):
        wp, wc = O.me_frame(clip[k], clip[k - 1], O.build_planes4(clip[k - 1], pad), O.balanced_params(), lam,
                            A.split_gate_for_qp(26), pad=pad)
        assert np.array_equal(outs[k - 1][0].cpu().numpy()[:, :5], wp[:, :5]), k
        assert np.array_equal(outs[k - 1][1].cpu().numpy(), wc), k


@pytest.mark.parametrize("cw,ch,pad,n", [(176, 144, 32, 1), (176, 144, 7, 9), (352, 288, 32, 3), (640, 368, 32, 30),
                                         (208, 112, 5, 2), (16, 16, 3, 40)])
def test_hpel_band_lengths(acc, cw, ch, pad, n):
    """Bands of 6, 12 and 24 rows by the size of the call, heights that leave a
    short last band, planes of odd widths."""
    rng = np.random.default_rng(cw + n)
    frames = rng.integers(0, 256, (n, ch, cw)).astype(np.uint8)
    got = acc.hpel_build(dev(acc, frames), pad=pad)
    acc.sync()
    for i in {0, n // 2, n - 1}:
        assert np.array_equal(got[i].cpu().numpy(), O.build_planes4(frames[i], pad)), i


@pytest.mark.parametrize("w,h,chroma,n", [(48, 112, True, 2), (16, 128, False, 1), (32, 144, True, 3), (6400, 48, False, 1),
                                          (16, 16, True, 70), (160, 272, False, 2)])
def test_deblock_row_groups(acc, w, h, chroma, n):
    """7, 8, 9 and 17 MB rows in groups of eight, one-column pictures, a picture
    wide enough for fewer rows per group, luma only, more pictures than one
    launch takes."""
    rng = np.random.default_rng(w + h)
    qp, nmb = 33, (w // 16) * (h // 16)
    frames, keep, cases = [], [], []
    for f in range(n):
        src, ref = texture(rng, h, w), texture(rng, h, w)
        picks = synthetic_picks(rng, nmb)
        coeffs, rec = O.mc_tq_rec_frame(src, ref, picks, qp, 6)
        ru = rv = None
        if chroma:
            a, b = O.downsample2x(src), O.downsample2x(ref)
            _, ru, rv = O.mc_tq_chroma_frame(a, 255 - a, b, 255 - b, picks, qp)
        d = [dev(acc, x) if x is not None else None for x in (rec, ru, rv, picks, coeffs)]
        keep += d
        cases.append((d, rec, ru, rv, picks, coeffs))
        frames.append(A.DeblockFrame(d[0].data_ptr(), d[1].data_ptr() if chroma else None,
                                     d[2].data_ptr() if chroma else None, w, h, d[3].data_ptr(), d[4].data_ptr(), qp, 0,
                                     0, 0))
    acc.deblock_frames(frames)
    acc.sync()
    for k, (d, rec, ru, rv, picks, coeffs) in enumerate(cases):
        wy, wu, wv = O.deblock_frame(rec, ru, rv, picks, coeffs, qp)
        assert np.array_equal(d[0].cpu().numpy(), wy), k
        if chroma:
            assert np.array_equal(d[1].cpu().numpy(), wu) and np.array_equal(d[2].cpu().numpy(), wv), k


@pytest.mark.parametrize("R,checked", [(1, 6), (2, 6), (5, 4), (11, 2), (12, 2), (24, 1), (33, 1), (64, 1)])
def test_satd_grid_stages(acc, R, checked):
    """SATD grid and argmin where a stage's phases and runs change: one run and
    all phases (small R), several runs, a last run that is nearly empty, one run
    per stage (R = 64)."""
    rng = np.random.default_rng(R)
    cw, ch, pad = 48, 32, 32
    src, ref = texture(rng, ch, cw), texture(rng, ch, cw)
    planes = O.build_planes4(ref, pad)
    d_src, d_pl = dev(acc, src), dev(acc, planes)
    pic = A.Picture(d_src.data_ptr(), d_pl.data_ptr(), cw, ch, pad)
    nmb, n, lam, tab = 6, 2 * R + 1, 3.25, O.mv_cost_table()
    centers = rng.integers(-64, 65, (nmb, 2)).astype(np.int32)
    pmv = rng.integers(-64, 65, (nmb, 2)).astype(np.int32)
    _, satd, best = acc.fullpel_grid(pic, R, dev(acc, centers), dev(acc, pmv), 1, 1, dev(acc, tab), lam)
    acc.sync()
    satd, best = satd.cpu().numpy(), best.cpu().numpy()
    for m in range(nmb - checked, nmb):
        cx, cy = (centers[m] + 2) >> 2
        lead = None
        for i in range(n * n):  # raster order, strict <
            mvx, mvy = int(cx + i % n - R) * 4, int(cy + i // n - R) * 4
            d = O.candidate_dist(src, ref, planes, 0, (m % 3) * 16, (m // 3) * 16, 16, 16, mvx, mvy)
            assert satd[m, i] == d, (m, i)
            rate = O.lib().or_mvbits(1, O.ptr(tab, O.u16p), mvx - int(pmv[m, 0])) + \
                O.lib().or_mvbits(1, O.ptr(tab, O.u16p), mvy - int(pmv[m, 1]))
            c = int(d) + int(lam * rate)
            if lead is None or c < lead[2]:
                lead = [mvx, mvy, c, int(d)]
        assert best[m].tolist() == lead, m


@pytest.mark.parametrize("cw,ch,pan", [(16, 64, (0, 3)), (32, 48, (5, 0)), (64, 16, (-6, 2)), (96, 80, (17, -9)),
                                       (160, 128, (0, 0)), (416, 96, (40, 7))])
def test_lookahead_small_and_odd_pictures(acc, cw, ch, pan):
    """HalfRes chains of one column, one row, odd and even column counts (two
    columns share a window) and pictures smaller than a window, on noise and on
    a panning texture."""
    rng = np.random.default_rng(cw * 7 + ch)
    tex = texture(rng, ch + 3 * abs(pan[1]) + 8, cw + 3 * abs(pan[0]) + 8)
    oy, ox = (3 * abs(pan[1]) if pan[1] < 0 else 0), (3 * abs(pan[0]) if pan[0] < 0 else 0)
    clip = np.stack([tex[oy + k * pan[1]:oy + k * pan[1] + ch, ox + k * pan[0]:ox + k * pan[0] + cw] for k in range(3)] +
                    [rng.integers(0, 256, (ch, cw)).astype(np.uint8) for _ in range(2)])
    clip = np.ascontiguousarray(clip)
    full = dev(acc, clip)
    half = acc.downsample2x(full)
    intra, inter, mvs = acc.lookahead_costs(full, half, 2)
    acc.sync()
    assert np.array_equal(half.cpu().numpy(), np.stack([O.downsample2x(f) for f in clip]))
    wi, wn, wm = O.lookahead_clip(clip, 2)
    assert np.array_equal(intra.cpu().numpy(), wi)
    assert np.array_equal(inter.cpu().numpy(), wn)
    assert np.array_equal(mvs.cpu().numpy(), wm)
