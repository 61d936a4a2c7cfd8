"""Cases of the encoder pixel path whose speed is followed: what an encoder has
this library do, through its public entry points, on seeded synthetic clips.

Each case is a dict of plain values; ``prepare`` builds what the caller has in
hand (clips, buffers, a network, a batch handle), ``run`` is one pass through
the entry points, ``work`` the bytes and operations a pass cannot do without,
and ``exact`` the float outputs (the proposal network's) in 64 bits.

The clips have the statistics of rusty_h264_b200/synth.py's 1080p workload (a
panning textured background with sub-pixel detail, textured rectangles at
quarter-pel velocities, sensor noise), generated on the GPU at any size.
"""
import ctypes as C

import numpy as np
import torch
import torch.nn.functional as F

from rusty_h264_b200 import accel as A
from rusty_h264_b200 import mvnet

DEV = "cuda:0"
PAD = 32
DZ = 6
NPARAMS = mvnet.NPARAMS
_acc = None


def acc():
    """The process's library context (an encoder keeps one)."""
    global _acc
    if _acc is None:
        _acc = A.Accel(0)
    return _acc


# ---- the cases ----------------------------------------------------------------

def listed():
    return [
        # the encoder's main loop over a 1080p clip: every P frame searched, predicted and
        # reconstructed against the deblocked reconstruction of the one before
        {"name": "closed_1080p", "kind": "closed", "w": 1920, "h": 1080, "n": 60, "qp": 27, "learned": False},
        # the same from and to host buffers, for a small clip
        {"name": "closed_host_cif", "kind": "closed_host", "w": 352, "h": 288, "n": 30, "qp": 26},
        # the loop with the learned proposals (lookahead for the guide MVs, network, learned search)
        {"name": "closed_learned_720p", "kind": "closed", "w": 1280, "h": 720, "n": 24, "qp": 32, "learned": True},
        # one P frame at a time, as a live encoder codes it: planes, then the fused step
        {"name": "step_720p", "kind": "step", "w": 1280, "h": 720, "qp": 27},
        # plain motion estimation of several streams of uneven size at once, with MC + T/Q of the picks
        {"name": "path_mixed", "kind": "path", "streams": "352x288,352x288,1280x720,1280x720,1920x1080", "n": 16,
         "qp": 27},
        # two GOP steps of such streams over three references through the batched runtime
        {"name": "batch_mixed", "kind": "batch", "streams": "352x288,352x288,1280x720,1920x1080", "g": 8, "nref": 3,
         "qp": 27},
        # the mb-tree lookahead of a 1080p clip at half resolution (the default mode)
        {"name": "lookahead_1080p", "kind": "lookahead", "w": 1920, "h": 1080, "n": 60, "mode": 2},
        # the reconstruction side as separate calls: luma, chroma, deblocking
        {"name": "recon_1080p", "kind": "recon", "w": 1920, "h": 1080, "n": 8, "qp": 30},
        # the proposal network's logits of a batch of frame pairs (evaluation, inference)
        {"name": "net_forward", "kind": "forward", "w": 1920, "h": 1080, "n": 4},
        # its gradients, on the batch that training uses
        {"name": "net_grads", "kind": "grads", "w": 1920, "h": 1080, "n": 4},
        # exhaustive SAD and SATD cost grids at +-32 with the argmin
        {"name": "grid_720p", "kind": "grid", "w": 1280, "h": 720, "r": 32},
        # the smallest call: one CIF picture's half-pel planes
        {"name": "hpel_cif", "kind": "hpel", "w": 352, "h": 288, "n": 1},
    ]


def draw(rng):
    """One more case of the same ranges: sizes spread over their logarithm, most of them no multiple of 16."""
    def log(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    def size(max_px=1920 * 1080):
        while True:
            w, h = 2 * log(88, 960), 2 * log(72, 540)
            if w * h <= max_px:
                return w, h

    kind = rng.choice(["closed", "closed_host", "closed", "step", "path", "batch", "lookahead", "recon", "forward",
                       "grads", "grid", "hpel"])
    qp = rng.choice([22, 26, 27, 30, 32, 37])
    w, h = size()
    if kind == "closed":
        return {"kind": kind, "w": w, "h": h, "n": log(4, 40), "qp": qp, "learned": rng.random() < 0.4}
    if kind == "closed_host":
        return {"kind": kind, "w": w, "h": h, "n": log(4, 30), "qp": qp}
    if kind == "step":
        return {"kind": kind, "w": w, "h": h, "qp": qp}
    if kind in ("path", "batch"):
        sizes = [size(1280 * 720) for _ in range(rng.randint(1, 4))]
        s = ",".join("%dx%d" % x for x in sizes)
        if kind == "path":
            return {"kind": kind, "streams": s, "n": log(3, 16), "qp": qp}
        return {"kind": kind, "streams": s, "g": log(2, 8), "nref": rng.randint(1, 4), "qp": qp}
    if kind == "lookahead":
        return {"kind": kind, "w": w, "h": h, "n": log(4, 60), "mode": rng.choice([0, 1, 2, 2, 2])}
    if kind == "recon":
        return {"kind": kind, "w": w, "h": h, "n": log(1, 8), "qp": qp}
    if kind in ("forward", "grads"):
        return {"kind": kind, "w": w, "h": h, "n": rng.randint(1, 4)}
    if kind == "grid":
        w, h = size(1280 * 720)
        return {"kind": kind, "w": w, "h": h, "r": log(4, 32)}
    return {"kind": kind, "w": w, "h": h, "n": log(1, 16)}


# ---- inputs ---------------------------------------------------------------------

def _coded(v):
    return (v + 15) // 16 * 16


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _noise(g, H, W, base):
    """Four octaves of bilinearly interpolated random lattices, in [0, 1]."""
    out = torch.zeros((H, W), device=DEV)
    amp, tot, cell = 1.0, 0.0, base
    for _ in range(4):
        lat = torch.rand((H // cell + 2, W // cell + 2), generator=g, device=DEV)
        yy, xx = torch.arange(H, device=DEV) / cell, torch.arange(W, device=DEV) / cell
        y0, x0 = yy.long(), xx.long()
        fy, fx = (yy - y0)[:, None], (xx - x0)[None, :]
        a, b = lat[y0][:, x0], lat[y0][:, x0 + 1]
        c, d = lat[y0 + 1][:, x0], lat[y0 + 1][:, x0 + 1]
        out += amp * ((a * (1 - fx) + b * fx) * (1 - fy) + (c * (1 - fx) + d * fx) * fy)
        tot += amp
        amp *= 0.5
        cell = max(cell // 2, 1)
    return out / tot


def _tex4(g, H, W, base, lo, span, sigma):
    """A texture at four times the resolution, with sub-pixel detail."""
    t = (lo + span * _noise(g, H, W, base)).repeat_interleave(4, 0).repeat_interleave(4, 1)
    return t + torch.randn(t.shape, generator=g, device=DEV) * sigma


def clip(w, h, n, seed, chroma=False):
    """n frames of luma (n, ch, cw), edge-clamped to whole MBs, and with
    `chroma` the two chroma planes (n, ch/2, cw/2)."""
    g = _gen(seed)
    cw, ch = _coded(w), _coded(h)
    vx4, vy4 = 5, -2
    mx, my = abs(vx4) * n // 4 + 8, abs(vy4) * n // 4 + 8
    tex = _tex4(g, h + 2 * my, w + 2 * mx, 64, 20.0, 215.0, 6.0)
    host = np.random.default_rng(int(seed))
    rects = []
    for _ in range(8):
        rw, rh = int(host.integers(32, min(257, w - 8))), int(host.integers(32, min(257, h - 8)))
        rects.append((rw, rh, _tex4(g, rh + 1, rw + 1, 16, 0.0, 255.0, 12.0), int(host.integers(0, (w - rw) * 4)),
                      int(host.integers(0, (h - rh) * 4)), int(round(host.uniform(-6, 6) * 4)),
                      int(round(host.uniform(-6, 6) * 4))))
    y = torch.empty((n, ch, cw), dtype=torch.uint8, device=DEV)
    rows = torch.arange(ch, device=DEV).clamp(max=h - 1)
    cols = torch.arange(cw, device=DEV).clamp(max=w - 1)

    def down(t, oy, ox, hh, ww):  # the 4x4 box means of t from (oy, ox)
        return F.avg_pool2d(t[oy:oy + 4 * hh, ox:ox + 4 * ww][None, None], 4)[0, 0]

    for t in range(n):
        img = down(tex, my * 4 + vy4 * t, mx * 4 + vx4 * t, h, w)
        for rw, rh, tx, x4, y4, vx, vy in rects:
            px, py = x4 + vx * t, y4 + vy * t
            X, Y = px // 4, py // 4
            x0, y0, x1, y1 = max(X, 0), max(Y, 0), min(X + rw, w), min(Y + rh, h)
            if x1 > x0 and y1 > y0:
                img[y0:y1, x0:x1] = down(tx, py % 4, px % 4, rh, rw)[y0 - Y:y1 - Y, x0 - X:x1 - X]
        img = img + torch.randn((h, w), generator=g, device=DEV) * 1.5
        y[t] = img.round().clamp(0, 255).to(torch.uint8)[rows][:, cols]
    if not chroma:
        return y
    uv = 128 + torch.randn((2, n, ch // 2, cw // 2), generator=g, device=DEV)
    uv = uv.round().clamp(0, 255).to(torch.uint8)
    return y, uv[0].contiguous(), uv[1].contiguous()


def _lam(qp):
    return float(np.sqrt(A.frame_lambda(qp)) * 1.25)


def _zeros(shape, dtype):
    return torch.zeros(shape, dtype=dtype, device=DEV)


def _net_params(seed):
    """He-normal weights; the head's biases are a prior of small motions
    around the background's, as a trained head holds one."""
    rng = np.random.default_rng(int(seed) + 77)
    parts = []
    for out, fan in ((16, 18), (32, 144), (32, 288), (256, 1168), (296, 256)):
        wt = rng.standard_normal((out, fan)) * np.sqrt(2.0 / min(fan, 1158))
        if fan == 1168:
            wt[:, 1158:] = 0
        b = np.zeros(out)
        if out == 296:
            wt[289:] = 0
            wt *= 0.3
            c = np.arange(289)
            b[:289] = -0.15 * ((c % 17 - 7) ** 2 + (c // 17 - 8) ** 2)
        parts += [wt.ravel(), b]
    return np.concatenate(parts).astype(np.float32)


def _net(seed):
    net = mvnet.MvNet(acc(), seed=1)
    net.set_params(_net_params(seed))
    return net


def _net_inputs(case, seed):
    """Frame pairs of a clip, neighbour MVs around the pan, labels."""
    w, h, n = case["w"], case["h"], case["n"]
    y = clip(w, h, n + 1, seed)
    nmb = (y.shape[2] // 16) * (y.shape[1] // 16)
    rng = np.random.default_rng(int(seed) + 5)
    mv = np.round(rng.normal((5, -2) * 3, 6.0, (n * nmb, 6)))
    nmv = torch.from_numpy(np.clip(mv, -160, 160).astype(np.int16)).to(DEV)
    lab = torch.from_numpy(mvnet.class_of_mv(np.round(rng.normal((5, -2), 8.0, (n * nmb, 2))))).to(DEV)
    return y, nmv, lab


def _synthetic_picks(n, nmb, seed):
    """Picks as the search leaves them: mostly 16x16, MVs around the pan."""
    rng = np.random.default_rng(int(seed) + 9)
    p = np.zeros((n, nmb, 6), np.int32)
    p[..., 0] = rng.choice([0, 1, 2], (n, nmb), p=[0.7, 0.15, 0.15])
    p[..., 1:5] = np.round(rng.normal((5, -2, 5, -2), 4.0, (n, nmb, 4)))
    same = p[..., 0] == 0
    p[..., 3:5] = np.where(same[..., None], p[..., 1:3], p[..., 3:5])
    return torch.from_numpy(p).to(DEV)


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return state["run"](state)


# ---- the closed loop ------------------------------------------------------------------

def _prepare_closed(case, seed):
    a = acc()
    y, u, v = clip(case["w"], case["h"], case["n"], seed, chroma=True)
    n, ch, cw = y.shape
    nmb = (cw // 16) * (ch // 16)
    out = {"picks": _zeros((n, nmb, 6), torch.int32), "costs": _zeros((n, nmb, 2), torch.int64),
           "coeffs": _zeros((n, nmb, 256), torch.int16), "ccoeffs": _zeros((n, nmb, 128), torch.int16),
           "rec_y": torch.empty_like(y), "rec_u": torch.empty_like(u), "rec_v": torch.empty_like(v)}
    planes = _zeros((A.closed_plane_bytes(n, cw, ch),), torch.uint8)
    net = props = fb = half = la = None
    if case["learned"]:
        net = _net(seed)
        props, fb = _zeros((n, nmb, 16), torch.int32), _zeros((n, nmb), torch.int32)
        half, la = _zeros((n, ch // 2, cw // 2), torch.uint8), _zeros((4, n, nmb), torch.int32)
        out |= {"props": props, "fallback": fb}
    p = lambda t: 0 if t is None else t.data_ptr()  # noqa: E731
    qp = case["qp"]
    job = A.ClosedDev(p(y), p(u), p(v), p(out["rec_y"]), p(out["rec_u"]), p(out["rec_v"]), p(planes), n, cw, ch,
                      _lam(qp), A.split_gate_for_qp(qp), qp, DZ, None if net is None else net.h.value, 4096,
                      0 if la is None else p(la[2:]), p(out["picks"]), p(out["costs"]), p(out["coeffs"]),
                      p(out["ccoeffs"]), p(props), p(fb))
    return {"run": _run_closed, "acc": a, "job": job, "params": A.default_me_params(), "out": out, "net": net,
            "half": half, "la": la, "y": y, "keep": (u, v, planes)}


def _run_closed(s):
    a, y = s["acc"], s["y"]
    if s["net"] is not None:
        n, ch, cw = y.shape
        la, half = s["la"], s["half"]
        st = a._stream()
        a._check(a.L.h264a_downsample2x(a.ctx, y.data_ptr(), cw, ch, n, cw * ch, half.data_ptr(), st))
        a._check(a.L.h264a_lookahead_costs(a.ctx, y.data_ptr(), half.data_ptr(), cw, ch, n, 2, la[0].data_ptr(),
                                           la[1].data_ptr(), la[2:].data_ptr(), st))
    a.closed_frames(s["job"], s["params"])
    return s["out"]


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _prepare_closed_host(case, seed):
    y, u, v = (_pinned(t) for t in clip(case["w"], case["h"], case["n"], seed, chroma=True))
    n, ch, cw = y.shape
    nmb = (cw // 16) * (ch // 16)
    out = {k: torch.zeros(shape, dtype=dt, pin_memory=True).numpy() for k, shape, dt in (
        ("picks", (n, nmb, 6), torch.int32), ("costs", (n, nmb, 2), torch.int64),
        ("coeffs", (n, nmb, 256), torch.int16), ("ccoeffs", (n, nmb, 128), torch.int16),
        ("rec_y", y.shape, torch.uint8), ("rec_u", u.shape, torch.uint8), ("rec_v", v.shape, torch.uint8))}
    return {"run": _run_closed_host, "acc": acc(), "yuv": (y, u, v), "qp": case["qp"],
            "params": A.default_me_params(), "out": out}


def _run_closed_host(s):
    qp = s["qp"]
    return s["acc"].pixel_path_closed(*s["yuv"], s["params"], _lam(qp), A.split_gate_for_qp(qp), qp, DZ, out=s["out"])


def _prepare_step(case, seed):
    y, u, v = clip(case["w"], case["h"], 2, seed, chroma=True)
    _, ch, cw = y.shape
    nmb = (cw // 16) * (ch // 16)
    qp = case["qp"]
    out = {"picks": _zeros((nmb, 6), torch.int32), "costs": _zeros((nmb, 2), torch.int64),
           "coeffs": _zeros((nmb, 256), torch.int16), "ccoeffs": _zeros((nmb, 128), torch.int16),
           "rec_y": torch.empty_like(y[0]), "rec_u": torch.empty_like(u[0]), "rec_v": torch.empty_like(v[0])}
    planes = _zeros((1, 4, ch + 2 * PAD, cw + 2 * PAD), torch.uint8)
    me = A.MeFrame(A.Picture(y[1].data_ptr(), planes.data_ptr(), cw, ch, PAD), _lam(qp), A.split_gate_for_qp(qp),
                   out["picks"].data_ptr(), out["costs"].data_ptr())
    step = A.ClosedStep(me, u[1].data_ptr(), v[1].data_ptr(), u[0].data_ptr(), v[0].data_ptr(),
                        out["rec_y"].data_ptr(), out["rec_u"].data_ptr(), out["rec_v"].data_ptr(),
                        out["coeffs"].data_ptr(), out["ccoeffs"].data_ptr(), qp, DZ, 0, 0, 0)
    return {"run": _run_step, "acc": acc(), "yuv": (y, u, v), "planes": planes, "step": step, "out": out,
            "params": A.default_me_params()}


def _run_step(s):
    s["acc"].hpel_build(s["yuv"][0][:1], PAD, out=s["planes"])
    s["acc"].closed_step(s["step"], s["params"])
    return s["out"]


# ---- several streams ------------------------------------------------------------------------

def _sizes(case):
    return [tuple(int(v) for v in s.split("x")) for s in case["streams"].split(",")]


def _prepare_path(case, seed):
    qp, n = case["qp"], case["n"]
    streams, mf, tf, out = [], [], [], []
    for i, (w, h) in enumerate(_sizes(case)):
        y = clip(w, h, n, seed + 1000 * i)
        _, ch, cw = y.shape
        nmb = (cw // 16) * (ch // 16)
        planes = _zeros((n - 1, 4, ch + 2 * PAD, cw + 2 * PAD), torch.uint8)
        picks, costs = _zeros((n - 1, nmb, 6), torch.int32), _zeros((n - 1, nmb, 2), torch.int64)
        coeffs = _zeros((n - 1, nmb, 256), torch.int16)
        for f in range(1, n):
            pic = A.Picture(y[f].data_ptr(), planes[f - 1].data_ptr(), cw, ch, PAD)
            mf.append(A.MeFrame(pic, _lam(qp), A.split_gate_for_qp(qp), picks[f - 1].data_ptr(),
                                costs[f - 1].data_ptr()))
            tf.append(A.TqFrame(pic, picks[f - 1].data_ptr(), qp, DZ, coeffs[f - 1].data_ptr()))
        streams.append((y, planes))
        out.append({"picks": picks, "costs": costs, "coeffs": coeffs})
    return {"run": _run_path, "acc": acc(), "streams": streams, "me": mf, "tq": tf, "out": out,
            "params": A.default_me_params()}


def _run_path(s):
    a = s["acc"]
    for y, planes in s["streams"]:
        a.hpel_build(y[:-1], PAD, out=planes)
    a.me_frames(s["me"], s["params"])
    a.mc_tq_frames(s["tq"])
    return s["out"]


def _prepare_batch(case, seed):
    qp, g, nref = case["qp"], case["g"], case["nref"]
    n = 2 * g + 1
    nslots = -(-max(n, g + nref + 1) // g) * g
    streams, out, keep = [], [], []
    for i, (w, h) in enumerate(_sizes(case)):
        cw, ch = _coded(w), _coded(h)
        nmb = (cw // 16) * (ch // 16)
        src = _zeros((nslots, ch, cw), torch.uint8)
        src[:n] = clip(w, h, n, seed + 1000 * i)
        planes = _zeros((nslots, 4 * (cw + 2 * PAD) * (ch + 2 * PAD)), torch.uint8)
        picks, costs = _zeros((nslots, nmb, 8), torch.int32), _zeros((nslots, nmb, 2), torch.int64)
        coeffs = _zeros((nslots, nmb, 256), torch.int16)
        streams.append(A.BatchStream(cw, ch, PAD, src.data_ptr(), planes.data_ptr(), picks.data_ptr(),
                                     costs.data_ptr(), _lam(qp), A.split_gate_for_qp(qp), coeffs.data_ptr(), qp, DZ))
        out.append({"picks": picks[1:n], "costs": costs[1:n], "coeffs": coeffs[1:n]})
        keep.append((src, planes, picks, costs, coeffs))
    b = acc().batch_create(streams, A.BatchConfig(g, nslots, nref, 1, 0), A.default_me_params())
    return {"run": _run_batch, "batch": b, "g": g, "out": out, "keep": keep}


def _run_batch(s):
    for k in range(2):
        s["batch"].step(k, s["g"])
    return s["out"]


# ---- the lookahead, the reconstruction side, the grids, the planes ------------------------------

def _prepare_lookahead(case, seed):
    y = clip(case["w"], case["h"], case["n"], seed)
    return {"run": _run_lookahead, "acc": acc(), "y": y, "mode": case["mode"]}


def _run_lookahead(s):
    half = s["acc"].downsample2x(s["y"])
    intra, inter, mvs = s["acc"].lookahead_costs(s["y"], half, s["mode"])
    return {"half": half, "intra": intra, "inter": inter, "mvs": mvs}


def _prepare_recon(case, seed):
    qp, n = case["qp"], case["n"]
    y, u, v = clip(case["w"], case["h"], n + 1, seed, chroma=True)
    _, ch, cw = y.shape
    nmb = (cw // 16) * (ch // 16)
    planes = acc().hpel_build(y[:n], PAD)
    picks = _synthetic_picks(n, nmb, seed)
    out = {"coeffs": _zeros((n, nmb, 256), torch.int16), "ccoeffs": _zeros((n, nmb, 128), torch.int16),
           "rec_y": torch.empty_like(y[1:]), "rec_u": torch.empty_like(u[1:]), "rec_v": torch.empty_like(v[1:])}
    rec, chroma, db = [], [], []
    for f in range(n):
        ry, ru, rv = out["rec_y"][f].data_ptr(), out["rec_u"][f].data_ptr(), out["rec_v"][f].data_ptr()
        pk, co = picks[f].data_ptr(), out["coeffs"][f].data_ptr()
        pic = A.Picture(y[f + 1].data_ptr(), planes[f].data_ptr(), cw, ch, PAD)
        rec.append(A.TqRecFrame(A.TqFrame(pic, pk, qp, DZ, co), ry))
        chroma.append(A.TqChromaFrame(u[f + 1].data_ptr(), v[f + 1].data_ptr(), u[f].data_ptr(), v[f].data_ptr(), cw,
                                      ch, pk, qp, out["ccoeffs"][f].data_ptr(), ru, rv))
        db.append(A.DeblockFrame(ry, ru, rv, cw, ch, pk, co, qp, 0, 0, 0))
    return {"run": _run_recon, "acc": acc(), "rec": rec, "chroma": chroma, "db": db, "out": out,
            "keep": (y, u, v, planes, picks)}


def _run_recon(s):
    a = s["acc"]
    a.mc_tq_rec_frames(s["rec"])
    a.mc_tq_chroma_frames(s["chroma"])
    a.deblock_frames(s["db"])
    return s["out"]


def _prepare_grid(case, seed):
    y = clip(case["w"], case["h"], 2, seed)
    _, ch, cw = y.shape
    planes = acc().hpel_build(y[:1], PAD)
    return {"run": _run_grid, "acc": acc(), "pic": A.Picture(y[1].data_ptr(), planes.data_ptr(), cw, ch, PAD),
            "r": case["r"], "lam": _lam(27), "keep": (y, planes)}


def _run_grid(s):
    sad, satd, best = s["acc"].fullpel_grid(s["pic"], s["r"], lam=s["lam"])
    return {"sad": sad, "satd": satd, "best": best}


def _prepare_hpel(case, seed):
    y = clip(case["w"], case["h"], case["n"], seed)
    n, ch, cw = y.shape
    return {"run": _run_hpel, "acc": acc(), "y": y,
            "out": torch.empty((n, 4, ch + 2 * PAD, cw + 2 * PAD), dtype=torch.uint8, device=DEV)}


def _run_hpel(s):
    return s["acc"].hpel_build(s["y"], PAD, out=s["out"])


# ---- the proposal network ------------------------------------------------------------------------

def _prepare_net(case, seed, fn):
    y, nmv, lab = _net_inputs(case, seed)
    pairs = torch.tensor([[y[f].data_ptr(), y[f - 1].data_ptr()] for f in range(1, case["n"] + 1)],
                         dtype=torch.int64, device=DEV)
    return {"run": fn, "net": _net(seed), "y": y, "nmv": nmv, "lab": lab, "pairs": pairs, "n": case["n"]}


def _prepare_forward(case, seed):
    return _prepare_net(case, seed, _run_forward)


def _prepare_grads(case, seed):
    return _prepare_net(case, seed, _run_grads)


def _run_forward(s):
    ch, cw = s["y"].shape[1:]
    return s["net"].forward(s["pairs"].data_ptr(), s["n"], cw, ch, s["nmv"].data_ptr())


def _run_grads(s):
    ch, cw = s["y"].shape[1:]
    g, loss = s["net"].grads(s["pairs"].data_ptr(), s["n"], cw, ch, s["nmv"].data_ptr(), s["lab"].data_ptr())
    return {"grads": g, "loss": loss}


def _logits64(p, y, nmv, n):
    """The network in 64 bits: flat parameters p, frames y, MV features."""
    o = [0]

    def take(*shape):
        k = int(np.prod(shape))
        o[0] += k
        return p[o[0] - k:o[0]].reshape(shape)

    x = torch.stack([(y[:-1].double() - 128) / 64, (y[1:].double() - 128) / 64], 1)
    for co, ci in ((16, 2), (32, 16), (32, 32)):
        wt, b = take(co, 3, 3, ci), take(co)
        x = F.relu(F.conv2d(x, wt.permute(0, 3, 1, 2), b, stride=2, padding=1))
    mh, mw = y.shape[1] // 16, y.shape[2] // 16
    f = F.unfold(x, 6, padding=2, stride=2).reshape(n, 32, 36, mh * mw).permute(0, 3, 2, 1).reshape(n * mh * mw, 1152)
    mv = nmv.double().clamp(-128, 128) / 64
    f = torch.cat([f, mv, torch.zeros((len(mv), 10), dtype=torch.float64, device=DEV)], 1)
    w4, b4, w5, b5 = take(256, 1168), take(256), take(296, 256), take(296)
    return F.relu(f @ w4.T + b4) @ w5.T + b5


def exact(case, seed):
    if case["kind"] not in ("forward", "grads"):
        return None  # whole numbers: held to equality
    y, nmv, lab = _net_inputs(case, seed)
    p = torch.from_numpy(_net_params(seed)).to(DEV).double()
    if case["kind"] == "forward":
        with torch.no_grad():
            return _logits64(p, y, nmv, case["n"])
    p.requires_grad_(True)
    loss = F.cross_entropy(_logits64(p, y, nmv, case["n"])[:, :289], lab.long())
    loss.backward()
    return {"grads": p.grad, "loss": loss.detach().reshape(1)}


# ---- the work of a pass ------------------------------------------------------------------------------

#: integer operations of one MB's motion search: about 1,300 4x4 Hadamard evaluations of 112 operations
#: (the count the search itself reports on these clips)
ME_OPS = 1300 * 112
#: bytes an MB's search and T/Q write: picks 24, costs 16, luma levels 512
ME_OUT = 24 + 16 + 512
#: multiply-adds x 2 of one MB of the network: three convolutions, two dense layers
NET_FLOPS = 2 * (64 * 16 * 18 + 16 * 32 * 144 + 4 * 32 * 288 + 256 * 1168 + 296 * 256)


def work(case):
    kind = case["kind"]
    if kind in ("path", "batch"):
        sizes = _sizes(case)
        frames = case["n"] - 1 if kind == "path" else 2 * case["g"]
        mbs = frames * sum((_coded(w) // 16) * (_coded(h) // 16) for w, h in sizes)
        planes = frames * sum(4 * (_coded(w) + 2 * PAD) * (_coded(h) + 2 * PAD) for w, h in sizes)
        refs = 1 if kind == "path" else case["nref"]
        return {"bytes": mbs * (256 + ME_OUT) + planes, "flops": mbs * ME_OPS * refs}
    cw, ch = _coded(case["w"]), _coded(case["h"])
    px, mb = cw * ch, (cw // 16) * (ch // 16)
    plane = 4 * (cw + 2 * PAD) * (ch + 2 * PAD)
    n = case.get("n", 1)
    if kind in ("closed", "closed_host"):
        f = NET_FLOPS if case.get("learned") else 0
        return {"bytes": n * (px * 3 + mb * (ME_OUT + 256)), "flops": (n - 1) * mb * (ME_OPS + f)}
    if kind == "step":
        return {"bytes": px * 4.5 + plane + mb * (ME_OUT + 256), "flops": mb * ME_OPS}
    if kind == "lookahead":
        # about 17 SATD evaluations of four (half resolution) or sixteen blocks per MB
        return {"bytes": n * (px * 1.25 + mb * 16), "flops": (n - 1) * mb * 17 * (4 if case["mode"] == 2 else 16) * 112}
    if kind == "recon":
        return {"bytes": n * (px * 4.5 + mb * (24 + 512 + 256)), "flops": n * px * 1.5 * 40}
    if kind == "forward":
        return {"bytes": n * (2 * px + mb * (12 + 296 * 4)) + 4 * NPARAMS, "flops": n * mb * NET_FLOPS}
    if kind == "grads":
        return {"bytes": n * (2 * px + mb * 14) + 8 * NPARAMS, "flops": 3 * n * mb * NET_FLOPS}
    if kind == "grid":
        cand = (2 * case["r"] + 1) ** 2
        return {"bytes": 2 * px + mb * cand * 8, "flops": mb * cand * (16 * 112 + 64)}
    return {"bytes": n * (px + plane), "flops": n * plane * 12}
