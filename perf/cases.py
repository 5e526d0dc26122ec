"""The workloads whose speed this framework is judged by.

Each case is one call a user's program makes: through the C ABI
(include/houghline_gb300.h, hl_proposal.h, hl_circle.h) where the program
keeps its results on the device or in arrays of its own, through the Python
classes where it wants objects.  Images are seeded synthetic edge maps
(straight segments and salt noise, or rings), made on the GPU and resident
there, as an edge detector in front of the transform leaves them; the handle,
with its workspace and angle table, is kept from call to call.

The kinds:
  plain     HoughLine::houghLine on one image, lines left on the device or
            returned to the host (sync)
  batch     many images of uneven size in one pipeline (CUDA-graph replay)
  tiles     the tiled caller: piecenum x piecenum cells of one image
  points    houghLine over a coordinate set
  draw      houghLineImg: the lines of one image drawn into another
  circles   HoughCircle::houghcircle on one image
  pieces    many ROIs of one image, circles (pieceCircle's batch)
  proposal  the learned proposal stage, exact windowed vote, fall-back
  forward   the proposal network alone, logits of B occupancy maps
  train     one training step of the network (forward, backward, Adam)
"""
from __future__ import annotations

import ctypes as C
import json
import math

import numpy as np
import torch

from opencuda_gb300 import _lib
from opencuda_gb300.houghcircle import HoughCircle
from opencuda_gb300.houghline import HoughLine, Image
from opencuda_gb300.proposal import HEAD_R, HEAD_T, NET_IN, WEIGHTS, HoughNet


# ---- the cases -----------------------------------------------------------------

def listed():
    return [
        # a camera-sized thumbnail, one call at a time: latency and launches count
        dict(name="plain_512", kind="plain", w=512, h=512, x1=0, y1=0, T=180, derho=1.0, thr=100,
             K=16, nseg=8, ppm=10000, sync=True),
        # a full-HD frame with a ragged ROI at an odd offset, half-degree steps
        dict(name="plain_1080p_roi", kind="plain", w=1913, h=1077, x1=5, y1=3, T=360, derho=1.0,
             thr=280, K=64, nseg=24, ppm=20000, sync=False),
        # the headline size: a scanned page / satellite tile at quarter-degree steps
        dict(name="plain_4096", kind="plain", w=4096, h=4096, x1=0, y1=0, T=720, derho=1.0,
             thr=300, K=256, nseg=64, ppm=20000, sync=False),
        # a data set of uneven images through one pipeline, as a service batches them
        dict(name="batch_256_uneven", kind="batch", n=256, lo=256, hi=2048, T=360, K=32),
        # the recogniser's grid of cells over one image: many small images at once
        dict(name="tiles_8x8_2048", kind="tiles", w=2048, h=2048, pieces=8, T=180, thr=60, K=16,
             nseg=64, ppm=10000),
        # a coordinate set (the guidingset argument) of a 1024 x 1024 scene
        dict(name="points_24k", kind="points", w=1024, h=1024, T=180, thr=150, K=16, nseg=16,
             ppm=20000),
        # the lines of an image drawn back over it (houghLineImg)
        dict(name="draw_2048", kind="draw", w=2048, h=2048, T=360, thr=300, K=32, nseg=32,
             ppm=10000),
        # circle detection at the class's default radii and thresholds
        dict(name="circles_1024", kind="circles", w=1024, h=1024, rmin=5, rmax=50, thr=100, K=32,
             rings=24, ppm=10000),
        # the same image cut into pieces, ten circles each
        dict(name="pieces_4x4_1024", kind="pieces", w=1024, h=1024, pieces=4, rmin=5, rmax=50,
             thr=100, K=10, rings=24, ppm=10000),
        # proposal-guided detection over a batch, at the calibrated selection
        dict(name="proposal_32x2048", kind="proposal", n=32, spec=4, T=360, K=32),
        # the proposal network on a batch of maps: what a detector in front of the vote runs
        dict(name="forward_64", kind="forward", B=64),
        # one step of training it, at the end of the cosine schedule
        dict(name="train_32", kind="train", B=32, lr=1e-5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above: sizes over their logarithm, odd ones
    among them, at most the largest listed case's work."""
    kind = rng.choice(["plain", "plain", "plain", "batch", "tiles", "points", "draw", "circles",
                       "pieces", "proposal", "forward", "train"])
    T = rng.choice([90, 180, 180, 360, 360, 720])
    if kind == "plain":
        w, h = _log(rng, 200, 4096), _log(rng, 200, 4096)
        x1, y1 = rng.choice([(0, 0), (rng.randint(0, 31), rng.randint(0, 9))])
        derho = rng.choice([1.0, 1.0, 1.0, 2.0])
        return dict(kind=kind, w=w, h=h, x1=x1, y1=y1, T=T, derho=derho,
                    thr=int(0.15 * max(w, h) * derho), K=rng.choice([16, 32, 64, 256]),
                    nseg=rng.randint(4, 64), ppm=rng.randint(5000, 30000),
                    sync=rng.random() < 0.5)
    if kind == "batch":
        lo = _log(rng, 128, 512)
        return dict(kind=kind, n=_log(rng, 2, 200), lo=lo, hi=_log(rng, 2 * lo, 2048),
                    T=rng.choice([180, 360]), K=rng.choice([16, 32]))
    if kind == "tiles":
        w, h = _log(rng, 500, 2600), _log(rng, 500, 2600)
        p = rng.randint(2, 10)
        return dict(kind=kind, w=w, h=h, pieces=p, T=rng.choice([90, 180, 360]),
                    thr=int(0.25 * max(w, h) / p), K=16, nseg=rng.randint(8, 64),
                    ppm=rng.randint(5000, 20000))
    if kind == "points":
        w, h = _log(rng, 200, 2048), _log(rng, 200, 2048)
        return dict(kind=kind, w=w, h=h, T=rng.choice([90, 180, 360]),
                    thr=int(0.15 * max(w, h)), K=rng.choice([16, 64]), nseg=rng.randint(4, 32),
                    ppm=rng.randint(5000, 30000))
    if kind == "draw":
        w, h = _log(rng, 300, 3000), _log(rng, 300, 3000)
        return dict(kind=kind, w=w, h=h, T=rng.choice([180, 360]), thr=int(0.15 * max(w, h)),
                    K=rng.choice([8, 16, 32, 64]), nseg=rng.randint(4, 48),
                    ppm=rng.randint(5000, 20000))
    if kind in ("circles", "pieces"):
        w, h = _log(rng, 200, 1300), _log(rng, 200, 1300)
        rmin = rng.randint(0, 20)
        rmax = rmin + rng.randint(5, 50)
        c = dict(kind=kind, w=w, h=h, rmin=rmin, rmax=rmax, thr=max(40, 2 * rmax), K=32,
                 rings=rng.randint(4, 32), ppm=rng.randint(2000, 15000))
        if kind == "pieces":
            c.update(pieces=rng.randint(2, 4), K=10)
        return c
    if kind == "proposal":
        return dict(kind=kind, n=_log(rng, 2, 32), spec=rng.choice([4, 5]), T=360,
                    K=rng.choice([16, 32]))
    if kind == "forward":
        return dict(kind=kind, B=_log(rng, 1, 128))
    return dict(kind=kind, B=_log(rng, 2, 32), lr=1e-5)


# ---- inputs --------------------------------------------------------------------

def _scenes(params):
    """Edge maps of the given scene parameters, each in a pitched device buffer."""
    n = len(params)
    ps = (_lib.hl_scene_params * n)(*params)
    descs = (_lib.hl_image_desc * n)()
    imgs = []
    for i, p in enumerate(ps):
        pitch = (p.width + 511) // 512 * 512
        buf = torch.zeros((p.height, pitch), dtype=torch.uint8, device="cuda")
        descs[i] = _lib.hl_image_desc(buf.data_ptr(), pitch, p.width, p.height, 0, 0,
                                      p.width, p.height)
        im = Image(buf[:, :p.width])
        im._buf = buf
        imgs.append(im)
    _lib.check(_lib.load().hl_synth_scenes_device(ps, n, descs, None), "hl_synth_scenes_device")
    return imgs


def _scene(c, seed, extra_w=0, extra_h=0):
    """One edge map of w x h: nseg segments of 10-100% of the diagonal, ppm salt."""
    w, h = c["w"] + extra_w, c["h"] + extra_h
    d = int(math.hypot(w, h))
    return _scenes([_lib.hl_scene_params(w, h, c["nseg"], d // 10, d, c["ppm"], 0,
                                         seed * 7919 + 17)])[0]


def _rings(c, seed):
    """An edge map of c["rings"] one-pixel rings with radii in the voted range
    (at least 8) and ppm salt."""
    w, h = c["w"], c["h"]
    rs = np.random.RandomState(seed % (1 << 31))
    pitch = (w + 511) // 512 * 512
    buf = torch.zeros((h, pitch), dtype=torch.uint8, device="cuda")
    im = buf[:, :w]
    g = torch.Generator(device="cuda").manual_seed(seed)
    im[torch.rand((h, w), generator=g, device="cuda") < c["ppm"] * 1e-6] = 255
    yy = torch.arange(h, device="cuda", dtype=torch.float32)[:, None]
    xx = torch.arange(w, device="cuda", dtype=torch.float32)[None, :]
    for _ in range(c["rings"]):
        r = rs.randint(max(8, c["rmin"]), max(9, c["rmin"] + 1, c["rmax"] + 1))
        a, b = rs.randint(0, w), rs.randint(0, h)
        im[(torch.sqrt((xx - a) ** 2 + (yy - b) ** 2) - r).abs() < 0.5] = 255
    out = Image(im)
    out._buf = buf
    return out


def _spec(kind, seed, n, lo=0, hi=0):
    """Scene parameters of a workload spec; with lo / hi, uneven sides in [lo, hi]."""
    if not lo:
        ps = (_lib.hl_scene_params * n)()
        _lib.check(_lib.load().hl_synth_spec(kind, seed, n, ps), "hl_synth_spec")
        return list(ps)
    rs = np.random.RandomState(seed % (1 << 31))
    out = []
    for i in range(n):
        w, h = int(rs.randint(lo, hi + 1)), int(rs.randint(lo, hi + 1))
        d = int(math.hypot(w, h))
        out.append(_lib.hl_scene_params(w, h, int(rs.randint(4, 33)), d // 10, d,
                                        int(rs.randint(5000, 30001)), 0, seed * 1000003 + i))
    return out


def _maps(B, seed):
    """Occupancy maps and coarse geometries of B images of 2048 x 2048 scenes'
    statistics: salt at 1-4% per pixel averaged over 8 x 8 cells, and lines."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    dens = 0.01 + 0.03 * torch.rand((B, 1, 1), generator=g, device="cuda")
    salt = torch.rand((B, 64, NET_IN, NET_IN), generator=g, device="cuda") < dens[:, None]
    occ = salt.sum(1, dtype=torch.float32)
    yy = torch.arange(NET_IN, device="cuda", dtype=torch.float32)[:, None] + 0.5
    xx = torch.arange(NET_IN, device="cuda", dtype=torch.float32)[None, :] + 0.5
    th = torch.rand((B, 16), generator=g, device="cuda") * math.pi
    px = torch.rand((B, 16, 2), generator=g, device="cuda") * NET_IN
    c, s = th.cos(), th.sin()
    rho = px[..., 0] * c + px[..., 1] * s
    for k in range(16):
        d = xx * c[:, k, None, None] + yy * s[:, k, None, None] - rho[:, k, None, None]
        occ += 8.0 * (d.abs() < 0.5)
    occ = (occ.clamp(max=64.0) / 64.0).to(torch.bfloat16)
    R = 2 * int(math.floor(math.hypot(2048, 2048) + 0.5)) + 1
    geo = (_lib.hl_coarse_geom * B)(*[_lib.hl_coarse_geom(32.0, -float(R // 2), HEAD_R / R, 64,
                                                          64, 0)] * B)
    # where the drawn lines lie in the coarse cells (the training target)
    wrap = th >= math.pi
    t = (torch.where(wrap, th - math.pi, th) / (math.pi / HEAD_T)).long().clamp(0, HEAD_T - 1)
    r = torch.floor((8.0 * rho + R // 2) * (HEAD_R / R)).long().clamp(0, HEAD_R - 1)
    tgt = torch.zeros((B, HEAD_T, HEAD_R), dtype=torch.float32, device="cuda")
    tgt[torch.arange(B, device="cuda")[:, None], t, r] = 1.0
    return occ.view(torch.int16).contiguous(), geo, tgt


def _net():
    net = HoughNet()
    net.load(WEIGHTS)
    return net


def _lines_out(n, K):
    """Device arrays of n x K line records (as 32-bit words) and n counts."""
    return (torch.zeros((n, K, 3), dtype=torch.int32, device="cuda"),
            torch.zeros(n, dtype=torch.int32, device="cuda"))


class _State:
    pass


def prepare(case, seed):
    c, s = case, _State()
    s.case, s.kind, s.L = c, c["kind"], _lib.load()
    if s.kind in ("plain", "draw", "points", "tiles"):
        s.hl = HoughLine(detheta=math.pi / c["T"], derho=c.get("derho", 1.0),
                         threshold=c["thr"])
    if s.kind == "plain":
        im = _scene(c, seed, c["x1"] + 11 * bool(c["x1"]), c["y1"] + 3 * bool(c["y1"]))
        s.img = Image(im.data, (c["x1"], c["y1"], c["x1"] + c["w"], c["y1"] + c["h"]))
        s.desc = s.img.desc()
        s.lines, s.count = _lines_out(1, c["K"])
    elif s.kind == "batch":
        s.hl = HoughLine(detheta=math.pi / c["T"])
        s.hl.set_batch_graph(True)
        s.imgs = _scenes(_spec(0, seed, c["n"], c["lo"], c["hi"]))
        s.descs = (_lib.hl_image_desc * c["n"])(*[im.desc() for im in s.imgs])
        s.thr = (C.c_int * c["n"])(*[int(0.15 * max(im.width, im.height)) for im in s.imgs])
        s.lines, s.count = _lines_out(c["n"], c["K"])
    elif s.kind == "tiles":
        s.img = _scene(c, seed)
        s.desc = s.img.desc()
        n = c["pieces"] ** 2
        s.out, s.cnt = (_lib.hl_line * (n * c["K"]))(), (C.c_int * n)()
    elif s.kind == "points":
        # raster order, as the reference's ImgConvert lists an image's points
        nz = torch.nonzero(_scene(c, seed).data == 255)
        s.xy = nz.flip(1).to(torch.int32).contiguous()
        s.out, s.lm = (_lib.hl_line * c["K"])(), C.c_int()
    elif s.kind == "draw":
        s.img = _scene(c, seed)
        s.dst = s.img.data.new_zeros(tuple(s.img._buf.shape))
        s.din = s.img.desc()
        s.dout = _lib.hl_image_desc(s.dst.data_ptr(), s.dst.stride(0), c["w"], c["h"], 0, 0,
                                    c["w"], c["h"])
        s.out, s.lm = (_lib.hl_line * c["K"])(), C.c_int()
    elif s.kind in ("circles", "pieces"):
        s.hc = HoughCircle(c["rmin"], c["rmax"], 50.0, 20, c["thr"])
        s.img = _rings(c, seed)
        if s.kind == "pieces":
            p = c["pieces"]
            cx, cy = c["w"] // p, c["h"] // p
            s.pieces = [Image(s.img.data, (x * cx, y * cy, x * cx + cx - 1, y * cy + cy - 1))
                        for y in range(p) for x in range(p)]
    elif s.kind == "proposal":
        s.hl = HoughLine(detheta=math.pi / c["T"])
        s.hl.set_batch_graph(True)
        s.net = _net()
        s.imgs = _scenes(_spec(c["spec"], seed, c["n"]))
        s.descs = (_lib.hl_image_desc * c["n"])(*[im.desc() for im in s.imgs])
        s.thr = (C.c_int * c["n"])(*[int(0.15 * max(im.width, im.height)) for im in s.imgs])
        sel = json.loads(WEIGHTS.with_name("proposal_selection.json").read_text())
        sel.update(sel["per_spec"][str(c["spec"])])
        s.opts = _lib.hl_proposal_opts(sel["p_cut"], sel["max_props"], sel["dilate_theta"],
                                       sel["dilate_rho"], 0, sel["top_m"], sel["nms"],
                                       sel["p_conf"])
        s.lines, s.count = _lines_out(c["n"], c["K"])
    else:
        s.net = _net()
        s.occ, s.geo, s.tgt = _maps(c["B"], seed)
    return s


# ---- one pass ------------------------------------------------------------------

def _host_lines(out, n):
    """The first n line records on the host as (angle, distance, votes) arrays,
    with zeros up to the records' room."""
    a = np.zeros(len(out), dtype=[("a", "<f4"), ("d", "<i4"), ("v", "<i4")])
    a[:n] = np.frombuffer(out, dtype=a.dtype, count=n)
    return {"angle": a["a"].copy(), "distance": a["d"].copy(), "votes": a["v"].copy()}


def _circle_rows(per, room):
    """Circles of every image as rows (image, k) -> a, b, radius, votes, with
    zeros up to the room, and their counts."""
    a = np.zeros((len(per), room, 4), np.int32)
    for i, p in enumerate(per):
        for k, q in enumerate(p):
            a[i, k] = q.astuple()
    return {"circles": a, "count": np.array([len(p) for p in per], np.int32)}


def run(state):
    s, c = state, state.case
    kind = s.kind
    if kind == "plain" and c["sync"]:
        rc, lines = s.hl.houghLine(s.img, None, c["K"])
        _lib.check(rc, "houghLine")
        got = np.zeros((c["K"], 3))
        for i, l in enumerate(lines):
            got[i] = l.astuple()
        return {"angle": got[:, 0].astype(np.float32), "distance": got[:, 1].astype(np.int32),
                "votes": got[:, 2].astype(np.int32)}
    if kind == "plain":
        rc = s.L.hl_plain_async(s.hl.handle, C.byref(s.desc), c["K"],
                                C.c_void_p(s.lines.data_ptr()), C.c_void_p(s.count.data_ptr()),
                                None)
        _lib.check(rc, "hl_plain_async")
        return {"lines": s.lines, "count": s.count}
    if kind == "batch":
        rc = s.L.hl_batch_async(s.hl.handle, s.descs, c["n"], s.thr, c["K"],
                                C.c_void_p(s.lines.data_ptr()), C.c_void_p(s.count.data_ptr()),
                                None)
        _lib.check(rc, "hl_batch_async")
        return {"lines": s.lines, "count": s.count}
    if kind == "tiles":
        rc = s.L.hl_tiles(s.hl.handle, C.byref(s.desc), c["pieces"], c["K"], s.out, s.cnt, None)
        _lib.check(rc, "hl_tiles")
        got = _host_lines(s.out, len(s.out))
        got["count"] = np.array(s.cnt, np.int32)
        return got
    if kind == "points":
        s.lm.value = c["K"]
        rc = s.L.hl_plain_points(s.hl.handle, C.c_void_p(s.xy.data_ptr()), int(s.xy.shape[0]),
                                 C.byref(s.lm), s.out, None)
        _lib.check(rc, "hl_plain_points")
        return _host_lines(s.out, s.lm.value)
    if kind == "draw":
        s.lm.value = c["K"]
        rc = s.L.hl_plain_draw(s.hl.handle, C.byref(s.din), C.byref(s.dout), C.byref(s.lm),
                               s.out, None)
        _lib.check(rc, "hl_plain_draw")
        got = _host_lines(s.out, s.lm.value)
        got["image"] = s.dst
        return got
    if kind == "circles":
        rc, cir = s.hc.houghcircle(s.img, None, c["K"])
        _lib.check(rc, "houghcircle")
        return _circle_rows([cir], c["K"])
    if kind == "pieces":
        rc, per = s.hc.houghcircleBatch(s.pieces, c["K"])
        _lib.check(rc, "houghcircleBatch")
        return _circle_rows(per, c["K"])
    if kind == "proposal":
        rc = s.L.hl_proposal_batch(s.hl.handle, s.net.handle, s.descs, c["n"], s.thr, c["K"],
                                   C.byref(s.opts), C.c_void_p(s.lines.data_ptr()),
                                   C.c_void_p(s.count.data_ptr()), None, None)
        _lib.check(rc, "hl_proposal_batch")
        return {"lines": s.lines, "count": s.count}
    if kind == "forward":
        return s.net.forward(s.occ, s.geo)
    loss = s.net.train_step(s.occ, s.geo, s.tgt, c["lr"], 40.0)
    return {"loss": np.array([loss], np.float32), "grads": s.net.get_grads(),
            "params": s.net.get_params()}


# ---- what a pass cannot do without ----------------------------------------------

def _points_of(w, h, nseg, ppm):
    return w * h * ppm * 1e-6 + 0.35 * nseg * math.hypot(w, h)


def work(case):
    """Bytes: every input read once, every output written once.  Operations: a
    vote of a line is two products, a sum and an increment; of a circle an
    increment; of the network, its multiplies and adds."""
    c, k = case, case["kind"]
    if k in ("plain", "tiles", "draw", "points"):
        n = _points_of(c["w"], c["h"], c["nseg"], c["ppm"])
        byts = 8 * n if k == "points" else c["w"] * c["h"]
        byts += 12 * c["K"] * (c["pieces"] ** 2 if k == "tiles" else 1)
        if k == "draw":   # a byte for every pixel of a line
            byts += c["K"] * max(c["w"], c["h"])
        return {"bytes": byts, "flops": 4 * n * c["T"]}
    if k == "batch":
        side = 0.5 * (c["lo"] + c["hi"])
        n = _points_of(side, side, 18, 17500)
        return {"bytes": c["n"] * (side * side + 12 * c["K"]), "flops": 4 * c["n"] * n * c["T"]}
    if k in ("circles", "pieces"):
        n = c["w"] * c["h"] * c["ppm"] * 1e-6 + c["rings"] * 2.8 * (c["rmin"] + c["rmax"])
        votes = n * sum(8 * r / math.sqrt(2) for r in range(c["rmin"], c["rmax"] + 1))
        return {"bytes": c["w"] * c["h"] + 16 * c["K"], "flops": votes}
    layers = [(128 * 128, 9, 32), (64 * 64, 288, 32), (64 * 64, 288, 32), (64 * 64, 288, 32),
              (64 * 64, 288, 32), (64 * 64, 288, 1)]
    fwd = sum(2 * p * kk * co for p, kk, co in layers) + 2 * 64 * 64 * HEAD_T
    params = sum(kk * co + co for _, kk, co in layers) + 2
    if k == "proposal":
        side = 2048
        n = _points_of(side, side, 28, 25000)
        # the image, the network, and at least the votes of its windows' own bins
        return {"bytes": c["n"] * (side * side + 12 * c["K"]),
                "flops": c["n"] * (fwd + 4 * n * 9)}
    io = c["B"] * 2 * NET_IN * NET_IN
    if k == "forward":
        return {"bytes": io + 4 * c["B"] * HEAD_T * HEAD_R + 2 * params, "flops": c["B"] * fwd}
    # training: the forward pass, and twice it for the two gradients; weights,
    # gradients and both Adam moments
    return {"bytes": io + 4 * c["B"] * HEAD_T * HEAD_R + 28 * params, "flops": 3 * c["B"] * fwd}


# ---- the network in 64 bits -----------------------------------------------------

_LAYERS = [(1, 32, 2, 1), (32, 32, 2, 1), (32, 32, 1, 1), (32, 32, 1, 1), (32, 32, 1, 1),
           (32, 1, 1, 0)]


def _net64(flat, occ, requires_grad):
    """Logits in double: 3 x 3 convolutions (weights [cout][ky][kx][cin], the
    flat FP32 parameters), ReLU, then the sums of the evidence over the coarse
    (angle, rho) bins."""
    import torch.nn.functional as F
    p = torch.from_numpy(flat).cuda().double()
    if requires_grad:
        p.requires_grad_()
    x = occ.view(torch.bfloat16).double()[:, None]
    o = 0
    for cin, cout, stride, relu in _LAYERS:
        w = p[o:o + cout * 9 * cin].reshape(cout, 3, 3, cin).permute(0, 3, 1, 2)
        # the network multiplies BF16 weights
        w = w + (w.detach().to(torch.float32).to(torch.bfloat16).double() - w.detach())
        o += cout * 9 * cin
        x = F.conv2d(x, w, p[o:o + cout], stride=stride, padding=1)
        o += cout
        if relu:
            x = F.relu(x)
    e = x[:, 0].reshape(x.shape[0], -1)
    R = 2 * int(math.floor(math.hypot(2048, 2048) + 0.5)) + 1
    th = ((np.arange(HEAD_T) + 0.5) * math.pi / HEAD_T)
    cc, ss = np.cos(th).astype(np.float32), np.sin(th).astype(np.float32)
    pos = ((np.arange(64, dtype=np.float32) + np.float32(0.5)) * np.float32(32.0))
    rho = (pos[None, None, :] * cc[:, None, None]) + (pos[None, :, None] * ss[:, None, None])
    bins = np.floor((rho - np.float32(-(R // 2))) * np.float32(HEAD_R / R)).astype(np.int64)
    bins = torch.from_numpy(np.clip(bins, 0, HEAD_R - 1).reshape(HEAD_T, -1)).cuda()
    h = torch.stack([torch.zeros((e.shape[0], HEAD_R), dtype=e.dtype, device=e.device)
                     .index_add(1, bins[t], e) for t in range(HEAD_T)], 1)
    return p, p[o] * h + p[o + 1]


def exact(case, seed):
    """The network's logits, loss, gradients and updated weights in double;
    the line and circle cases give whole numbers."""
    if case["kind"] not in ("forward", "train"):
        return None
    import torch.nn.functional as F
    occ, _, tgt = _maps(case["B"], seed)
    flat = np.load(WEIGHTS).astype(np.float32)
    train = case["kind"] == "train"
    p, z = _net64(flat, occ, train)
    if not train:
        return z
    y = tgt.double()
    loss = -(40.0 * y * F.logsigmoid(z) + (1 - y) * F.logsigmoid(-z)).mean()
    g, = torch.autograd.grad(loss, p)
    gc = g.clamp(-1.0, 1.0)
    # the first Adam step from zero moments: both bias corrections cancel
    new = p.detach() - case["lr"] * gc / (gc.abs() + 1e-8)
    return {"loss": loss.detach().reshape(1), "grads": g, "params": new}
