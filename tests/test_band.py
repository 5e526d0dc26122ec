"""Which tiles a vote item takes (hl_band.h, the code that the vote kernel runs) on
the CPU over many sizes: the segments of a sliding item share out the tiles of a row
without a gap or an overlap, an item of one rho window takes every tile that can
reach it.  And batches of sizes whose band edges fall within a float's last bits of
a tile's centre, bit for bit against the oracle."""
import ctypes as C
import math
import subprocess

import numpy as np
import pytest

from oracle import oracle as O

CAP = 1536        # rows of a window
# width, height, T, and a (theta slice, tile column, tile row) on a band's edge
EDGES = [(1970, 1413, 360, 5, 7, 29), (1220, 1517, 720, 16, 1, 18),
         (1290, 1141, 720, 14, 6, 33), (1730, 1601, 720, 8, 6, 27), (1980, 1873, 720, 4, 6, 20)]


@pytest.fixture(scope="module")
def band(tmp_path_factory):
    from opencuda_gb300 import build
    d = tmp_path_factory.mktemp("band")
    (d / "band.c").write_text(
        '#include "hl_band.h"\n'
        "void rows(int nseg, int adv, float half, const float *yk, int n, float cm, float icm,\n"
        "          float x0, int txn, int *out)\n"
        "{\n"
        "    for (int r = 0; r < n; r++)\n"
        "        for (int j = 0; j < nseg; j++, out += 2)\n"
        "            hl_band_tiles(j, nseg, adv, half, yk[r], cm, icm, x0, txn, out, out + 1);\n"
        "}\n"
        "void windows(int n, const float *lo, const float *hi, float tang, float c, float s,\n"
        "             float x1, const float *y, int rows, int txn, int *out)\n"
        "{\n"
        "    for (int j = 0; j < n; j++)\n"
        "        for (int r = 0; r < rows; r++)\n"
        "            for (int side = 0; side < 2; side++, out += 2)\n"
        "                hl_band_window(side, lo[j], hi[j], tang, c, s, x1, y[r], txn, out,\n"
        "                               out + 1);\n"
        "}\n")
    subprocess.run(["gcc", "-O2", "-shared", "-fPIC", "-I", str(build.CSRC), str(d / "band.c"),
                    "-o", str(d / "band.so"), "-lm"], check=True)
    lib = C.CDLL(str(d / "band.so"))
    F, I, P = C.c_float, C.c_int, C.c_void_p
    lib.rows.argtypes = [I, I, F, P, I, F, F, F, I, P]
    lib.windows.argtypes = [I, P, P, F, F, F, F, P, I, I, P]
    return lib


def _slices(w, h, T):
    """(middle cos, middle sin, segments, rows to slide, half) of every sliding
    slice of a w x h image, as the plan and the kernel compute them."""
    f = np.float32
    lx, ly = 0.5 * w + 128, 0.5 * h + 32
    det = math.pi / T
    dist = math.hypot(lx, ly)
    err = math.ceil(66 + dist * 16 * det + dist * 1e-5) + 4
    adv = (CAP - 2 * err - 4) // 4 * 4
    if 2 * adv < CAP:
        return
    for sl in range((T + 31) // 32):
        th = f(min(sl * 32 + 16, T - 1) * det)
        c, s = f(np.cos(th)), f(np.sin(th))
        half = math.ceil(lx * abs(float(c)) + ly * abs(float(s))) + 2.0
        nseg = math.ceil(2 * half / adv)
        if nseg > 1:
            yield c, s, nseg, adv, half


def test_every_tile_in_one_segment(band):
    f = np.float32
    rng = np.random.default_rng(7)
    sizes = [e[:3] for e in EDGES]
    sizes += [(int(rng.integers(800, 2600)), int(rng.integers(800, 2600)),
               int(rng.choice([180, 360, 720, 1440]))) for _ in range(4000)]
    seen = 0
    for w, h, T in sizes:
        tx, ty = (w + 127) // 128, (h + 31) // 32
        ctx, cty = f(0.5) * f(w - 1), f(0.5) * f(h - 1)
        for c, s, nseg, adv, half in _slices(w, h, T):
            cm = f(math.copysign(max(abs(float(c)), 1e-9), float(c)))
            yk = ((np.arange(ty) * 32 + 16).astype(f) - cty) * s
            out = np.empty((ty, nseg, 2), np.int32)
            band.rows(nseg, adv, half, yk.ctypes.data, ty, float(cm), float(f(1) / (cm * f(128))),
                      float((ctx - f(64)) * f(1 / 128)), tx, out.ctypes.data)
            o = out if cm > 0 else out[:, ::-1]
            assert np.all(o[:, 0, 0] == 0) and np.all(o[:, -1, 1] == tx), (w, h, T)
            assert np.array_equal(o[:, :-1, 1], o[:, 1:, 0]) and np.all(o[..., 0] <= o[..., 1]), \
                (w, h, T)
            seen += nseg * ty
    assert seen > 100000


def _windows(w, h, sl, c, s, det, derho, cap):
    """(number of windows, rows, first offset, lo, hi, tang) of one block, as
    hl_api.cpp's block_band and band_windows compute them."""
    T = len(c)
    k0, k1 = sl * 32, min(sl * 32 + 32, T) - 1
    km = min(k0 + 16, T - 1)
    x, y = 0.5 * w, 0.5 * h
    ac, as_ = (np.abs(v[k0:k1 + 1].astype(float)) for v in (c, s))
    half, tile = float(np.max(x * ac + y * as_)), float(np.max(64 * ac + 16 * as_))
    slack = 4 + math.hypot(w, h) / derho / (1 << 19)
    first = -math.ceil(half / derho + slack)
    n = (1 - 2 * first + cap - 1) // cap
    rows = (1 - 2 * first + n - 1) // n
    d = max(k1 - km, km - k0) * det
    far = (x + 128) * abs(float(c[km])) + (y + 128) * abs(float(s[km]))
    out = tile + (1 - math.cos(min(d, math.pi))) * far + 2 + slack * derho
    j = np.arange(n)
    return (n, rows, first, (first * derho - out + j * rows * derho).astype(np.float32),
            ((first + rows) * derho + out + j * rows * derho).astype(np.float32),
            math.sin(d) if d < math.pi / 2 else 1.0)


def test_windows_take_every_tile_that_reaches_them(band):
    f = np.float32
    rng = np.random.default_rng(11)
    cases = [(1, 1, 180, 1.0, 1536), (1, 2000, 90, 0.25, 512), (3000, 1, 45, 0.1, 1536),
             (128, 32, 7, 0.5, 128), (4096, 4096, 1, 1.0, 256), (1000, 900, 3, 0.05, 1536),
             (65535, 40, 180, 1.0, 1536), (40, 65535, 180, 1.0, 1536)]
    for _ in range(150):
        w, h = (int(math.exp(rng.uniform(math.log(20), math.log(3000)))) for _ in range(2))
        cases.append((w, h, int(rng.choice([20, 45, 90, 180, 360, 720])),
                      float(rng.choice([0.05, 0.1, 0.25, 0.5, 1.0, 3.0])),
                      int(rng.choice([128, 303, 682, 1536]))))
    taken = needed = 0
    for w, h, T, derho, cap in cases:
        det = math.pi / T
        th = (np.arange(T) * det).astype(f)
        c, s = np.cos(th), np.sin(th)
        tx, ty = (w + 127) // 128, (h + 31) // 32
        ctx, cty = f(0.5) * f(w - 1), f(0.5) * f(h - 1)
        yy = (np.arange(ty) * 32 + 16).astype(f) - cty
        for sl in range((T + 31) // 32):
            n, rows, first, lo, hi, tang = _windows(w, h, sl, c, s, det, derho, cap)
            pick = np.unique(rng.integers(0, n, 6))
            lo, hi = np.ascontiguousarray(lo[pick]), np.ascontiguousarray(hi[pick])
            ks = np.arange(sl * 32, min(sl * 32 + 32, T))
            km = min(sl * 32 + 16, T - 1)
            out = np.empty((len(pick), ty, 2, 2), np.int32)
            band.windows(len(pick), lo.ctypes.data, hi.ctypes.data, tang, float(c[km]),
                         float(s[km]), float(f(64) - ctx), yy.ctypes.data, ty, tx, out.ctypes.data)
            assert out.min() >= 0 and out.max() <= tx
            # the sides do not overlap: no point is voted twice
            assert np.all(out[:, :, 0, 1] <= out[:, :, 1, 0]) or np.all(
                (out[..., 1] <= out[..., 0]).any(-1) | (out[:, :, 0, 1] <= out[:, :, 1, 0]))
            t = np.arange(tx)
            got = ((t >= out[..., :1]) & (t < out[..., 1:])).sum(2)
            assert got.max() <= 1
            # the rows that a tile's corners reach at every theta, two to spare
            xs = np.stack([t * 128, np.minimum(t * 128 + 127, w - 1)])[:, None, :]
            ys = np.stack([np.arange(ty) * 32, np.minimum(np.arange(ty) * 32 + 31, h - 1)])
            mn = np.full((len(ks), ty, tx), 1e300)
            mx = -mn
            cc, ss = c[ks].astype(float)[:, None, None], s[ks].astype(float)[:, None, None]
            for a in range(2):
                for b in range(2):
                    v = (xs[a] * cc + ys[b][:, None] * ss) / derho
                    mn, mx = np.minimum(mn, v), np.maximum(mx, v)
            base = np.floor((float(ctx) * cc + float(cty) * ss) / derho)
            lo_r, hi_r = np.floor(mn - base) - 2, np.ceil(mx - base) + 2
            assert lo_r.min() >= first and hi_r.max() <= first + n * rows, (w, h, T, derho)
            for q, j in enumerate(pick):
                need = ((hi_r >= first + j * rows) & (lo_r < first + (j + 1) * rows)).any(0)
                assert np.all(got[q][need]), (w, h, T, derho, cap, sl, j)
                needed += need.sum()
                taken += got[q].sum()
    assert taken < 1.6 * needed, (taken, needed)


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,T,sl,tx,ty", EDGES)
def test_batches_with_a_tile_on_a_band_edge(cuda, w, h, T, sl, tx, ty):
    """Sixteen images (their slices slide): strokes at the slice's middle angle in
    the tile and its neighbours, counted by one segment each."""
    from opencuda_gb300.houghline import HoughLine, Image
    det = math.pi / T
    hl = HoughLine(detheta=det, thresang=1e-3, thresdis=2)
    c, s = hl.trig_table()
    th = (sl * 32 + 16) * det
    x0, y0 = max(0, (tx - 1) * 128), ty * 32
    imgs = []
    for seed in (1, 2):
        img = np.where(np.random.default_rng(seed).random((h, w)) < 0.01, 255, 0).astype(np.uint8)
        yy, xx = np.mgrid[y0:min(y0 + 32, h), x0:min(x0 + 384, w)]
        rho = xx * math.cos(th) + yy * math.sin(th) + seed
        img[y0:y0 + 32, x0:x0 + 384][np.abs(rho - 9 * np.round(rho / 9)) < 0.5] = 255
        imgs.append(img)
    dev = [Image.from_host(im) for im in imgs]
    thr = 60
    hl.setThreshold(thr)
    plain = []
    for im, d in zip(imgs, dev):
        rc, got = hl.houghLine(d, None, 1024)
        want = O.houghline(im, c, s, det, 1.0, thr, hl.getThresAng(), hl.getThresDis(), 1024)[0]
        assert rc == 0 and len(want) > 8 and [l.astuple() for l in got] == want
        plain.append(want)
    rc, res = hl.houghLineBatch(dev * 8, 1024, [thr] * 16)
    assert rc == 0
    for i, got in enumerate(res):
        assert [l.astuple() for l in got] == plain[i % 2], i
