"""GPU: blocks voted in windows of rows -- several windows a block, groups of tile
rows, parts of a window's points, slices of few angles, the exact conversion, rho 0
inside a window -- whole accumulators and lines, single images and batches, bit for
bit against the oracle."""
import math

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _scene(w, h, seed, noise):
    rng = np.random.default_rng(seed)
    img = np.where(rng.random((h, w)) < noise, 255, 0).astype(np.uint8)
    img[h // 2, :] = 255
    img[:, w // 3] = 255
    n = min(w, h)
    img[np.arange(n), np.arange(n)] = 255
    img[0, 0] = img[0, -1] = img[-1, 0] = img[-1, -1] = 255
    return img


@pytest.mark.parametrize("w,h,T,derho,rows", [
    (512, 512, 180, 0.1, 0),
    (512, 512, 180, 0.05, 0),
    (129, 65, 60, 0.05, 0),
    (1, 700, 45, 0.02, 0),
    (700, 1, 45, 0.02, 0),
    (300, 200, 3, 0.02, 0),          # a slice of three angles
    (400, 300, 33, 0.05, 0),         # a last slice of one
    (700, 500, 180, 0.25, 168),      # the smallest windows
    (260, 4200, 90, 0.1, 0),         # more tile rows than a group holds, parts
    (4200, 260, 90, 0.1, 0),
    (1500, 1200, 90, 0.1, 0),        # parts of windows, merged
    (333, 257, 45, 2.0e-4, 0),       # rho bins past 2^22
    (200, 190, 360, 1.0, 0),         # images of one window, step 1
])
def test_windows(cuda, w, h, T, derho, rows):
    from opencuda_gb300.houghline import HoughLine, Image
    det = math.pi / T
    hl = HoughLine(detheta=det, derho=derho)
    if rows:
        hl.set_vote_shape(rows, 0)
    c, s = hl.trig_table()
    for seed, noise in ((1, 0.02), (2, 0.004)):
        img = _scene(w, h, seed, noise)
        dev = Image.from_host(img)
        want, wmin, _ = O.vote_image(img, c, s, derho)
        for _ in range(2):
            acc, rho_min = hl.accumulator(dev)
            assert rho_min == wmin and np.array_equal(acc.cpu().numpy(), want)
        for thr in (int(want.max() * 0.5), max(1, int(want.max() * 0.05))):
            lines_want = O.houghline(img, c, s, det, derho, thr, hl.getThresAng(),
                                     hl.getThresDis(), 16)[0]
            hl.setThreshold(thr)
            for _ in range(2):
                rc, lines = hl.houghLine(dev, None, 16)
                assert rc == 0 and [l.astuple() for l in lines] == lines_want


@pytest.mark.parametrize("T,derho", [(180, 0.1), (60, 0.03), (360, 0.25), (180, 1.0)])
def test_batches_in_windows(cuda, T, derho):
    from opencuda_gb300.houghline import HoughLine, Image
    det = math.pi / T
    hl = HoughLine(detheta=det, derho=derho)
    c, s = hl.trig_table()
    imgs = [_scene(w, h, w, 0.01) for w, h in ((611, 507), (130, 900), (1000, 33), (512, 512),
                                               (1, 1), (257, 2100))]
    dev = [Image.from_host(im) for im in imgs]
    for frac in (0.5, 0.1):
        thr = [max(1, int(frac * min(im.shape))) for im in imgs]
        rc, res = hl.houghLineBatch(dev, 16, thr)
        assert rc == 0
        for im, t, got in zip(imgs, thr, res):
            want = O.houghline(im, c, s, det, derho, t, hl.getThresAng(), hl.getThresDis(), 16)[0]
            assert [l.astuple() for l in got] == want, im.shape
