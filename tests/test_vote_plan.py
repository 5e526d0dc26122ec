"""GPU: the vote's regions, windows and stores where they can go wrong -- tile
edges, ROIs of one row or column, more tile rows than a list of runs holds,
slices of few angles, rho steps above and below a pixel (32-bit slabs, several
windows a tile, the exact conversion), the smallest windows, sliding windows --
bit for bit against the oracle, with whole accumulators and peak-only calls in
turn on one handle (each leaves the buffer as the other needs it)."""
import math

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hl_mod(cuda):
    from opencuda_gb300.houghline import HoughLine, Image
    return HoughLine, Image


def _scene(w, h, seed, noise=0.03):
    rng = np.random.default_rng(seed)
    img = np.where(rng.random((h, w)) < noise, 255, 0).astype(np.uint8)
    img[h // 2, :] = 255
    img[:, w // 3] = 255
    n = min(w, h)
    img[np.arange(n), np.arange(n)] = 255
    img[0, 0] = img[0, -1] = img[-1, 0] = img[-1, -1] = 255
    return img


def _want(hl, img, thr, k, det, derho):
    c, s = hl.trig_table()
    return O.houghline(img, c, s, det, derho, thr, hl.getThresAng(), hl.getThresDis(), k)[0]


@pytest.mark.parametrize("w,h,det,derho,rows", [
    (128, 32, math.pi / 180, 1.0, 0),
    (129, 33, math.pi / 180, 1.0, 0),
    (1300, 1, math.pi / 360, 1.0, 0),
    (1, 1300, math.pi / 360, 1.0, 0),
    (1000, 5000, math.pi / 180, 1.0, 0),      # 157 tile rows
    (2100, 1500, math.pi / 20, 1.0, 0),       # one slice of 20 angles
    (2048, 2048, math.pi / 90, 1.0, 0),       # a last slice of 26
    (2048, 1536, math.pi / 360, 2.0, 0),
    (4096, 3000, math.pi / 180, 8.0, 0),      # counts may pass 16 bits
    (300, 200, math.pi / 45, 0.03, 0),        # a tile's range exceeds a window
    (300, 200, math.pi / 4, 1.5e-4, 0),       # rho bins past 2^22
    (1500, 1100, math.pi / 360, 1.0, 8),      # the smallest windows
    (2048, 2048, math.pi / 5760, 1.0, 0),     # whole slices an item, sliding windows
])
def test_accumulators_and_peaks_in_turn(hl_mod, w, h, det, derho, rows):
    HoughLine, Image = hl_mod
    hl = HoughLine(detheta=det, derho=derho)
    if rows:
        hl.set_vote_shape(rows, 0)
    c, s = hl.trig_table()
    for seed in (1, 2):
        img = _scene(w, h, seed)
        dev = Image.from_host(img)
        acc, rho_min = hl.accumulator(dev)
        want, wmin, _ = O.vote_image(img, c, s, derho)
        assert rho_min == wmin and np.array_equal(acc.cpu().numpy(), want)
        # a threshold that separates, and one that floods the candidates
        for thr in (int(want.max() * 0.6), max(1, int(want.max() * 0.02))):
            if want.size > 1 << 25 and thr < want.max() * 0.5:
                continue
            hl.setThreshold(thr)
            for _ in range(2):
                rc, lines = hl.houghLine(dev, None, 16)
                assert rc == 0
                assert [l.astuple() for l in lines] == _want(hl, img, thr, 16, det, derho)


@pytest.mark.parametrize("det,derho", [(math.pi / 360, 1.0), (math.pi / 45, 0.5),
                                       (math.pi / 1440, 2.0), (math.pi / 40, 0.06)])
def test_batches_reuse_their_accumulators(hl_mod, det, derho):
    """Uneven batches, flooded candidate lists between separating thresholds (an
    image of more than 2^17 peaks fails the call, not the next one), a second
    batch of other sizes in the same buffers."""
    HoughLine, Image = hl_mod
    hl = HoughLine(detheta=det, derho=derho)
    c, s = hl.trig_table()
    sizes = [[(256, 256), (2048, 1800), (33, 700), (1900, 40), (1024, 1024), (1, 1)],
             [(1800, 2048), (64, 64), (700, 1024), (129, 31)]]
    for b in range(2):
        imgs = [_scene(w, h, 10 * b + i) for i, (w, h) in enumerate(sizes[b])]
        dev = [Image.from_host(im) for im in imgs]
        for frac in (0.5, 0.04, 0.5):
            thr = [max(1, int(frac * max(im.shape))) for im in imgs]
            rc, res = hl.houghLineBatch(dev, 16, thr)
            npk = [len(O.peaks(O.vote_image(im, c, s, derho)[0], t)) for im, t in zip(imgs, thr)]
            if max(npk) > 1 << 17:
                assert rc == -7
                continue
            assert rc == 0
            for im, t, got in zip(imgs, thr, res):
                assert [l.astuple() for l in got] == _want(hl, im, t, 16, det, derho), im.shape


def test_blocks_whole_and_split_in_one_batch(hl_mod):
    """More blocks than CTAs, each most of a CTA's share: some are voted whole,
    the rest in regions that fill the gaps."""
    HoughLine, Image = hl_mod
    det = math.pi / 300
    hl = HoughLine(detheta=det)
    imgs = [_scene(640, 480, 100 + i) for i in range(20)]
    dev = [Image.from_host(im) for im in imgs]
    for thr in (300, 25):
        rc, res = hl.houghLineBatch(dev, 16, [thr] * len(imgs))
        assert rc == 0
        for im, got in zip(imgs, res):
            assert [l.astuple() for l in got] == _want(hl, im, thr, 16, det, 1.0)


@pytest.mark.parametrize("derho", [0.5, 0.25, 0.1, 0.03])
def test_fine_rho_steps(hl_mod, derho):
    """Regions of one window and of several, for one image and for a batch."""
    HoughLine, Image = hl_mod
    det = math.pi / 60
    hl = HoughLine(detheta=det, derho=derho)
    imgs = [_scene(w, h, w) for w, h in ((611, 507), (130, 900), (1000, 33))]
    dev = [Image.from_host(im) for im in imgs]
    c, s = hl.trig_table()
    for im, d in zip(imgs, dev):
        acc, rho_min = hl.accumulator(d)
        want, wmin, _ = O.vote_image(im, c, s, derho)
        assert rho_min == wmin and np.array_equal(acc.cpu().numpy(), want)
    thr = [max(im.shape) // 2 for im in imgs]
    rc, res = hl.houghLineBatch(dev, 16, thr)
    assert rc == 0
    for im, t, got in zip(imgs, thr, res):
        assert [l.astuple() for l in got] == _want(hl, im, t, 16, det, derho), im.shape
