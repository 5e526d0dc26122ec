"""GPU: circle counts where few edge pixels are about: tiles, and cells of a warp,
that cannot pass the threshold are not counted -- whole circles alone in the image
at thresholds on both sides of their count, next to tile edges and image edges, and
sparse noise with rings -- against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _circle(img, cx, cy, r):
    """The pixels that a cell at (cx, cy) counts for radius r: where it votes."""
    h, w = img.shape
    one = np.zeros((2 * r + 3, 2 * r + 3), np.uint8)
    one[r + 1, r + 1] = 255
    dy, dx = np.nonzero(O.circle_vote(one, r, r)[0])
    y, x = cy + dy - r - 1, cx + dx - r - 1
    ok = (y >= 0) & (y < h) & (x >= 0) & (x < w)
    img[y[ok], x[ok]] = 255


@pytest.mark.parametrize("r", [1, 7, 31, 32, 45, 64, 89])
def test_one_circle_at_its_own_count(cuda, r):
    from opencuda_gb300.houghcircle import HoughCircle
    from opencuda_gb300.houghline import Image
    w, h = 1100, 300
    for cx, cy in ((r + 3, r + 3), (1023, 31), (1024, 160), (127, 96), (640, 299 - r), (5, 150)):
        img = np.zeros((h, w), np.uint8)
        _circle(img, cx, cy, r)
        dev = Image.from_host(img)
        top = int(O.circle_vote(img, r, r).max())
        for thr in (top // 2, top - 5, top - 1, top):
            if thr < 0:
                continue
            want, n = O.houghcircle(img, r, r, thr, 0.5, 1, 64)
            if n > 4096:
                continue
            rc, got = HoughCircle(r, r, 0.5, 1, thr).houghcircle(dev, None, 64)
            assert rc == 0 and [c.astuple() for c in got] == list(want), (cx, cy, thr)
        assert thr == top and not want


@pytest.mark.parametrize("density", [0.0002, 0.001, 0.004, 0.02])
@pytest.mark.parametrize("rmin,rmax", [(3, 12), (40, 47), (80, 91)])
def test_sparse_noise_with_rings(cuda, density, rmin, rmax):
    from opencuda_gb300.houghcircle import HoughCircle
    from opencuda_gb300.houghline import Image
    rng = np.random.default_rng(rmax)
    imgs = []
    for w, h in ((1200, 230), (200, 400)):
        img = np.where(rng.random((h, w)) < density, 255, 0).astype(np.uint8)
        for i in range(4):
            _circle(img, int(rng.integers(0, w)), int(rng.integers(0, h)), rmin + i)
        imgs.append(img)
    dev = [Image.from_host(im) for im in imgs]
    top = max(int(O.circle_vote(im, rmin, rmax).max()) for im in imgs)
    done = 0
    for thr in (top // 4, top // 2, 3 * top // 4, top - 1):
        want = [O.houghcircle(im, rmin, rmax, thr, 4.0, 3, 32) for im in imgs]
        if max(n for _, n in want) > 4096:
            continue
        done += 1
        for d, (circ, _) in zip(dev, want):
            rc, got = HoughCircle(rmin, rmax, 4.0, 3, thr).houghcircle(d, None, 32)
            assert rc == 0 and [c.astuple() for c in got] == list(circ), thr
        rc, per = HoughCircle(rmin, rmax, 4.0, 3, thr).houghcircleBatch(dev, 32)
        assert rc == 0
        assert [[c.astuple() for c in p] for p in per] == [list(c) for c, _ in want]
    assert done >= 2
