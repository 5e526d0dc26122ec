"""GPU: circle counts on bit planes where they can go wrong -- widths around words,
units and tiles of the bit rows, maxima on the tiles' edges, the fullest counts,
thresholds past the planes, radii on both sides of the limit -- against the
oracle, counts and circles, for one image and for batches."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _noise(w, h, density, seed):
    rng = np.random.default_rng(seed)
    return np.where(rng.random((h, w)) < density, 255, 0).astype(np.uint8)


@pytest.fixture(scope="module")
def mod(cuda):
    from opencuda_gb300.houghcircle import HoughCircle
    from opencuda_gb300.houghline import Image
    return HoughCircle, Image


@pytest.mark.parametrize("w,h,rmin,rmax,density", [
    (1, 1, 0, 3, 1.0),
    (31, 40, 0, 9, 0.2),
    (32, 33, 1, 6, 0.2),
    (129, 130, 3, 9, 0.1),
    (257, 65, 2, 8, 0.1),
    (1025, 70, 4, 7, 0.1),      # two tiles of 20 words
    (2100, 80, 5, 8, 0.1),      # three tiles
    (400, 300, 86, 92, 0.1),    # bit planes and votes in one call
    (380, 380, 87, 90, 1.0),    # every offset of the largest radii counts
    (64, 64, 90, 95, 0.3),      # votes only
])
def test_counts_and_circles(mod, w, h, rmin, rmax, density):
    HoughCircle, Image = mod
    img = _noise(w, h, density, w + h)
    dev = Image.from_host(img)
    want = O.circle_vote(img, rmin, rmax)
    hc = HoughCircle(rmin, rmax)
    assert np.array_equal(hc.accumulator(dev).cpu().numpy(), want)
    # thresholds from the lowest that the candidate list takes, so maxima lie on
    # every edge of the tiles; and two past all counts
    done = 0
    for thr in sorted({0, int(want.max() * 0.5), int(want.max() * 0.7), 511, 512, 5000}):
        circ, n = O.houghcircle(img, rmin, rmax, thr, 0.5, 1, 64)
        rc, got = HoughCircle(rmin, rmax, 0.5, 1, thr).houghcircle(dev, None, 64)
        if n > 4096:
            assert rc == -3
            continue
        assert rc == 0
        assert [c.astuple() for c in got] == list(circ), thr
        done += 1
    assert done >= 3


@pytest.mark.parametrize("rmin,rmax,thr", [(3, 9, 20), (87, 92, 60)])
def test_batches_of_uneven_sizes(mod, rmin, rmax, thr):
    HoughCircle, Image = mod
    imgs = [_noise(w, h, 0.08, w) for w, h in ((1100, 130), (1, 1), (40, 300), (256, 256), (700, 33))]
    rc, per = HoughCircle(rmin, rmax, 4.0, 3, thr).houghcircleBatch(
        [Image.from_host(im) for im in imgs], 12)
    assert rc == 0
    for im, got in zip(imgs, per):
        want, n = O.houghcircle(im, rmin, rmax, thr, 4.0, 3, 12)
        assert n <= 4096 and [c.astuple() for c in got] == list(want), im.shape


@pytest.mark.parametrize("rmin,rmax", [(0, 44), (45, 89)])
def test_offsets_of_every_radius(mod, rmin, rmax):
    HoughCircle, Image = mod
    img = _noise(203, 190, 0.3, rmax)
    got = HoughCircle(rmin, rmax).accumulator(Image.from_host(img)).cpu().numpy()
    assert np.array_equal(got, O.circle_vote(img, rmin, rmax))
