"""GPU: a captured batch follows what changes between its calls -- the merge
thresholds, the angle table's place, buffers that an uncaptured call moved."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture()
def pair(cuda):
    """Two handles alike, the first with captured batches."""
    from opencuda_gb300.houghline import HoughLine
    hls = [HoughLine(detheta=math.pi / 180, threshold=120) for _ in range(2)]
    hls[0].set_batch_graph(True)
    return hls


def _images(sizes):
    from opencuda_gb300.houghline import Image
    out = []
    for i, (w, h) in enumerate(sizes):
        img = np.where(np.random.default_rng(i).random((h, w)) < 0.02, 255, 0).astype(np.uint8)
        for x in range(20, w - 4, 37):
            img[:, x] = img[:, x + 3] = 255
        out.append(Image.from_host(img))
    return out


def _same(pair, dev, K=64):
    (rc, got), (rc2, want) = [hl.houghLineBatch(dev, K) for hl in pair]
    assert rc == rc2 == 0 and got == want
    return want


def test_merge_thresholds(pair):
    dev = _images([(512, 300), (400, 400), (301, 640)])
    seen = []
    for dis, ang in ((50, 0.08), (2, 0.08), (2, 0.001), (50, 0.08)):
        for hl in pair:
            assert hl.setThresDis(dis) == 0 and hl.setThresAng(ang) == 0
        seen.append([len(l) for l in _same(pair, dev)])
    assert seen[0] != seen[1] and seen[1] != seen[2]


def test_theta_step_changed_and_restored(pair):
    dev = _images([(512, 300), (400, 400), (301, 640)])
    _same(pair, dev)
    for hl in pair:
        for d in (math.pi / 720, math.pi / 1440, math.pi / 180):
            assert hl.setDeTheta(d) == 0
    _same(pair, dev)


def test_uncaptured_call_in_between(pair):
    dev, tiny = _images([(512, 300), (400, 400)]), _images([(48, 16)] * 300)
    _same(pair, dev)
    pair[0].set_batch_graph(False)
    _same(pair, tiny)
    pair[0].set_batch_graph(True)
    _same(pair, dev)
    _same(pair, tiny)
