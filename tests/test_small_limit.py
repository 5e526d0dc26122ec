"""GPU: images whose rho range is the longest that one cluster launch takes, and the
ones beside it, against the oracle."""
import math

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [2, 180, 256])
@pytest.mark.parametrize("w,h,R", [(906, 3, 1813), (907, 3, 1815), (641, 642, 1815),
                                   (908, 3, 1817)])
def test_longest_rho_ranges(cuda, w, h, R, T):
    from opencuda_gb300.houghline import HoughLine, Image
    det = math.pi / T
    img = np.where(np.random.default_rng(w).random((h, w)) < 0.05, 255, 0).astype(np.uint8)
    img[h // 2, :] = 255
    hl = HoughLine(detheta=det, threshold=200)
    assert hl.geometry(w, h).numrho == R
    c, s = hl.trig_table()
    want = O.houghline(img, c, s, det, 1.0, 200, hl.getThresAng(), hl.getThresDis(), 16)[0]
    rc, lines = hl.houghLine(Image.from_host(img), None, 16)
    assert rc == 0 and [l.astuple() for l in lines] == want
