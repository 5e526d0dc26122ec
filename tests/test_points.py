"""The coordinate-list vote against the oracle, bit for bit: list lengths
around its parts, negative and far coordinates, more rows than one window,
thetas off a whole slice, rho step 2, and rho past the magic constant."""
import math

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _lines(xy, T, derho, thr, k, cuda):
    import torch
    from opencuda_gb300.houghline import HoughLine
    hl = HoughLine(detheta=math.pi / T, derho=derho, threshold=thr)
    rc, lines = hl.houghLineCor(torch.from_numpy(xy).to(cuda), k)
    assert rc == 0
    c, s = hl.trig_table()
    ax, ay = np.abs(xy.astype(np.float64)).max(0)
    d = int(math.floor((math.sqrt(ax * ax + ay * ay) + 1.0) / derho + 0.5))
    acc, dropped = O.vote_points(xy, c, s, -d, 2 * d + 1, derho)
    assert dropped == 0
    w, h = (int(v) for v in xy.max(0) - xy.min(0))
    g = O.geom(len(c), -d, 2 * d + 1, O.ref_numrho(w, h, derho), hl.getDeTheta(),
               hl.getThresDis(), hl.getThresAng())
    want, _, _ = O.rank_merge(acc, g, O.peaks(acc, thr), k)
    return [l.astuple() for l in lines], want


@pytest.mark.parametrize("n,T,derho,lo,hi", [
    (1, 180, 1.0, 5, 6),
    (7, 180, 1.0, -40, 40),
    (1023, 33, 1.0, 0, 300),
    (1025, 31, 1.0, -500, 700),
    (5000, 180, 2.0, -900, 900),
    (30011, 180, 1.0, 0, 1100),
    (20000, 97, 1.0, 0, 5000),        # several windows a slice
    (4096, 64, 1.0, -30000, -20000),  # a box far from the origin
])
def test_points_match_oracle(cuda, n, T, derho, lo, hi):
    rng = np.random.default_rng(n + T)
    xy = rng.integers(lo, hi, size=(n, 2)).astype(np.int32)
    m = n // 3   # a line among them
    xy[:m, 1] = lo + (xy[:m, 0] - lo) // 2
    got, want = _lines(xy, T, derho, 3 if n < 2000 else 12, 24, cuda)
    assert got == want


def test_points_repeat_and_grow(cuda):
    """The same handle over lists of other sizes: nothing is left over."""
    import torch
    from opencuda_gb300.houghline import HoughLine
    rng = np.random.default_rng(2)
    hl = HoughLine(threshold=5)
    lists = [rng.integers(0, s, size=(m, 2)).astype(np.int32)
             for s, m in ((300, 900), (900, 6000), (200, 50))]
    alone = []
    for xy in lists:
        alone.append(HoughLine(threshold=5).houghLineCor(torch.from_numpy(xy).to(cuda), 16)[1])
    for _ in range(2):
        for xy, want in zip(lists, alone):
            assert hl.houghLineCor(torch.from_numpy(xy).to(cuda), 16)[1] == want


def test_points_beyond_the_magic_constant(cuda):
    """|rho| past 2^22 (R >= 2^22): the exact conversion."""
    rng = np.random.default_rng(3)
    xy = rng.integers(-1500000, 1700000, size=(300, 2)).astype(np.int32)
    xy[:40] = xy[0] + np.arange(40)[:, None] * np.array([0, 1], np.int32)
    got, want = _lines(xy, 4, 1.0, 8, 8, cuda)
    assert got == want and len(want) > 0
