"""GPU: a batch with more bins above the threshold than the candidate list holds,
noted by one warp an image and at the end by one warp alone, so that the list can
be full exactly where a step of the warp ends: the bins after it are missing, and
the peak pass has to know."""
import math

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_candidates_past_a_full_list(cuda):
    from opencuda_gb300.houghline import HoughLine, Image
    det, side, K = math.pi / 32, 430, 8192
    hl = HoughLine(detheta=det, thresang=0.0, thresdis=0)
    hl.set_vote_shape(0, 64)       # a producer and one voting warp
    c, s = hl.trig_table()

    def scene(seed, noise):
        rng = np.random.default_rng(seed)
        return np.where(rng.random((side, side)) < noise, 255, 0).astype(np.uint8)

    def want(img):
        return O.houghline(img, c, s, det, 1.0, 0, 0.0, 0, K)[0]

    # the dense image is voted longest: its bins are the last to be noted
    dense = scene(0, 0.2)
    dense_want, dense_dev = want(dense), Image.from_host(dense)
    bins = np.count_nonzero(O.vote_image(dense, c, s)[0])
    g = hl.geometry(side, side)
    n = 6
    room = (65536 + n * g.numrho * g.theta_pad // 128) * 5 // 4
    for trial in range(40):
        rest = [scene(100 + 7 * trial + i, 0.005 + 0.0005 * ((trial + i) % 5)) for i in range(n - 1)]
        noted = sum(np.count_nonzero(O.vote_image(im, c, s)[0]) for im in rest)
        assert noted < room < noted + bins, (noted, room, bins)
        rc, res = hl.houghLineBatch([Image.from_host(im) for im in rest] + [dense_dev], K, [0] * n)
        assert rc == 0
        assert [l.astuple() for l in res[-1]] == dense_want, trial
        if trial % 8 == 0:
            for im, got in zip(rest, res):
                assert [l.astuple() for l in got] == want(im)
