"""GPU: a proposal call whose fall-back batch reports an error (an image of more
than 2^17 peaks), then the same handle's next calls."""
import math

import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


def test_fallback_error_then_next_call(cuda):
    from opencuda_gb300 import _lib
    from opencuda_gb300.houghline import HoughLine, Image
    from opencuda_gb300.proposal import HoughNet, proposal_batch
    det, K = math.pi / 720, 16
    imgs = [cases.synth(3, 8, i) for i in range(2)]
    imgs.append(np.where(np.random.default_rng(3).random((1024, 1024)) < 0.05, 255, 0)
                .astype(np.uint8))
    dev = [Image.from_host(im) for im in imgs]
    thr = [int(0.15 * max(im.shape)) for im in imgs]
    hl, plain, net = HoughLine(detheta=det), HoughLine(detheta=det), HoughNet(seed=4)
    rc, want = plain.houghLineBatch(dev, K, thr)
    assert rc == 0
    for _ in range(2):
        # every image falls back; the last one's threshold separates nothing
        assert proposal_batch(hl, net, dev, K, thr[:2] + [1], p_cut=1e-6, max_props=0)[0] == \
            _lib.CUDA_ERROR
        rc, got, st = proposal_batch(hl, net, dev, K, thr, p_cut=1e-6, max_props=0)
        assert rc == 0 and st["fallback"] == 3 and got == want
