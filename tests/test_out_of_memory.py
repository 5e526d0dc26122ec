"""GPU: calls that the device has no memory for fail, and the next ones do not
rely on what their buffers held."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _image(w, h, seed=0):
    img = np.where(np.random.default_rng(seed).random((h, w)) < 0.02, 255, 0).astype(np.uint8)
    img[h // 3, :] = 255
    img[:, w // 2] = 255
    return img


def _too_large(hl):
    """A batch whose accumulators need 400 GB."""
    from opencuda_gb300 import _lib
    from opencuda_gb300.houghline import Image
    small = Image.from_host(_image(64, 64))
    assert hl.setDeTheta(math.pi / 1440) == 0 and hl.setDeRho(7.0e-4) == 0
    g = hl.geometry(64, 64)
    n = 400 * 10 ** 9 // (4 * g.numrho * g.theta_pad)
    assert hl.houghLineBatch([small] * n, 4) == (_lib.OUT_OF_MEM, [])


def test_a_failed_allocation_is_reported_once(cuda):
    from opencuda_gb300.houghline import HoughLine, Image
    dev = Image.from_host(_image(500, 640))
    hl = HoughLine(detheta=math.pi / 180, threshold=100)
    want = hl.houghLine(dev, None, 16)
    assert want[0] == 0
    _too_large(hl)
    assert hl.setDeTheta(math.pi / 180) == 0 and hl.setDeRho(1.0) == 0
    assert hl.houghLine(dev, None, 16) == want
