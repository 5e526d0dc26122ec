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


def _dirty(torch, nbytes, n):
    """n freed blocks of about nbytes, full of ones."""
    keep = [torch.full((nbytes // 4,), 1, dtype=torch.int32, device="cuda") for _ in range(n)]
    torch.cuda.synchronize()
    del keep
    torch.cuda.empty_cache()


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


def test_accumulators_after_a_failed_allocation(cuda):
    """A batch that is too large, then the batch before it again: its accumulators
    are as large as they were, and not the ones that were left zero."""
    import torch
    from opencuda_gb300.houghline import HoughLine, Image
    dev = [Image.from_host(_image(500 + 30 * i, 640 - 20 * i, i)) for i in range(8)]
    hl = HoughLine(detheta=math.pi / 180, threshold=40)
    want = hl.houghLineBatch(dev, 32)
    assert want[0] == 0 and hl.houghLineBatch(dev, 32) == want
    _too_large(hl)
    assert hl.setDeTheta(math.pi / 180) == 0 and hl.setDeRho(1.0) == 0
    acc = sum(4 * hl.geometry(d.width, d.height).numrho * 192 for d in dev)
    _dirty(torch, acc + acc // 4, 16)
    assert hl.houghLineBatch(dev, 32) == want


@pytest.mark.parametrize("n", [1, 2])
def test_no_room_for_slabs(cuda, n):
    """With memory for everything but the slabs of a split vote (over 100 MB),
    the items add to the accumulator instead: four launches, the same lines."""
    import torch
    from opencuda_gb300.houghline import HoughLine, Image
    g = torch.Generator(device="cuda").manual_seed(5)
    buf = (torch.rand((8192, 8192), generator=g, device="cuda") < 0.002).to(torch.uint8) * 255
    buf[2000, :] = 255
    buf[:, 5000] = 255
    dev = [Image(buf, (0, 0, 8192, 8192 - 100 * i)) for i in range(n)]

    def call():
        hl = HoughLine(detheta=math.pi / 32, threshold=1000)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        got = hl.houghLine(dev[0], None, 16) if n == 1 else hl.houghLineBatch(dev, 16)
        torch.cuda.synchronize()
        used = free - torch.cuda.mem_get_info()[0]
        return got, used, hl.last_launch_count()

    call()
    want, used, launches = call()
    assert want[0] == 0 and launches == (5 if n == 1 else 4)
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - used + (60 << 20), dtype=torch.uint8,
                      device="cuda")
    try:
        got, less, launches = call()
    finally:
        del hog
        torch.cuda.empty_cache()
    assert got == want and launches == 4 and less < used
    # with the memory back a new handle has its slabs again
    assert call()[0] == want
