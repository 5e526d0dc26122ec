"""GPU: calls queued without a wait on a stream that the default stream does not
order itself with."""
import ctypes as C
import math

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _image(w, h, seed):
    img = np.where(np.random.default_rng(seed).random((h, w)) < 0.02, 255, 0).astype(np.uint8)
    img[h // 3, :] = 255
    img[:, w // 2] = 255
    return img


def test_geometries_alternate_on_one_stream(cuda):
    """Two ROI sizes in turn, nothing waited for in between: every call's vote
    reads its own plan."""
    import torch
    from opencuda_gb300 import _lib
    from opencuda_gb300.houghline import HoughLine, Image
    L = _lib.load()
    det, K, n = math.pi / 360, 16, 12
    hl = HoughLine(detheta=det, threshold=250)
    c, s = hl.trig_table()
    sizes = [(1900, 1100), (1300, 1700)]
    imgs = [_image(w, h, i) for i, (w, h) in enumerate(sizes)]
    dev = [Image.from_host(im) for im in imgs]
    want = [O.houghline(im, c, s, det, 1.0, 250, hl.getThresAng(), hl.getThresDis(), K)[0]
            for im in imgs]
    # every buffer at its largest, so that no later call allocates
    for d in dev:
        assert hl.houghLine(d, None, K)[0] == 0
    lines = torch.zeros((n, K, 3), dtype=torch.int32, device=cuda)
    counts = torch.zeros(n, dtype=torch.int32, device=cuda)
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    descs = [d.desc() for d in dev]
    for i in range(n):
        _lib.check(L.hl_plain_async(hl.handle, C.byref(descs[i % 2]), K,
                                    C.c_void_p(lines[i].data_ptr()),
                                    C.c_void_p(counts[i:].data_ptr()),
                                    C.c_void_p(st.cuda_stream)), "hl_plain_async")
    st.synchronize()
    got = lines.cpu().numpy()
    for i in range(n):
        m = int(counts[i])
        ang = got[i, :m, 0].copy().view(np.float32)
        assert [(float(a), int(d), int(v)) for a, d, v in
                zip(ang, got[i, :m, 1], got[i, :m, 2])] == want[i % 2], i


def test_first_calls_beside_a_busy_default_stream(cuda):
    """A new handle's first batch and first circles on a non-blocking stream while
    the default stream is busy: their fresh counters are cleared in order."""
    import torch
    from opencuda_gb300 import _lib
    from opencuda_gb300.houghcircle import HoughCircle
    from opencuda_gb300.houghline import HoughLine, Image
    L = _lib.load()
    det, K = math.pi / 180, 16
    imgs = [_image(700 + 60 * i, 500 + 90 * i, i) for i in range(4)]
    dev = [Image.from_host(im) for im in imgs]
    ref, hl = HoughLine(detheta=det, threshold=150), HoughLine(detheta=det, threshold=150)
    rc, want = ref.houghLineBatch(dev, K)
    assert rc == 0
    circ = [HoughCircle(), HoughCircle()]
    wantc = circ[0].houghcircle(dev[0], None, 8)
    # dirty memory for the buffers to come
    dirt = [torch.full((1 << 18,), 0x01010101, dtype=torch.int32, device=cuda) for _ in range(64)]
    torch.cuda.synchronize()
    del dirt
    torch.cuda.empty_cache()
    st = torch.cuda.Stream()
    a = torch.randn((8192, 8192), dtype=torch.bfloat16, device=cuda)
    for _ in range(40):
        b = a @ a
    rc, got = hl.houghLineBatch(dev, K, stream=st)
    assert rc == 0 and got == want
    gotc = circ[1].houghcircle(dev[0], None, 8, stream=st)
    assert gotc == wantc
    torch.cuda.synchronize()
    del b
