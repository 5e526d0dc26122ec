"""GPU: the pipelined compaction of tile groups (batches, callers without a
handle, images past the cooperative kernel) at its edges -- one tile, one tile
and a pixel, tiles missing from the last group, unaligned ROIs, no and all
points, more groups than the all-predecessor prefix takes -- exactly the points
of numpy, tile by tile in raster order."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,roi,noise", [
    (1, 1, None, 1.0),
    (128, 32, None, 0.1),
    (129, 33, None, 0.1),
    (640, 96, None, 1.0),
    (640, 96, None, 0.0),
    (1000, 700, (3, 1, 998, 700), 0.03),
    (1000, 700, (16, 5, 145, 38), 0.5),
    (4096, 2048, None, 0.02),
    (16384, 8400, None, 0.0005),      # 8416 groups: the chained prefix
])
def test_groups_match_numpy(cuda, w, h, roi, noise):
    import torch
    from opencuda_gb300 import _lib
    L = _lib.load()
    rng = np.random.default_rng(w + h)
    img = np.where(rng.random((h, w)) < noise, 255, rng.integers(0, 255, (h, w))).astype(np.uint8)
    x1, y1, x2, y2 = roi or (0, 0, w, h)
    sub = img[y1:y2, x1:x2] == 255
    rw, rh = x2 - x1, y2 - y1
    tx, ty = (rw + 127) // 128, (rh + 31) // 32
    ys, xs = np.nonzero(sub)
    order = np.lexsort((xs, ys, xs // 128, ys // 32))
    xs, ys = xs[order], ys[order]
    counts = np.bincount((ys // 32) * tx + xs // 128, minlength=tx * ty)
    t = torch.from_numpy(img).to(cuda)
    d = _lib.hl_image_desc(t.data_ptr(), t.stride(0), w, h, x1, y1, x2, y2)
    for _ in range(2):
        pts = torch.full((rw * rh + 16,), -1, dtype=torch.int32, device=cuda)
        off = torch.full((tx * ty + 1,), -1, dtype=torch.int32, device=cuda)
        cnt = torch.full((1,), -1, dtype=torch.int32, device=cuda)
        assert L.hl_compact_noalloc(C.byref(d), C.c_void_p(pts.data_ptr()),
                                    C.c_void_p(off.data_ptr()), C.c_void_p(cnt.data_ptr()),
                                    None) == 0
        st = C.c_int(-1)
        assert L.hl_compact_noalloc_status(C.byref(st), None) == 0 and st.value == 0
        n = len(xs)
        assert int(cnt.item()) == n
        assert np.array_equal(off.cpu().numpy(), np.concatenate(([0], np.cumsum(counts))))
        got = pts.cpu().numpy()
        assert np.array_equal(got[:n], (xs | (ys << 16)).astype(np.int32))
        assert np.all(got[n:] == -1)
