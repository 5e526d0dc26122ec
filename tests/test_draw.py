"""Line drawing against the per-pixel rule in numpy (float32, every operation
rounded as written): all angles, distances on both sides of zero and beyond
the image, rho steps, ROIs of odd sizes at odd offsets."""
import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _want(w, h, lines, cosv, sinv, derho):
    f = np.float32
    out = np.zeros((h, w), np.uint8)
    c = np.arange(w, dtype=f)[None, :]
    r = np.arange(h, dtype=f)[:, None]
    irho = f(1.0) / f(derho)
    for k, d in lines:
        x, y = (c * f(cosv[k])).astype(f), (r * f(sinv[k])).astype(f)
        if derho != 1:
            x, y = (x * irho).astype(f), (y * irho).astype(f)
        out[np.trunc((x + y).astype(f)).astype(np.int64) == d] = 255
    return out


@pytest.mark.parametrize("w,h,derho", [(1, 1, 1), (127, 129, 1), (640, 33, 1), (257, 500, 2),
                                       (300, 200, 7), (1025, 1023, 1)])
def test_draw_matches_per_pixel_rule(cuda, w, h, derho):
    import torch
    from opencuda_gb300 import _lib
    from opencuda_gb300.houghline import HoughLine
    hl = HoughLine(detheta=math.pi / 180, derho=float(derho))
    cosv, sinv = hl.trig_table()
    rng = np.random.default_rng(w * h + derho)
    ks = list(range(0, 180, 3)) + [1, 44, 45, 46, 89, 90, 91, 134, 135, 136, 179]
    diag = int(math.hypot(w, h) / derho) + 2
    lines = [(k, int(rng.integers(-diag, diag + 1))) for k in ks]
    lines += [(k, d) for k in (0, 45, 90, 135, 179) for d in (0, 1, -1, diag, -diag)]
    lines += [(10, 2**31 - 1), (100, -2**31), (60, 10**8)]
    theta = [np.float32(k * (math.pi / 180)) for k in range(180)]
    recs = (_lib.hl_line * len(lines))(*[_lib.hl_line(float(theta[k]), d, 1) for k, d in lines])
    buf = torch.zeros((h + 3, w + 10), dtype=torch.uint8, device=cuda)
    desc = _lib.hl_image_desc(buf.data_ptr(), buf.stride(0), w + 10, h + 3, 5, 2, 5 + w, 2 + h)
    rc = _lib.load().hl_draw_lines(hl.handle, C.byref(desc), recs, len(lines), None)
    assert rc == 0
    got = buf.cpu().numpy()
    want = np.zeros_like(got)
    want[2:2 + h, 5:5 + w] = _want(w, h, lines, cosv, sinv, derho)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("room", [3, 32, 2000])
def test_plain_draw_draws_the_lines_found(cuda, room):
    """hl_plain_draw with room for fewer lines than there are, for more, and
    past the queued launch: the image holds exactly the returned lines."""
    import cases
    import torch
    from opencuda_gb300 import _lib
    from opencuda_gb300.houghline import HoughLine, Image
    img = cases.synth_custom(900, 700, 12, 200, 900, 8000, 4)
    hl = HoughLine(detheta=math.pi / 360, threshold=150)
    cosv, sinv = hl.trig_table()
    src = Image.from_host(img)
    dst = torch.zeros((700, 900), dtype=torch.uint8, device=cuda)
    dd = _lib.hl_image_desc(dst.data_ptr(), 900, 900, 700, 0, 0, 900, 700)
    out, lm, ds = (_lib.hl_line * room)(), C.c_int(room), src.desc()
    rc = _lib.load().hl_plain_draw(hl.handle, C.byref(ds), C.byref(dd), C.byref(lm), out, None)
    assert rc == 0 and lm.value == len(hl.houghLine(src, None, room)[1]) > 0
    lines = [(int(round(out[i].angle / (math.pi / 360))), out[i].distance)
             for i in range(lm.value)]
    assert np.array_equal(dst.cpu().numpy(), _want(900, 700, lines, cosv, sinv, 1))
