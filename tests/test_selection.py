"""GPU: the proposal path's selection -- cut-offs, the top cells by bisection, local
maxima, dilation, the count and confidence fall-backs -- against the same rules in
numpy on the network's own logits: cells and windows selected, images that fall
back."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu
F = np.float32


def _level(v, target):
    if len(v) <= target:
        return F(-3.0e38)
    lo, hi = F(v.min() - F(1.0)), F(v.max())
    for _ in range(24):
        mid = F(F(0.5) * F(lo + hi))
        if int((v > mid).sum()) >= target:
            lo = mid
        else:
            hi = mid
    return lo


def _candidates(z, nms):
    if not nms:
        return np.ones_like(z, bool)
    out = np.zeros_like(z, bool)
    T, R = z.shape
    for t in range(T):
        for r in range(R):
            ok = True
            for tt in range(max(t - 1, 0), min(t + 2, T)):
                for rr in range(max(r - 1, 0), min(r + 2, R)):
                    if (tt, rr) != (t, r):
                        u = z[tt, rr]
                        ok &= not (u > z[t, r] or (u == z[t, r] and (tt, rr) < (t, r)))
            out[t, r] = ok
    return out


def _select(z, max_props, top_m, dt, dr, nms, conf):
    """(fallback, cells, windows) with both cut-offs at probability 1/2."""
    cand = _candidates(z, nms)
    v = z[cand]
    if (v > 0).sum() > max_props:
        return 1, 0, 0
    level = F(0)
    if top_m > 0:
        level = min(level, _level(v, top_m))
        if conf and len(v) > top_m and _level(v, top_m + 1) >= 0:
            return 2, 0, 0
    sel = cand & (z > level)
    grown = np.zeros_like(sel)
    for t, r in zip(*np.nonzero(sel)):
        grown[max(t - dt, 0):t + dt + 1, max(r - dr, 0):r + dr + 1] = True
    windows = 0
    for word in grown.reshape(-1, 32):      # runs of at most 8 in 32 rho cells
        n = 0
        for bit in list(word) + [False]:
            if not bit:
                windows += -(-n // 8)
            n = n + 1 if bit else 0
    return 0, int(grown.sum()), windows


@pytest.mark.parametrize("max_props,top_m,dt,dr,nms,conf", [
    (90 * 128, 0, 0, 0, False, False),
    (90 * 128, 5, 1, 2, False, False),
    (90 * 128, 300, 0, 1, False, True),
    (90 * 128, 12, 2, 40, True, False),
    (90 * 128, 1024, 3, 0, True, True),
    (50, 7, 0, 1, False, False),
    (0, 20, 1, 1, True, True),
])
@pytest.mark.parametrize("shift", [0.0, -1.5])
def test_selection_matches_numpy(cuda, max_props, top_m, dt, dr, nms, conf, shift):
    from opencuda_gb300.houghline import HoughLine, Image
    from opencuda_gb300.proposal import HoughNet, proposal_batch
    hl = HoughLine(detheta=np.pi / 360)
    net = HoughNet(seed=5)
    p = net.get_params()
    p[-1] += shift                          # the head's bias: fewer cells above the cut
    net.set_params(p)
    dev = [Image.from_host(cases.synth(3, 31, i)) for i in range(3)]
    occ, geos = net.occupancy(hl, dev)
    z = net.forward(occ, geos).cpu().numpy().astype(np.float32).reshape(-1, 90, 128)
    want = [_select(z[i], max_props, top_m, dt, dr, nms, conf) for i in range(len(dev))]
    rc, _, st = proposal_batch(hl, net, dev, 16, [300] * len(dev), p_cut=0.5,
                               max_props=max_props, dilate_theta=dt, dilate_rho=dr, top_m=top_m,
                               nms=nms, p_conf=0.5 if conf else 0.0)
    assert rc == 0
    assert st["fallback"] == sum(w[0] != 0 for w in want)
    assert st["cells"] == sum(w[1] for w in want)
    assert st["windows"] == sum(w[2] for w in want)
