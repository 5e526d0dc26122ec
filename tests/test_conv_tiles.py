"""The convolution kernels at the edges of their 8 x 16 output tiles, and the
coarse head where its fixed point leaves 32 bits, against the CPU oracle
(oracle/cnn_oracle.py).  Tolerances: outputs are BF16 roundings (2^-9) of sums
whose FP32 error is far below that, so 2^-7 of the value covers two roundings;
one-channel outputs are FP32 sums of 288 products, 1e-5 of their size."""
import ctypes as C

import numpy as np
import pytest

from oracle import cnn_oracle as CO
from test_cnn import _close, _dev_bf16, _run_conv, lib  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W", [(1, 1), (15, 7), (16, 8), (17, 9), (32, 16), (33, 17), (3, 200)])
@pytest.mark.parametrize("cin,cout,stride", [(32, 32, 1), (32, 32, 2), (32, 5, 1), (32, 16, 2),
                                             (32, 17, 1), (1, 32, 1), (1, 7, 2)])
def test_conv_at_tile_edges(lib, H, W, cin, cout, stride):  # noqa: F811
    import torch
    rng = np.random.default_rng(H * 1000 + W * 10 + cout + stride)
    x = CO.bf16_round(rng.standard_normal((3, H, W, cin)).astype(np.float32))
    w = CO.bf16_round((rng.standard_normal((cout, 9 * cin)) * 0.2).astype(np.float32))
    bias = rng.standard_normal(cout).astype(np.float32) * 0.1
    got = _run_conv(lib, torch, x, w, bias, stride, True)
    _close(got, CO.conv3x3(x, w, bias, stride, True))


@pytest.mark.parametrize("H,W", [(1, 1), (16, 8), (17, 9), (5, 70)])
def test_stride2_gradient_at_tile_edges(lib, H, W):  # noqa: F811
    import torch
    rng = np.random.default_rng(H * 100 + W)
    dy = CO.bf16_round(rng.standard_normal((2, H, W, 32)).astype(np.float32))
    w = CO.bf16_round((rng.standard_normal((32, 288)) * 0.2).astype(np.float32))
    got = _run_conv(lib, torch, dy, CO.transpose_weights(w), None, 2, False, mode=1)
    _close(got, CO.conv3x3_dx(dy, w, 2 * H, 2 * W, stride=2))


def test_weights_off_16_bytes(lib):  # noqa: F811
    """Weights whose address is only 2-byte aligned take scalar loads."""
    import torch
    rng = np.random.default_rng(3)
    x = CO.bf16_round(rng.standard_normal((1, 20, 11, 32)).astype(np.float32))
    w = CO.bf16_round((rng.standard_normal((32, 288)) * 0.2).astype(np.float32))
    buf = torch.zeros(32 * 288 + 1, dtype=torch.int16, device="cuda")
    buf[1:] = _dev_bf16(torch, w).flatten()
    dx, y = _dev_bf16(torch, x), torch.zeros((1, 20, 11, 32), dtype=torch.int16, device="cuda")
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    rc = lib.hl_cnn_conv3x3(C.c_void_p(dx.data_ptr()), C.c_void_p(buf.data_ptr() + 2), None,
                            C.c_void_p(y.data_ptr()), None, 1, 20, 11, 32, 32, 1, 0, 0,
                            C.c_void_p(st.data_ptr()), None)
    assert rc == 0
    torch.cuda.synchronize()
    got = CO.from_bf16_bits(y.cpu().numpy().view(np.uint16))
    _close(got, CO.conv3x3(x, w, None, 1, False))


@pytest.mark.parametrize("scale", [1.0, 3.0e3])
def test_head_beyond_32_bits(lib, scale):  # noqa: F811
    """scale 3000: evidence of hundreds, above the 128 that 32 bits of fixed
    point hold; tolerance as the network's own test (BF16 activations)."""
    import torch
    from opencuda_gb300.proposal import HoughNet
    rng = np.random.default_rng(8)
    occ = CO.bf16_round((rng.random((2, 256, 256)) < 0.1).astype(np.float32) * 0.25)
    geos = [(32.0, -2896.0, 128 / 5793.0, 64, 64), (16.0, -900.0, 128 / 1801.0, 13, 50)]
    net = HoughNet(seed=5)
    p = net.get_params()
    o = sum(co * 9 * ci + co for ci, co, _, _ in CO.LAYERS[:-1])
    p[o:o + 289] *= scale
    net.set_params(p)
    z = net.forward(_dev_bf16(torch, occ), HoughNet.geos(geos)).cpu().numpy()
    zr, _, e, _, _ = CO.net_forward(occ, geos, p.astype(np.float64))
    assert (np.abs(e).max() > 128) == (scale > 1)
    assert np.abs(z - zr).max() <= 1e-2 * max(1.0, np.abs(zr).max())


@pytest.mark.parametrize("B", [1, 3])
def test_training_step_gradients_and_update(lib, B):  # noqa: F811
    """Gradients of one to three maps against the oracle (5% of a layer's
    norm: BF16 activations and gradients, 2^-9 each, through six layers), and
    the first Adam step from them: w - lr g / (|g| + eps), both bias
    corrections cancelling, to FP32 rounding."""
    import torch
    from opencuda_gb300.proposal import HoughNet
    rng = np.random.default_rng(40 + B)
    occ = CO.bf16_round((rng.random((B, 256, 256)) < 0.05).astype(np.float32) * 0.125)
    geos = [(32.0, -2896.0, 128 / 5793.0, 64, 64), (16.0, -1448.0, 128 / 2897.0, 64, 50),
            (4.0, -300.0, 128 / 601.0, 9, 64)][:B]
    net = HoughNet(seed=21)
    p = net.get_params()
    tgt = (rng.random((B, 90, 128)) < 0.005).astype(np.float32)
    loss = net.train_step(_dev_bf16(torch, occ), HoughNet.geos(geos), torch.from_numpy(tgt).cuda(),
                          1e-3, 30.0)
    g, q = net.get_grads(), net.get_params()
    lref, gref = CO.net_loss_grads(occ, geos, p.astype(np.float64), tgt, 30.0)
    assert abs(loss - lref) <= 1e-3 * abs(lref) + 1e-5
    o = 0
    for ci, co, _, _ in CO.LAYERS:
        for n in (co * 9 * ci, co):
            a, b = g[o:o + n], gref[o:o + n]
            assert np.linalg.norm(a - b) <= 0.05 * max(np.linalg.norm(b), 1e-12), (o, n)
            o += n
    assert np.allclose(g[o:], gref[o:], rtol=1e-3, atol=1e-6)
    gc = np.clip(g.astype(np.float64), -1, 1)
    assert np.allclose(q, p - 1e-3 * gc / (np.abs(gc) + 1e-8), rtol=1e-5, atol=2e-6)
