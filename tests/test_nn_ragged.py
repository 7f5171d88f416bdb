"""Convolutions on images that 128-pixel tiles do not cover exactly, and layers of few tiles (output
channels split over CTAs, K blocks of 32 and 64 channels), on the TMA-fed tensor-core kernels against the
float64 reference.  Bounds: FP32 accumulation of K terms (K 2^-24 of their magnitudes' sum), then the
rounding to bfloat16 (2^-8 of the value)."""
import ctypes

import numpy as np
import pytest

from oracle import nn_ref

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SHAPES = [(1, 1, 1, 32, 3), (2, 5, 7, 64, 48), (1, 9, 24, 96, 128), (3, 18, 8, 128, 128), (1, 6, 192, 32, 64),
          (1, 3, 130, 64, 96), (2, 4, 4, 128, 96), (1, 17, 48, 96, 64), (1, 16, 24, 32, 3), (1, 5, 300, 64, 5),
          (1, 16, 16, 128, 128), (40, 8, 16, 64, 96)]


def bf(a):
    return torch.tensor(a, dtype=torch.float32).to(torch.bfloat16).cuda()


def host(t):
    return t.float().cpu().numpy().astype(np.float64)


@pytest.mark.parametrize("n,h,w,cin,cout", SHAPES)
def test_ragged_convolution_and_gradients(plbm, n, h, w, cin, cout):
    from portlbm_gb300 import warmstart as ws
    lib = ws._fns()
    assert lib.plbm_nn_conv_on_tensor_cores(h, w, cin, cout) == 1
    assert lib.plbm_nn_wgrad_on_tensor_cores(h, w, cin, cout) == 1
    rng = np.random.default_rng(h * w + cin)
    x = nn_ref.bf16_round(rng.standard_normal((n, h, w, cin)))
    wt = nn_ref.bf16_round(rng.standard_normal((cout, 9 * cin)) / np.sqrt(9 * cin))
    b = rng.standard_normal(cout).astype(np.float32)
    g = nn_ref.bf16_round(rng.standard_normal((n, h, w, cout)))
    xd, wd, gd, bd = bf(x), bf(wt), bf(g), torch.tensor(b).cuda()
    flipped = torch.tensor(wt.reshape(cout, 9, cin)[:, ::-1].transpose(2, 1, 0).copy(), dtype=torch.float32)
    flipped = flipped.to(torch.bfloat16).cuda()

    def close(got, ref, magnitudes, terms, rounded=True):
        assert (np.abs(got - ref) <= (2.0 ** -8 * np.abs(ref) if rounded else 0.0) + (terms + 2) * 2.0 ** -24 * magnitudes).all()

    # guard values behind the outputs: tiles reach beyond the image, stores must not
    y = torch.full((n * h * w * cout + 4096,), 7.0, dtype=torch.bfloat16, device="cuda")
    for relu in (0, 1):
        assert lib.plbm_nn_conv_fwd(xd.data_ptr(), wd.data_ptr(), bd.data_ptr(), y.data_ptr(), n, h, w, cin, cout, relu,
                                    None) == 0
        size = n * h * w * cout
        close(host(y[:size]).reshape(n, h, w, cout), nn_ref.conv_fwd(x, wt, b.astype(np.float64), bool(relu)),
              nn_ref.conv_fwd(np.abs(x), np.abs(wt), np.abs(b).astype(np.float64)), 9 * cin)
        assert (y[size:] == 7.0).all()
    # the same values from a buffer that TMA cannot read
    shifted = torch.empty(xd.numel() + 1, dtype=torch.bfloat16, device="cuda")[1:]
    shifted.copy_(xd.reshape(-1))
    y2 = torch.empty(size, dtype=torch.bfloat16, device="cuda")
    assert lib.plbm_nn_conv_fwd(shifted.data_ptr(), wd.data_ptr(), bd.data_ptr(), y2.data_ptr(), n, h, w, cin, cout, 1,
                                None) == 0
    close(host(y2).reshape(n, h, w, cout), nn_ref.conv_fwd(x, wt, b.astype(np.float64), True),
          nn_ref.conv_fwd(np.abs(x), np.abs(wt), np.abs(b).astype(np.float64)), 9 * cin)
    size = n * h * w * cin
    gx = torch.full((size + 4096,), 7.0, dtype=torch.bfloat16, device="cuda")
    for call in (lambda: lib.plbm_nn_conv_dgrad(gd.data_ptr(), wd.data_ptr(), gx.data_ptr(), n, h, w, cin, cout, None),
                 lambda: lib.plbm_nn_conv_dgrad_pre(gd.data_ptr(), wd.data_ptr(), flipped.data_ptr(), gx.data_ptr(), n, h,
                                                    w, cin, cout, None)):
        gx[:size].zero_()
        assert call() == 0
        close(host(gx[:size]).reshape(n, h, w, cin), nn_ref.conv_dgrad(g, wt, cin),
              nn_ref.conv_dgrad(np.abs(g), np.abs(wt), cin), 9 * cout)
        assert (gx[size:] == 7.0).all()
    start = rng.standard_normal((cout, 9 * cin)).astype(np.float32)
    gw, gb = torch.tensor(start).cuda(), torch.zeros(cout, device="cuda")
    assert lib.plbm_nn_conv_wgrad(xd.data_ptr(), gd.data_ptr(), gw.data_ptr(), gb.data_ptr(), n, h, w, cin, cout, None) == 0
    want, want_b = nn_ref.conv_wgrad(x, g)
    size_w, size_b = nn_ref.conv_wgrad(np.abs(x), np.abs(g))
    close(gw.double().cpu().numpy(), want + start, size_w + np.abs(start), n * h * w, rounded=False)
    close(gb.double().cpu().numpy(), want_b, size_b, n * h * w, rounded=False)
    failed = ctypes.c_int(1)
    assert lib.plbm_nn_status(ctypes.byref(failed)) == 0 and failed.value == 0


@pytest.mark.parametrize("n,h,w,cin,cout", [(5, 256, 128, 4, 32), (5, 256, 128, 3, 12), (4, 512, 64, 7, 5), (1, 2, 64, 3, 64),
                                           (3, 4, 256, 4, 3)])
def test_narrow_layers_of_many_and_few_tiles(plbm, n, h, w, cin, cout):
    """The kernel whose threads write the im2col rows, with more tiles than CTAs share the GPU and with few."""
    from portlbm_gb300 import warmstart as ws
    lib = ws._fns()
    assert lib.plbm_nn_conv_on_tensor_cores(h, w, cin, cout) == 1
    rng = np.random.default_rng(h + cin)
    x = nn_ref.bf16_round(rng.standard_normal((n, h, w, cin)))
    wt = nn_ref.bf16_round(rng.standard_normal((cout, 9 * cin)) / np.sqrt(9 * cin))
    b = rng.standard_normal(cout).astype(np.float32)
    xd, wd, bd = bf(x), bf(wt), torch.tensor(b).cuda()
    size = n * h * w * cout
    y = torch.full((size + 4096,), 7.0, dtype=torch.bfloat16, device="cuda")
    assert lib.plbm_nn_conv_fwd(xd.data_ptr(), wd.data_ptr(), bd.data_ptr(), y.data_ptr(), n, h, w, cin, cout, 0, None) == 0
    want = nn_ref.conv_fwd(x, wt, b.astype(np.float64), False)
    bound = 2.0 ** -8 * np.abs(want) + (9 * cin + 2) * 2.0 ** -24 * nn_ref.conv_fwd(np.abs(x), np.abs(wt), np.abs(b).astype(np.float64))
    assert (np.abs(host(y[:size]).reshape(n, h, w, cout) - want) <= bound).all()
    assert (y[size:] == 7.0).all()
    failed = ctypes.c_int(1)
    assert lib.plbm_nn_status(ctypes.byref(failed)) == 0 and failed.value == 0
