"""Weight and bias gradients of few pixels in small images, on both sides of the line between the mma.sync and the
TMA-fed kernel, against the float64 reference (bound: FP32 accumulation of P terms, of their magnitudes' sum)."""
import numpy as np
import pytest

from oracle import nn_ref

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,h,w", [(1, 4, 4), (8, 8, 8), (32, 4, 4), (33, 4, 4), (9, 8, 8), (1, 1, 1), (1, 31, 16),
                                   (40, 4, 4), (41, 4, 4), (40, 5, 7), (41, 5, 7)])
@pytest.mark.parametrize("bias", [True, False])
@pytest.mark.parametrize("cin,cout", [(96, 96), (128, 128), (32, 128), (96, 64), (64, 96), (128, 3)])
def test_weight_gradient(plbm, n, h, w, bias, cin, cout):
    from portlbm_gb300 import warmstart as ws
    lib = ws._fns()
    rng = np.random.default_rng(h * w + cin + cout)
    x, g = (nn_ref.bf16_round(rng.standard_normal((n, h, w, c))) for c in (cin, cout))
    start = rng.standard_normal((cout, 9 * cin)).astype(np.float32)
    xd, gd = (torch.tensor(a, dtype=torch.float32).to(torch.bfloat16).cuda() for a in (x, g))
    gw, gb = torch.tensor(start).cuda(), torch.zeros(cout, device="cuda")
    assert lib.plbm_nn_conv_wgrad(xd.data_ptr(), gd.data_ptr(), gw.data_ptr(), gb.data_ptr() if bias else None, n, h, w, cin,
                                  cout, None) == 0
    want, want_b = nn_ref.conv_wgrad(x, g)
    size, size_b = nn_ref.conv_wgrad(np.abs(x), np.abs(g))
    eps = (n * h * w + 2) * 2.0 ** -24
    assert (np.abs(gw.double().cpu().numpy() - want - start) <= eps * (size + np.abs(start))).all()
    assert (np.abs(gb.double().cpu().numpy() - want_b * bias) <= eps * size_b * bias).all()
