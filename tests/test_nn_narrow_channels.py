"""Every input channel count of the convolution whose threads write the im2col rows, at image edges and with channels
that leave part of a row's last chunk empty, against the float64 reference."""
import numpy as np
import pytest

from oracle import nn_ref

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("cin", [1, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("n,h,w,cout,relu", [(1, 2, 64, 16, 0), (3, 8, 16, 64, 1), (7, 128, 256, 9, 0)])
def test_narrow_input(plbm, cin, n, h, w, cout, relu):
    from portlbm_gb300 import warmstart as ws
    lib = ws._fns()
    assert lib.plbm_nn_conv_on_tensor_cores(h, w, cin, cout) == 1
    rng = np.random.default_rng(cin * 100 + h)
    x = nn_ref.bf16_round(rng.standard_normal((n, h, w, cin)))
    wt = nn_ref.bf16_round(rng.standard_normal((cout, 9 * cin)) / np.sqrt(9 * cin))
    b = rng.standard_normal(cout).astype(np.float32)
    xd, wd = (torch.tensor(a, dtype=torch.float32).to(torch.bfloat16).cuda() for a in (x, wt))
    bd = torch.tensor(b).cuda()
    size = n * h * w * cout
    y = torch.full((size + 4096,), 7.0, dtype=torch.bfloat16, device="cuda")
    assert lib.plbm_nn_conv_fwd(xd.data_ptr(), wd.data_ptr(), bd.data_ptr(), y.data_ptr(), n, h, w, cin, cout, relu, None) == 0
    got = y[:size].double().cpu().numpy().reshape(n, h, w, cout)
    want = nn_ref.conv_fwd(x, wt, b.astype(np.float64), bool(relu))
    # bfloat16 rounding of the result, FP32 accumulation of 9 cin terms and the bias
    bound = 2.0 ** -8 * np.abs(want) + (9 * cin + 2) * 2.0 ** -24 * nn_ref.conv_fwd(np.abs(x), np.abs(wt), np.abs(b).astype(np.float64))
    assert (np.abs(got - want) <= bound).all()
    assert (y[size:] == 7.0).all()
