"""Image extents that the operator's halvings do not divide: refused where an up-sampling would read beyond its
input, and the gradient of a pooling zero where it pooled nothing."""
import ctypes

import pytest

torch = pytest.importorskip("torch")
PLBM_ERR_ARGUMENT = -7


@pytest.mark.parametrize("n,h,w", [(1, 100, 64), (1, 64, 100), (2, 17, 16), (1, 8, 16), (0, 16, 16), (1, 0, 16), (1, 16, 0),
                                   (1, -16, 16)])
def test_forward_refuses_extents_that_do_not_halve(plbm, n, h, w):
    """Checked before anything is launched: no pointer is read."""
    from portlbm_gb300 import warmstart as ws
    lib = ws._fns()
    acts = (ctypes.c_void_p * 31)(*[4096] * 31)
    layers = (ws._CLayer * 19)(*[ws._CLayer(4096, 4096, 32, 32, 1)] * 19)
    assert lib.plbm_nn_unet_forward(4096, acts, layers, 5, n, h, w, None) == PLBM_ERR_ARGUMENT


@pytest.mark.parametrize("n,h,w,c", [(1, 15, 16, 8), (2, 16, 7, 3), (1, 1, 2, 8), (0, 2, 2, 8)])
def test_up_sampling_refuses_odd_extents(plbm, n, h, w, c):
    from portlbm_gb300 import warmstart as ws
    assert ws._fns().plbm_nn_up2(4096, 8192, n, h, w, c, None) == PLBM_ERR_ARGUMENT


@pytest.mark.gpu
@pytest.mark.parametrize("n,h,w,c", [(1, 5, 6, 8), (3, 8, 7, 32), (2, 9, 11, 3), (1, 1, 4, 8), (2, 7, 1, 5)])
def test_pooling_gradient_of_odd_extents(plbm, n, h, w, c):
    from portlbm_gb300 import warmstart as ws
    lib = ws._fns()
    gen = torch.Generator(device="cuda").manual_seed(h * w + c)
    pooled = torch.randn((n, h // 2, w // 2, c), generator=gen, device="cuda").to(torch.bfloat16)
    want = torch.zeros((n, h, w, c), device="cuda")
    want[:, :h // 2 * 2, :w // 2 * 2] = (0.25 * pooled.float()).repeat_interleave(2, 1).repeat_interleave(2, 2)
    got = torch.full((n, h, w, c), 7.0, device="cuda").to(torch.bfloat16)
    # room behind the pooled image, so that its address is one a kernel may form
    src = torch.cat([pooled.reshape(-1), torch.full((4 * w * c,), 9.0, dtype=torch.bfloat16, device="cuda")])
    assert lib.plbm_nn_pool2_bwd(src.data_ptr(), got.data_ptr(), n, h, w, c, None) == 0
    assert torch.equal(got.float(), want)
    skip, y = (torch.randn((n, h, w, c), generator=gen, device="cuda").to(torch.bfloat16) for _ in range(2))
    out, gb = torch.empty_like(skip), torch.zeros(c, device="cuda")
    assert lib.plbm_nn_relu_bwd_bias_from(ws.GRAD_POOL2, src.data_ptr(), skip.data_ptr(), y.data_ptr(), out.data_ptr(),
                                          gb.data_ptr(), n, h, w, c, None) == 0
    masked = torch.where(y > 0, (want + skip.float()).to(torch.bfloat16), 0.0)
    assert torch.equal(out, masked.to(torch.bfloat16))
