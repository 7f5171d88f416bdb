"""The operator's fused backward passes against the single kernels' entry points: the same bits in the
gradient, the bias gradient to FP32 summation order."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("source", ["plain", "up2", "pool2"])
@pytest.mark.parametrize("n,h,w,c", [(1, 2, 2, 8), (3, 6, 10, 96), (16, 16, 16, 128), (2, 64, 50, 32), (1, 4, 6, 3),
                                     (2, 34, 18, 24)])
def test_relu_backward_forms_its_gradient(plbm, source, n, h, w, c):
    from portlbm_gb300 import warmstart as ws
    lib = ws._fns()
    gen = torch.Generator(device="cuda").manual_seed(h * w + c)

    def rand(*shape):
        return torch.randn(shape, generator=gen, device="cuda").to(torch.bfloat16)

    y, skip = rand(n, h, w, c), rand(n, h, w, c)
    want, out = torch.empty_like(y), torch.empty_like(y)
    if source == "plain":
        src, code = rand(n, h, w, c), ws.GRAD
        want.copy_(src)
    elif source == "up2":
        src, code = rand(n, 2 * h, 2 * w, c), ws.GRAD_UP2
        assert lib.plbm_nn_up2_bwd(src.data_ptr(), want.data_ptr(), n, h, w, c, None) == 0
    else:
        src, code = rand(n, h // 2, w // 2, c), ws.GRAD_POOL2
        pooled = torch.empty_like(y)
        assert lib.plbm_nn_pool2_bwd(src.data_ptr(), pooled.data_ptr(), n, h, w, c, None) == 0
        assert lib.plbm_nn_add(pooled.data_ptr(), skip.data_ptr(), want.data_ptr(), want.numel(), None) == 0
    assert lib.plbm_nn_relu_bwd(y.data_ptr(), want.data_ptr(), want.numel(), None) == 0
    start = torch.randn(c, generator=gen, device="cuda")
    gb, kept = start.clone(), src.clone()
    assert lib.plbm_nn_relu_bwd_bias_from(code, src.data_ptr(), skip.data_ptr(), y.data_ptr(), out.data_ptr(),
                                          gb.data_ptr(), n, h, w, c, None) == 0
    torch.cuda.synchronize()
    assert torch.equal(out.view(torch.int16), want.view(torch.int16))
    assert torch.equal(src, kept)
    # FP32 summation of P terms: each partial sum is at most the sum of magnitudes
    terms = want.double().reshape(-1, c)
    bound = (terms.abs().sum(0) + start.double().abs()) * (n * h * w + 1) * 2.0 ** -24
    assert ((gb.double() - start.double() - terms.sum(0)).abs() <= bound).all()
    if source == "plain":     # in place
        assert lib.plbm_nn_relu_bwd_bias_from(code, src.data_ptr(), None, y.data_ptr(), src.data_ptr(), gb.data_ptr(),
                                              n, h, w, c, None) == 0
        assert torch.equal(src.view(torch.int16), want.view(torch.int16))


def test_arguments_are_checked(plbm):
    from portlbm_gb300 import warmstart as ws
    lib = ws._fns()
    t = torch.zeros(1, 2, 2, 8, dtype=torch.bfloat16, device="cuda")
    gb = torch.zeros(8, device="cuda")
    p = t.data_ptr()
    for source, skip, n in ((3, p, 1), (ws.GRAD_POOL2, None, 1), (ws.GRAD, None, 0)):
        assert lib.plbm_nn_relu_bwd_bias_from(source, p, skip, p, p, gb.data_ptr(), n, 2, 2, 8, None) != 0


@pytest.mark.parametrize("p,c", [(8, 1), (8, 3), (1000, 3), (65536 * 3 + 8, 3), (4096, 5), (24, 60), (120000, 12), (77, 3)])
def test_narrow_bias_gradient(plbm, p, c):
    """The bias gradient that comes with the weight gradient of a layer without ReLU, a few channels wide."""
    from portlbm_gb300 import warmstart as ws
    lib = ws._fns()
    gen = torch.Generator(device="cuda").manual_seed(p + c)
    g = torch.randn((1, 1, p, c), generator=gen, device="cuda").to(torch.bfloat16)
    x = torch.zeros((1, 1, p, 1), dtype=torch.bfloat16, device="cuda")
    gw, start = torch.zeros(c * 9, device="cuda"), torch.randn(c, generator=gen, device="cuda")
    gb = start.clone()
    assert lib.plbm_nn_conv_wgrad(x.data_ptr(), g.data_ptr(), gw.data_ptr(), gb.data_ptr(), 1, 1, p, 1, c, None) == 0
    terms = g.double().reshape(-1, c)
    bound = (terms.abs().sum(0) + start.double().abs()) * (p + 1) * 2.0 ** -24
    assert ((gb.double() - start.double() - terms.sum(0)).abs() <= bound).all()


@pytest.mark.parametrize("p,c", [(8, 1), (8, 3), (104, 3), (77, 3), (65536, 3), (1000, 5), (333, 16), (640000, 3)])
def test_mean_squared_error(plbm, p, c):
    from portlbm_gb300 import warmstart as ws
    lib = ws._fns()
    gen = torch.Generator(device="cuda").manual_seed(p + c)
    pred = torch.randn((p, c), generator=gen, device="cuda").to(torch.bfloat16)
    target = torch.randn((p, c), generator=gen, device="cuda")
    mask = (torch.rand(p, generator=gen, device="cuda") < 0.3).to(torch.int8)
    inv = 1.0 / max(1, int((mask == 0).sum()) * c)
    grad, loss = torch.empty_like(pred), torch.zeros(1, device="cuda")
    assert lib.plbm_nn_mse(pred.data_ptr(), target.data_ptr(), mask.data_ptr(), grad.data_ptr(), loss.data_ptr(), p, c,
                           inv, None) == 0
    d = torch.where((mask == 0)[:, None], pred.float() - target, 0.0)
    inv32 = torch.tensor(inv, dtype=torch.float32, device="cuda")
    assert torch.equal(grad, (2.0 * d * inv32).to(torch.bfloat16))
    want = (d.double() ** 2).sum() * inv
    assert abs(loss.double() - want) <= want * (p * c + 3) * 2.0 ** -24
