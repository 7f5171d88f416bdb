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
