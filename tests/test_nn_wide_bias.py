"""Bias gradients of layers with more channels than a block of the 16-byte kernel has units for (2048)."""
import subprocess
import sys

import pytest

from conftest import ROOT

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("c", [2048, 2056, 4096])
def test_no_division_by_zero_on_the_host(plbm, c):
    """In a process of its own.  Without a GPU the launch fails before a pointer is used."""
    if torch.cuda.is_available():
        pytest.skip("the addresses are made up")
    code = ("from portlbm_gb300 import warmstart as ws; lib = ws._fns(); "
            f"print(lib.plbm_nn_relu_bwd_bias(4096, 8192, 4096, 4, {c}, None), "
            f"lib.plbm_nn_relu_bwd_bias_from(0, 4096, None, 8192, 4096, 4096, 1, 2, 2, {c}, None))")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.split() == ["-4", "-4"], (r.returncode, r.stdout, r.stderr)


@pytest.mark.gpu
@pytest.mark.parametrize("source", ["in place", "plain", "up2", "pool2"])
@pytest.mark.parametrize("n,h,w,c", [(1, 2, 4, 2048), (2, 4, 6, 2056), (1, 16, 16, 4096)])
def test_wide_layers(plbm, source, n, h, w, c):
    from portlbm_gb300 import warmstart as ws
    lib = ws._fns()
    gen = torch.Generator(device="cuda").manual_seed(c + h)

    def rand(*shape):
        return torch.randn(shape, generator=gen, device="cuda").to(torch.bfloat16)

    y, skip, out = rand(n, h, w, c), rand(n, h, w, c), torch.empty((n, h, w, c), dtype=torch.bfloat16, device="cuda")
    gb = torch.zeros(c, device="cuda")
    if source in ("in place", "plain"):
        src = rand(n, h, w, c)
        g = src.float()
    elif source == "up2":
        src = rand(n, 2 * h, 2 * w, c)
        f = src.float()     # the four terms in the kernel's order
        g = (f[:, ::2, ::2] + f[:, ::2, 1::2] + f[:, 1::2, ::2] + f[:, 1::2, 1::2]).to(torch.bfloat16).float()
    else:
        src = rand(n, h // 2, w // 2, c)
        pooled = (0.25 * src.float()).to(torch.bfloat16).float()
        g = pooled.repeat_interleave(2, 1).repeat_interleave(2, 2) + skip.float()
    want = torch.where(y > 0, g.to(torch.bfloat16), torch.zeros((), dtype=torch.bfloat16, device="cuda"))
    if source == "in place":
        assert lib.plbm_nn_relu_bwd_bias(y.data_ptr(), src.data_ptr(), gb.data_ptr(), n * h * w, c, None) == 0
        out = src
    else:
        code = {"plain": ws.GRAD, "up2": ws.GRAD_UP2, "pool2": ws.GRAD_POOL2}[source]
        assert lib.plbm_nn_relu_bwd_bias_from(code, src.data_ptr(), skip.data_ptr(), y.data_ptr(), out.data_ptr(),
                                              gb.data_ptr(), n, h, w, c, None) == 0
    assert torch.equal(out, want)
    terms = want.double().reshape(-1, c)      # FP32 summation of P terms
    assert ((gb.double() - terms.sum(0)).abs() <= terms.abs().sum(0) * (n * h * w + 1) * 2.0 ** -24).all()
