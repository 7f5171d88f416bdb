"""A launch that is refused is reported by its own call, and not again by the next one."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_the_next_call_succeeds(plbm):
    from portlbm_gb300 import warmstart as ws
    lib = ws._fns()
    t, f = torch.ones(64, 8, dtype=torch.bfloat16, device="cuda"), torch.zeros(512, device="cuda")
    m = torch.zeros(64, dtype=torch.int8, device="cuda")
    p = t.data_ptr()
    refused = (lambda: lib.plbm_nn_mse(p, f.data_ptr(), m.data_ptr(), p, f.data_ptr(), 0, 8, 1.0, None),   # empty grids
               lambda: lib.plbm_nn_add(p, p, p, 0, None),
               lambda: lib.plbm_nn_pool2(p, p, 1, 0, 8, 8, None))
    for call in refused:
        assert call() != 0
        assert lib.plbm_nn_relu_bwd(p, p, 512, None) == 0
        assert lib.plbm_nn_up2_bwd(p, p, 1, 2, 2, 8, None) == 0
    props = plbm.Properties("nptl", "stream", False, 32, 100, 10, "circle", 16, 32, 0.0, 0.0, 1.02, 0.0, 0.0, 1.0, 0.8)
    assert refused[0]() != 0
    hd = plbm.create_handler(props, precision="f32")
    hd.run_steps(5)
    hd.close()
