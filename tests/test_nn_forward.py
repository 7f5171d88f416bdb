"""The operator's one-call forward pass and its input assembly against the single kernels' entry points:
the same bits in every activation, for layers of few and many tiles and a batch beyond one launch's
samples."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,h,w", [(1, 16, 128), (2, 48, 64), (3, 256, 256), (17, 128, 128)])
def test_one_call_forward_is_the_layers_one_by_one(plbm, n, h, w):
    from portlbm_gb300 import warmstart as ws
    model = ws.NeuralOperator(3)
    lib = model.lib
    for i, layer in enumerate(model.layers):
        layer.b.copy_(0.01 * torch.arange(layer.cout, device="cuda") - 0.1)
    rng = np.random.default_rng(n)
    masks = torch.from_numpy((rng.random((n, h, w)) < 0.3).astype(np.int8)).cuda()
    x = model.assemble(masks, [ws.features(w, 1.02 + 0.001 * i, 1.0, 0.8) for i in range(n)])
    out = model.forward(x, n, h, w)
    got = model.acts
    s = torch.cuda.current_stream().cuda_stream or None

    def buf(*shape):
        return torch.empty(shape, dtype=torch.bfloat16, device="cuda")

    def conv(layer, v, name):
        y = buf(*v.shape[:3], layer.cout)
        assert lib.plbm_nn_conv_fwd(v.data_ptr(), layer.wb.data_ptr(), layer.b.data_ptr(), y.data_ptr(), *v.shape[:3],
                                    layer.cin, layer.cout, int(layer.relu), s) == 0
        assert torch.equal(y.view(torch.int16), got[name].view(torch.int16)), name
        return y

    cur, skips = x, []
    for lvl in range(5):
        cur = conv(model.enc[2 * lvl + 1], conv(model.enc[2 * lvl], cur, f"e{lvl}a"), f"e{lvl}b")
        skips.append(cur)
        if lvl < 4:
            p = buf(n, h >> lvl + 1, w >> lvl + 1, cur.shape[-1])
            assert lib.plbm_nn_pool2(cur.data_ptr(), p.data_ptr(), n, h >> lvl, w >> lvl, cur.shape[-1], s) == 0
            assert torch.equal(p, got[f"p{lvl}"])
            cur = p
    for k, lvl in enumerate((3, 2, 1, 0)):
        u = buf(n, h >> lvl, w >> lvl, cur.shape[-1])
        assert lib.plbm_nn_up2(cur.data_ptr(), u.data_ptr(), n, h >> lvl, w >> lvl, cur.shape[-1], s) == 0
        assert torch.equal(u, got[f"u{lvl}"])
        a = conv(model.dec[2 * k], u, f"d{lvl}a")
        t = torch.empty_like(a)
        assert lib.plbm_nn_add(a.data_ptr(), skips[lvl].data_ptr(), t.data_ptr(), t.numel(), s) == 0
        assert torch.equal(t, got[f"s{lvl}"])
        cur = conv(model.dec[2 * k + 1], t, f"d{lvl}b")
    assert torch.equal(conv(model.head, cur, "out"), out)


@pytest.mark.parametrize("n,h,w", [(1, 3, 5), (64, 7, 9), (130, 33, 17), (2, 300, 260)])
def test_assembly_from_host_scalars(plbm, n, h, w):
    from portlbm_gb300 import warmstart as ws
    model = ws.NeuralOperator(0)
    rng = np.random.default_rng(n)
    masks = torch.from_numpy((rng.random((n, h, w)) < 0.4).astype(np.int8)).cuda()
    feats = rng.standard_normal((n, 3)).astype(np.float32)
    x = model.assemble(masks, feats)
    y = torch.empty_like(x)
    f = torch.from_numpy(feats).cuda()
    assert model.lib.plbm_nn_assemble(masks.data_ptr(), f.data_ptr(), y.data_ptr(), n, h, w, 4,
                                      torch.cuda.current_stream().cuda_stream or None) == 0
    assert torch.equal(x.view(torch.int16), y.view(torch.int16))
