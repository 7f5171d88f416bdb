"""The activations a forward pass keeps are a dict of tensors, in the order they are computed."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_activations_are_a_dict(plbm):
    from portlbm_gb300 import warmstart as ws
    model = ws.NeuralOperator(1)
    assert not hasattr(model, "acts")
    x = torch.randn((2, 32, 16, 4), device="cuda").to(torch.bfloat16)
    out = model.forward(x, 2, 32, 16)
    acts = model.acts
    assert isinstance(acts, dict) and acts is model.acts
    names = ["in"]
    for lvl in range(5):
        names += [f"e{lvl}a", f"e{lvl}b"] + ([f"p{lvl}"] if lvl < 4 else [])
    for lvl in (3, 2, 1, 0):
        names += [f"u{lvl}", f"d{lvl}a", f"s{lvl}", f"d{lvl}b"]
    assert list(acts) == names + ["out"]
    assert acts["in"] is x and acts["out"] is out and "e0a" in acts and "e9a" not in acts
    assert {k: tuple(v.shape) for k, v in acts.items()}["e4b"] == (2, 2, 1, 128)
    kept = acts["d0b"].clone()
    model.forward(torch.zeros_like(x), 2, 32, 16)     # a pass of its own: what was kept stays
    assert model.acts is not acts and torch.equal(acts["d0b"], kept)


def test_backward_reads_the_dict(plbm):
    from portlbm_gb300 import warmstart as ws
    model = ws.NeuralOperator(1)
    x, g = (torch.randn((1, 16, 16, c), device="cuda").to(torch.bfloat16) for c in (4, 3))
    model.forward(x, 1, 16, 16)
    model.acts["in"] = torch.zeros_like(x)            # the first layer's weight gradient is then zero
    model.zero_grad()
    model.backward(g)
    assert float(model.enc[0].gw.abs().max()) == 0.0 and float(model.enc[1].gw.abs().max()) > 0.0
