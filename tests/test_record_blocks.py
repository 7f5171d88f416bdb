"""Block shapes of small domains in the collision layout: the values do not depend on them (the stream layout's
blocks are others)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alg", ["nptl", "lptl", "nsol"])
@pytest.mark.parametrize("precision", ["f64_q60", "f64_strict", "f64_fast", "f32", "bf16s"])
@pytest.mark.parametrize("w,h", [(3, 4), (62, 30), (95, 131), (803, 61), (1201, 33), (513, 129)])
def test_records_and_stream_agree(plbm, alg, precision, w, h):
    mask = (np.random.default_rng(w).random((h, w)) < 0.15).astype(np.int8)
    results = []
    for lay in ("collision", "stream"):
        props = plbm.Properties(alg, lay, False, 1024, 10 ** 6, 10 ** 6, "circle", h, w, 0.0, 0.0, 1.03, 0.0, 0.0, 1.0, 0.7)
        hd = plbm.create_handler(props, precision=precision, mask=mask)
        hd.run_steps(7)
        hd.run_steps(1)
        hd.run_steps(22)
        hd.sync_results()
        results.append([hd.get_densities(), hd.get_x_velocities(), hd.get_y_velocities(), hd.get_absolute_velocities()])
        hd.close()
    for a, b in zip(*results):
        assert np.array_equal(a, b)
