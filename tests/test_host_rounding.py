"""Boundary constants are formed on the host with every operation rounded, as the oracle's: with an inlet
velocity the drop-in form is bit-identical to it on machines with fused multiply-adds too."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("alg", ["nptl", "lptl", "npol", "nsol"])
@pytest.mark.parametrize("v_in,v_out", [((0.2, 0.0), (0.0, 0.0)), ((0.07, 0.013), (0.11, -0.003))])
def test_velocity_boundaries(plbm, oracle_mod, alg, v_in, v_out):
    w, h, steps = 67, 35, 30
    props = plbm.Properties(alg, "stream", False, 64, steps, steps, "circle", h, w, v_in[0], v_in[1], 1.013, v_out[0],
                            v_out[1], 0.987, 0.8)
    hd = plbm.create_handler(props)
    hd.start()
    hd.block_until_finished()
    o = oracle_mod.Oracle(alg, "stream", 64, "circle", w, h, inlet_velocity=v_in, inlet_density=1.013,
                          outlet_velocity=v_out, outlet_density=0.987, relaxation_time=0.8)
    o.run(steps)
    for i, got in enumerate((hd.get_densities(), hd.get_x_velocities(), hd.get_y_velocities(),
                             hd.get_absolute_velocities())):
        assert np.array_equal(got, o.result(i))
    hd.close()
