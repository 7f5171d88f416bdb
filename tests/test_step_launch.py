"""Launch shapes of the step kernels: blocks shrink on small domains until every SM has several, and
steps are chained by programmatic dependent launches.  The drop-in form stays identical to the oracle
at the edges of that rule, with result steps and residuals between the steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alg,lay", [("nptl", "stream"), ("nptl", "collision"), ("lptl", "bundle"), ("npol", "stream"),
                                     ("nsol", "stream"), ("nsol", "collision")])
@pytest.mark.parametrize("w,h,wg", [(2, 2, 64), (33, 3, 1024), (129, 17, 256), (310, 257, 1024), (97, 130, 100)])
def test_small_domains_match_the_oracle(plbm, oracle_mod, alg, lay, w, h, wg):
    if alg == "nsol" and wg == 100:
        pytest.skip("nsol refuses this work-group size")
    props = plbm.Properties(alg, lay, False, wg, 10 ** 6, 10 ** 6, "Hagen-Poiseuille", h, w, 0.0, 0.0, 1.05, 0.0, 0.0,
                            1.0, 0.7)
    hd = plbm.create_handler(props)
    o = oracle_mod.Oracle(alg, lay, wg, "Hagen-Poiseuille", w, h, inlet_density=1.05, relaxation_time=0.7)
    for steps in (1, 2, 37, 64):
        hd.run_steps(steps)
        hd.mass_momentum()
        hd.sync_results()
        o.run(steps)
        for i, got in enumerate((hd.get_densities(), hd.get_x_velocities(), hd.get_y_velocities())):
            assert np.array_equal(got, o.result(i)), (steps, i)
    hd.close()
