"""Porous domains between a quarter and a half of L2: nptl's plain steps by vectorised rows, its steps with results by
the scalar kernel, against lptl's scalar steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f16s", "bf16s", "f16c"])
@pytest.mark.parametrize("w,h", [(2003, 501), (1529, 971), (2497, 433), (509, 2311), (1201, 801), (1301, 907)])
def test_plain_and_result_steps(plbm, precision, w, h):
    mask = plbm.porous_disks(w, h, 5, 0.75)
    results = []
    for alg in ("nptl", "lptl"):
        props = plbm.Properties(alg, "stream", False, 1024, 10 ** 6, 10 ** 6, "circle", h, w, 0.0, 0.0, 1.03, 0.0, 0.0, 1.0, 0.6)
        hd = plbm.create_handler(props, precision=precision, mask=mask)
        got = []
        for n in (1, 9, 4, 2):
            hd.run_steps(n)
            hd.sync_results()
            got += [hd.get_densities(), hd.get_x_velocities(), hd.get_y_velocities(), hd.get_absolute_velocities()]
        results.append(got)
        hd.close()
    for a, b in zip(*results):
        assert np.array_equal(a, b)
