"""The kernels that are issued, counted at the launch: run_launches' forecast, frames and batches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alg,lay,precision,w,h", [("nptl", "stream", "f16s", 2401, 1511), ("nptl", "stream", "f64_q60", 3031, 2507),
                                                   ("lptl", "bundle", "f32", 400, 100), ("nptl", "collision", "f64_strict", 400, 100),
                                                   ("npol", "stream", "f32", 100, 60), ("nsol", "stream", "f64_q60", 100, 60)])
@pytest.mark.parametrize("graph", [True, False])
def test_the_forecast_is_what_is_issued(plbm, alg, lay, precision, w, h, graph):
    props = plbm.Properties(alg, lay, False, 1024, 10 ** 6, 10 ** 6, "circle", h, w, 0.0, 0.0, 1.03, 0.0, 0.0, 1.0, 0.6)
    hd = plbm.create_handler(props, precision=precision, use_graph=graph)
    assert hd.launches() == 0
    for n in (1, 70, 9, 8, 4, 5, 130, 7, 2, 200):
        before, want = hd.launches(), hd.run_launches(n)
        hd.run_steps(n)
        assert hd.launches() - before == want, n
    hd.close()


@pytest.mark.parametrize("frame,steps,want", [(10, 40, 4 * 6), (9, 45, 5 * 5), (7, 21, 3 * 5)])
def test_frames(plbm, frame, steps, want):
    """Of a frame's steps the last writes results; the others go four to two launches, the rest one by one."""
    props = plbm.Properties("nptl", "stream", False, 1024, steps, frame, "circle", 100, 400, 0.0, 0.0, 1.03, 0.0, 0.0, 1.0, 0.6)
    hd = plbm.create_handler(props, precision="f32")
    hd.start()
    hd.block_until_finished()
    assert hd.launches() == want
    hd.close()


def test_batch(plbm):
    doms = [{"mask": np.zeros((40, 50 + i), np.int8), "relaxation_time": 0.7, "inlet_density": 1.02} for i in range(3)]
    b = plbm.Batch(doms, precision="f32")
    b.run(22, mode="persistent_graph")    # a graph of 16 (8 launches), 5 plain (3), one with results
    assert b.launches() == 12
    b.run(9, mode="persistent")           # 8 plain steps in 4
    assert b.launches() == 17
    b.run(5, mode="per_domain")
    assert b.launches() == 17 + 15
    b.close()


@pytest.mark.parametrize("precision,vec,w,h,copies,two", [
    ("f16s", True, 62, 900, 20, True), ("f16s", True, 62, 1700, 20, False), ("f16s", False, 62, 1700, 20, True),
    ("f16s", True, 95, 1700, 20, True), ("f16s", True, 95, 3000, 60, False), ("f16c", True, 128, 2300, 60, True),
    ("f64_q60", False, 64, 1700, 20, False), ("f64_q60", False, 95, 1700, 20, True), ("f32", False, 62, 1700, 20, True)])
def test_batches_of_narrow_domains(plbm, precision, vec, w, h, copies, two):
    """Strips many more than warps: single steps where those are as good; the values are the same."""
    m = (np.random.default_rng(w).random((h, w)) < 0.1).astype(np.int8)
    doms = [{"mask": m, "relaxation_time": 0.7, "inlet_density": 1.02}] * copies
    many, single = (plbm.Batch(doms, precision=precision) for _ in range(2))
    for b in (many, single):
        b.set_tile(32, 4 + 256 * 2 + (plbm.BATCH_TILE_VEC if vec else 0), 4)
    many.run(9, mode="persistent")
    assert many.launches() == (5 if two else 9)
    many.run(18, mode="persistent_graph")
    assert many.launches() == (5 + 10 if two else 27)    # an odd first step, 16 in 8 launches, one with results
    for _ in range(27):
        single.run(1)
    for i in (0, copies - 1):
        for which in range(3):
            assert np.array_equal(many.result(i, which), single.result(i, which))
    many.close()
    single.close()


@pytest.mark.parametrize("precision,candidates", [("f32", 21), ("f16s", 42)])
def test_autotune_times_single_steps(plbm, precision, candidates):
    """The tile it chooses shapes steps with results and left-over ones, not two-step launches."""
    doms = [{"mask": np.zeros((40, 50), np.int8), "relaxation_time": 0.7, "inlet_density": 1.02}]
    b = plbm.Batch(doms, precision=precision)
    b.autotune(9)
    assert b.launches() == candidates * 9
    b.run(9, mode="persistent")
    assert b.launches() == candidates * 9 + 5
    b.close()
