"""Batches advance plain steps two a launch (k_batch_two_steps): identical to single steps of the same
batch, for domains at the edges of a strip's columns, in every storage form, for odd and even runs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(2, 3), (30, 17), (31, 40), (59, 5), (61, 64), (64, 33), (200, 90), (121, 7)]


def batch(plbm, precision, copies):
    doms = []
    for c in range(copies):
        for i, (w, h) in enumerate(SIZES):
            mask = plbm.porous_disks(w, h, 7 * i + c, 0.8, 1.0, 3.0) if w > 8 and h > 8 else np.zeros((h, w), np.int8)
            doms.append({"mask": mask, "relaxation_time": 0.6 + 0.04 * i, "inlet_density": 1.01 + 0.004 * i,
                         "outlet_density": 1.0})
    return plbm.Batch(doms, precision=precision)


# 3, 12 and 90 copies: pieces of one, two and four rows
@pytest.mark.parametrize("precision,copies", [("f32", 3), ("f32", 12), ("f32", 90), ("f16s", 3), ("bf16s", 12),
                                              ("f16c", 3), ("f64_q60", 12)])
@pytest.mark.parametrize("mode", ["persistent", "persistent_graph"])
def test_batch_two_step_launches_are_single_steps(plbm, precision, copies, mode):
    many, single = batch(plbm, precision, copies), batch(plbm, precision, copies)
    for n in (5, 2, 39, 20):
        many.run(n, mode=mode)
        for _ in range(n):
            single.run(1, mode="persistent")     # a result step: a launch of its own
        for i in list(range(len(SIZES))) + [copies * len(SIZES) - 1]:
            for which in range(4):
                assert np.array_equal(many.result(i, which), single.result(i, which)), (n, i, which)
    many.close()
    single.close()
