"""Two-step launches of nptl and lptl (csrc/plbm_pair.cuh, domains whose lattices exceed L2 and small ones) against
single steps of the same handler: the same values, whatever the domain's remainders of a strip's
columns and rows, the number of steps, the gather and the layout."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def handler(plbm, alg, lay, precision, w, h, porous, rho_in=1.03):
    props = plbm.Properties(alg, lay, False, 1024, 10 ** 6, 10 ** 6, "circle", h, w, 0.0, 0.0, rho_in, 0.0, 0.0, 1.0, 0.6)
    mask = None
    if porous:   # disks need room; small domains take single solid nodes
        small = min(w, h) < 64
        mask = (np.random.default_rng(w * h).random((h, w)) < 0.2).astype(np.int8) if small else plbm.porous_disks(w, h, 5, 0.75)
    return plbm.create_handler(props, precision=precision, mask=mask)


def fields(hd):
    hd.sync_results()
    return [hd.get_densities(), hd.get_x_velocities(), hd.get_y_velocities(), hd.get_absolute_velocities()]


# two-step launches are taken from 0.5 (shifted forms) and 8 (f64_q60) times L2's 129 MB of lattices on, and
# up to 65536 nodes (row pitch included) by the shifted forms
SIZES = {"f32": [(1603, 1153), (31, 60001), (60, 30011), (2501, 1801)],
         "f16s": [(2401, 1511), (61, 60007), (2130, 2011)], "bf16s": [(2401, 1511)], "f16c": [(2431, 1517)],
         "f64_q60": [(3031, 2507), (4111, 4093)]}
SMALL = [(2, 2), (2, 9), (3, 5), (4, 3), (29, 4), (30, 31), (31, 7), (32, 64), (33, 20), (61, 100), (62, 30), (512, 128),
         (1003, 63), (513, 128)]
MIDDLE = [(353, 257), (1003, 401)]       # two steps a launch in porous records, single steps elsewhere
for form in ("f32", "f16s", "bf16s", "f16c"):
    SIZES[form] += MIDDLE
SIZES["f32"] += SMALL
SIZES["f16s"] += SMALL
SIZES["bf16s"] += SMALL[2::4]
SIZES["f16c"] += SMALL[3::4]
CASES = [(p, w, h) for p, sizes in SIZES.items() for w, h in sizes]


@pytest.mark.parametrize("precision,w,h", CASES)
@pytest.mark.parametrize("alg,lay,porous", [("nptl", "stream", True), ("lptl", "bundle", False), ("nptl", "collision", True)])
def test_two_step_launches_are_single_steps(plbm, precision, w, h, alg, lay, porous):
    many, single = (handler(plbm, alg, lay, precision, w, h, porous) for _ in range(2))
    for n in (5, 4, 18, 3, 9):
        many.run_steps(n)                       # n - 1 plain steps, four at a time, then a result step
        for _ in range(n):
            single.run_steps(1)                 # a result step: always a launch of its own
        for a, b in zip(fields(many), fields(single)):
            assert np.array_equal(a, b), n
    many.close()
    single.close()


@pytest.mark.parametrize("precision", ["f16s", "bf16s", "f16c"])
def test_vectorised_rows_of_large_domains(plbm, precision):
    """nptl steps vectorised rows in the stream layout there, lptl the scalar kernel."""
    a, b = (handler(plbm, alg, "stream", precision, 2411, 1519, porous) for alg, porous in (("nptl", True), ("lptl", True)))
    for _ in range(6):
        a.run_steps(1)
        b.run_steps(1)
    for x, y in zip(fields(a), fields(b)):
        assert np.array_equal(x, y)
    a.close()
    b.close()


def test_frames_and_precision_change(plbm):
    """A run with frames (graphs of two-step launches and a result step) and a change of storage form
    keep to the single steps' values."""
    w, h = 2401, 1511
    props = plbm.Properties("nptl", "stream", False, 1024, 43, 10, "circle", h, w, 0.0, 0.0, 1.03, 0.0, 0.0, 1.0, 0.6)
    a, b = plbm.create_handler(props, precision="f16s"), handler(plbm, "nptl", "stream", "f16s", w, h, False)
    a.start()
    a.block_until_finished()
    for _ in range(43):
        b.run_steps(1)
    b.sync_results()
    assert np.array_equal(a.get_x_velocities(), b.get_x_velocities())
    for hd in (a, b):
        hd.set_precision("f32")
    a.run_steps(14)
    for _ in range(14):
        b.run_steps(1)
    for x, y in zip(fields(a), fields(b)):
        assert np.array_equal(x, y)
    a.close()
    b.close()


@pytest.mark.parametrize("precision,w,h,pairs", [("f16s", 2401, 1511, True), ("f64_q60", 3031, 2507, True),
                                                 ("f64_q60", 400, 100, False), ("f64_strict", 400, 100, False),
                                                 ("f32", 400, 100, True), ("f32", 512, 129, False)])
def test_launch_accounting(plbm, precision, w, h, pairs):
    """run_launches follows the schedule: an odd first step, four plain steps in two launches, the rest
    and the result step one by one."""
    hd = handler(plbm, "nptl", "stream", precision, w, h, False)
    for n, want in ((1, 1), (4, 4), (5, 3), (8, 6), (9, 5), (70, 36)):
        assert hd.run_launches(n) == (want if pairs else n), n
    hd.run_steps(1)
    for n, want in ((8, 6), (9, 7), (10, 6)):
        assert hd.run_launches(n) == (want if pairs else n), n
    assert hd.run_launches(0) == 0
    hd.close()
