"""Which handlers step two a launch: large domains, small ones and porous records, but not those whose single steps are
as good (narrow rows, open records a little beyond half of L2); and that the values there are the single steps'."""
import numpy as np
import pytest

from test_two_steps import CASES, SMALL, fields, handler

pytestmark = pytest.mark.gpu

# domain, geometry and layout that step singly, beside the nearest that step two a launch
RULES = [("f32", 31, 37501, "nptl", "stream", False, False), ("f32", 33, 18751, "nptl", "stream", False, True),
         ("f32", 32, 37501, "lptl", "bundle", False, False), ("f32", 32, 37501, "nptl", "bundle", True, True),
         ("f32", 31, 37501, "nptl", "collision", False, True), ("f16s", 31, 64001, "lptl", "bundle", False, True),
         ("bf16s", 31, 64001, "lptl", "stream", False, False), ("bf16s", 31, 64001, "nptl", "stream", False, True),
         ("bf16s", 32, 64001, "nptl", "collision", False, False), ("bf16s", 31, 64001, "nptl", "collision", False, True),
         ("f16c", 61, 34376, "lptl", "stream", False, False), ("f16c", 155, 13001, "lptl", "stream", False, True),
         ("f16c", 61, 34376, "nptl", "stream", False, True), ("f16c", 91, 62501, "nptl", "bundle", False, True),
         ("f32", 1301, 901, "nptl", "collision", False, False), ("f32", 1301, 901, "lptl", "collision", False, True),
         ("f32", 1301, 901, "nptl", "collision", True, True), ("f32", 1601, 1101, "nptl", "collision", False, True),
         ("f16c", 1601, 1201, "nptl", "collision", False, False), ("f16s", 1601, 1201, "nptl", "collision", False, True),
         ("f16c", 129, 1501, "lptl", "collision", True, True), ("f16c", 127, 1501, "lptl", "collision", True, False),
         ("f64_q60", 250, 31251, "nptl", "stream", False, False), ("f64_q60", 200, 35715, "nptl", "stream", False, True),
         ("f64_q60", 250, 31251, "lptl", "collision", False, True)]


@pytest.mark.parametrize("precision,w,h,alg,lay,porous,two", RULES)
def test_rules(plbm, precision, w, h, alg, lay, porous, two):
    many, single = (handler(plbm, alg, lay, precision, w, h, porous) for _ in range(2))
    assert many.run_launches(18) == (10 if two else 18)
    for n in (6, 9):
        many.run_steps(n)
        for _ in range(n):
            single.run_steps(1)
        for a, b in zip(fields(many), fields(single)):
            assert np.array_equal(a, b), n
    many.close()
    single.close()


@pytest.mark.parametrize("precision,w,h", CASES)
@pytest.mark.parametrize("alg,lay,porous", [("nptl", "stream", True), ("lptl", "bundle", False), ("nptl", "collision", True)])
def test_the_cases_of_two_step_launches_take_them(plbm, precision, w, h, alg, lay, porous):
    """test_two_steps.py compares handlers at these sizes with single steps: that they do step two a launch."""
    hd = handler(plbm, alg, lay, precision, w, h, porous)
    records = lay == "collision" and hd.gather_form() == "porous"
    two = (w, h) in SMALL[:-1] or w * h > 1.5e6 and (w, precision) != (31, "f32") or records
    if precision != "f64_q60":
        assert hd.run_launches(18) == (10 if two else 18)
    else:
        assert hd.run_launches(18) == 10
    hd.close()
