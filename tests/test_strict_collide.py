"""The F64_STRICT collision on the integer pipe (csrc/plbm_strict.cuh): bit-identical to the plain
double sequence wherever it says its result counts, and the drop-in form identical to the oracle
where nodes leave its range and take the FP64 sequence."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def strict_binary(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("strict") / "strict_test")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "portlbm_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "strict_test.cpp"), "-o", out], check=True)
    return out


@pytest.mark.parametrize("kind,least", [("flow", 0.9), ("unit", 0.9), ("axis", 0.9), ("tiny", 0.99), ("rest", 1.0),
                                        ("short", 0.5), ("ties", 0.5), ("wild", 0.3)])
def test_fixed_point_collision_is_the_double_sequence(strict_binary, kind, least):
    r = subprocess.run([strict_binary, kind, "200000", "3"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    compared, total = (int(v) for v in r.stdout.replace("compared", "").split("of"))
    assert compared >= least * total


@pytest.mark.gpu
@pytest.mark.parametrize("alg,lay", [("nptl", "stream"), ("lptl", "collision"), ("npol", "bundle"), ("nsol", "collision"),
                                     ("nsol", "stream")])
@pytest.mark.parametrize("rho_in,tau", [(1.9, 0.9), (1.02, 0.51), (1.2, 3.0)])
def test_strict_form_mixes_both_paths(plbm, oracle_mod, alg, lay, rho_in, tau):
    """Strong inlet fronts (|f - feq| and the velocity beyond the fixed-point range near them) beside
    quiet regions: one run holds nodes of both paths."""
    w, h, steps = 75, 33, 120
    props = plbm.Properties(alg, lay, False, 64, steps, steps, "circle", h, w, 0.0, 0.0, rho_in, 0.0, 0.0, 1.0, tau)
    hd = plbm.create_handler(props)
    hd.start()
    hd.block_until_finished()
    o = oracle_mod.Oracle(alg, lay, 64, "circle", w, h, inlet_density=rho_in, relaxation_time=tau)
    o.run(steps)
    for i, got in enumerate((hd.get_densities(), hd.get_x_velocities(), hd.get_y_velocities(),
                             hd.get_absolute_velocities())):
        assert np.array_equal(got, o.result(i))
    hd.close()
