"""The drop-in form at boundary states that take its nodes out of the integer-pipe collision's range, where the
steps run on the FP64 pipe alone, and at the edges of that rule: bit-identical to the oracle."""
import ctypes

import numpy as np
import pytest

# inlet density, outlet density, inlet velocity, relaxation time
STATES = [(2.5, 2.45, 0.0, 0.9), (0.3, 0.3, 0.0, 0.9), (1.0, 1.0, 0.2, 0.8), (1.0, 0.5, 0.0, 0.9),          # FP64 alone
          (1.5, 1.01, 0.0, 0.9), (1.4, 1.4, 0.0, 0.9), (0.45, 0.45, 0.0, 0.9), (1.0, 1.0, 0.17, 0.8)]        # both


@pytest.mark.gpu
@pytest.mark.parametrize("alg,lay", [(a, l) for a in ("nptl", "lptl", "npol", "nsol") for l in ("stream", "collision", "bundle")])
@pytest.mark.parametrize("rho_in,rho_out,v,tau", STATES)
def test_strict_form_is_the_oracle(plbm, oracle_mod, alg, lay, rho_in, rho_out, v, tau):
    w, h, steps = 67, 35, 90
    props = plbm.Properties(alg, lay, False, 64, steps, steps, "circle", h, w, v, 0.0, rho_in, 0.0, 0.0, rho_out, tau)
    hd = plbm.create_handler(props)
    hd.start()
    hd.block_until_finished()
    o = oracle_mod.Oracle(alg, lay, 64, "circle", w, h, inlet_velocity=(v, 0.0), inlet_density=rho_in,
                          outlet_density=rho_out, relaxation_time=tau)
    o.run(steps)
    for i, got in enumerate((hd.get_densities(), hd.get_x_velocities(), hd.get_y_velocities(),
                             hd.get_absolute_velocities())):
        assert np.array_equal(got, o.result(i))
    hd.close()


@pytest.mark.gpu
def test_entry_without_allocations(plbm):
    """Its first call loads both kernels: a later call whose boundaries take the other one allocates nothing."""
    import torch

    import test_zz_no_alloc as z
    w, h = 70, 40
    mask = z._mask(w, h)
    lib = z._lib(plbm)
    lat0, lat1, flags, res = z._buffers(mask, w, h)
    free = None
    for rho_in, rho_out in ((1.05, 1.0), (2.05, 2.0), (1.05, 1.0), (0.3, 0.3)):
        args = z.NoallocArgs(lat0.data_ptr(), lat1.data_ptr(), flags.data_ptr(), res.data_ptr(), w, h, 0.8, rho_in, 0.0, 0.0,
                             rho_out, 0.0, 0.0, 0, 60, 1, None)
        assert lib.plbm_nptl_steps_noalloc(ctypes.byref(args)) == 0, lib.plbm_noalloc_last_error()
        torch.cuda.synchronize()
        now = torch.cuda.mem_get_info()[0]
        assert free in (None, now)
        free = now
        got = res.cpu().numpy().reshape(4, -1)
        props = plbm.Properties("nptl", "stream", False, 64, 60, 60, "circle", h, w, 0.0, 0.0, rho_in, 0.0, 0.0, rho_out, 0.8)
        hd = plbm.create_handler(props, mask=mask)
        hd.run_steps(60)
        hd.sync_results()
        for i, want in enumerate((hd.get_densities(), hd.get_x_velocities(), hd.get_y_velocities(),
                                  hd.get_absolute_velocities())):
            assert np.array_equal(got[i], want)
        hd.close()
        free = torch.cuda.mem_get_info()[0]
