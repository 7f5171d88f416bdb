"""Arguments that the operator's entry points turn down before anything is launched: no pointer is read."""
import pytest

PLBM_ERR_ARGUMENT = -7


@pytest.mark.parametrize("n,h,w,y", [(0, 4, 4, 4096), (-1, 4, 4, 4096), (1, 0, 4, 4096), (1, 4, 0, 4096), (1, 4, 4, 4098),
                                     (1, 4, 4, 4100)])
def test_assembly_from_host_scalars(plbm, n, h, w, y):
    """As plbm_nn_assemble, an empty batch; and an output that 8-byte stores cannot reach."""
    import ctypes
    from portlbm_gb300 import warmstart as ws
    values = (ctypes.c_float * 3)()
    assert ws._fns().plbm_nn_assemble_host(4096, values, y, n, h, w, None) == PLBM_ERR_ARGUMENT
