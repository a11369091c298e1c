"""The mixed traversal's variants: each can be asked for, the automatic choice is a
value of its own, and it gives the general kernel's sums where the rule picks
another one."""
import ctypes as C

import numpy as np
import pytest

from openvort_gb300 import abi, gpu, workloads as W

pytestmark = pytest.mark.gpu


def _occupancy(ctx):
    """Resident blocks of four warps an SM: another number for each register budget."""
    fn = gpu.load()["_Z19ov_traversal_blocksP6ov_ctxiiPi"]
    fn.restype, fn.argtypes = C.c_int, [C.c_void_p, C.c_int, C.c_int, C.c_void_p]
    per_sm = C.c_int(0)
    fn(ctx.handle, abi.OV_PREC_MIXED, 4, C.byref(per_sm))
    return per_sm.value


@pytest.mark.parametrize("loops,picked", [(448, 1), (1100, 4)])   # few long items; enough items for 32 warps an SM
def test_general_kernel_can_be_asked_for(loops, picked):
    ht = W.random_walk_tangle(loops, 256, D=0.15, seed=8)
    ctx = gpu.Context(0, params=W.config_params("rw"), precision=abi.OV_PREC_MIXED)
    assert ctx.get_tuning().high_occupancy == -1
    ctx.upload(ht)
    blocks, vels = {}, {}
    for ho in (-1, 0, picked):
        ctx.set_tuning(high_occupancy=ho)
        assert ctx.get_tuning().high_occupancy == ho
        blocks[ho] = _occupancy(ctx)
        ctx.update_tangle(0.0)
        vels[ho] = np.array(ctx.download(ht, abi.OV_F_VELS).vels)
    ctx.close()
    assert blocks[-1] == blocks[picked] != blocks[0]
    for ho in (-1, picked):
        np.testing.assert_array_equal(vels[ho], vels[0])


@pytest.mark.parametrize("value", [-2, 5])
def test_no_such_variant(value):
    ctx = gpu.Context(0, params=W.config_params("rw"), precision=abi.OV_PREC_MIXED)
    with pytest.raises(gpu.OVError):
        ctx.set_tuning(high_occupancy=value)
    ctx.close()
