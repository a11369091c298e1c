"""Parts of the split walk at both sides of every line of their number (16, 8, 4,
2 parts and whole walks), and a grid that
has a warp for each of them."""
import ctypes as C

import numpy as np
import pytest

from openvort_gb300 import abi, gpu, workloads as W
from tests._util import node_rel_err

pytestmark = pytest.mark.gpu

SMS = 152


def _nodes(line):
    """Nodes, a multiple of 32, whose (tile, 27 query points) items an SM times the root of the
    nodes come closest below a line."""
    return int((line * SMS * 32 / 27) ** (2 / 3)) // 32 * 32


@pytest.mark.parametrize("n", [_nodes(k) + d for k in (1000, 6900, 27500, 54000) for d in (0, 32)])
def test_same_walk_on_both_sides_of_a_line(n):
    base = W.random_walk_tangle(n // 32, 32, D=0.1, seed=n)
    got = []
    for walk in (abi.OV_WALK_FP64, abi.OV_WALK_SPLIT):
        ht = W.HostTangle(base.pos.copy(), base.conn[:, 0], base.conn[:, 1], base.box_lo, base.box_hi)
        ctx = gpu.Context(0, params=W.config_params("rw"))
        ctx.set_walk(walk)
        ctx.upload(ht)
        ctx.update_tangle(0.0)
        ctx.download(ht)
        st = ctx.stats()
        ctx.close()
        got.append((np.array(ht.vels), [st[k] for k in ("visits", "accepts", "error_word")]))
    assert got[0][1] == got[1][1] and got[0][1][2] == 0
    assert node_rel_err(got[1][0], got[0][0]) < 1e-10   # the FP64 parity tolerance


@pytest.mark.parametrize("n,parts", [(62, 16), (496, 16), (4096, 8)])
def test_grid_has_a_warp_for_each_part(n, parts):
    """Blocks of four warps: one for every four of tiles * 27 * parts, up to four an SM."""
    blocks = gpu.load()["_Z19ov_traversal_blocksP6ov_ctxiiPi"]
    ht = W.random_walk_tangle(2, n // 2, D=0.1, seed=1)
    ctx = gpu.Context(0, params=W.config_params("rw"))
    ctx.upload(ht)
    blocks.restype = C.c_int
    blocks.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_void_p]
    per_sm = C.c_int(0)
    got = blocks(ctx.handle, abi.OV_PREC_FP64, 4, C.byref(per_sm))
    ctx.close()
    items = (n + 31) // 32 * 27 * parts
    assert got >= min(items // 4, per_sm.value * SMS)
