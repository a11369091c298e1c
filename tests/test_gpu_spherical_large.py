"""The spherical section's split walk in whole walks (S = 1, above 768 (tile, query
point) items an SM) and in parts, on both sides of that line, against the all-FP64
walk: the same cells visited and accepted, the same velocities."""
import numpy as np
import pytest

from openvort_gb300 import abi, gpu, workloads as W

pytestmark = pytest.mark.gpu

NODES = 769 * 152 // 18 * 32   # the smallest with 769 items an SM, to a tile


@pytest.mark.parametrize("rings", [NODES // 25 - 40, NODES // 25 + 60])   # 25 nodes a ring
def test_split_walk_equals_fp64_walk(rings):
    p = gpu.sph_params_default()
    got = []
    for walk in (abi.OV_WALK_FP64, abi.OV_WALK_SPLIT):
        t = W.spherical_tangle(rings, seed=5, line=False, empty=2)
        ctx = gpu.Context(0)
        ctx.set_walk(walk)
        ctx.sph_update(t, p, 0.0)
        st = ctx.stats()
        ctx.close()
        got.append((np.array(t.vels[:-2]), [st[k] for k in ("visits", "accepts")], st["error_word"]))
    assert got[0][1] == got[1][1] and got[0][2] == got[1][2]
    # the FP64 parity tolerance of the other spherical tests
    err = np.linalg.norm(got[1][0] - got[0][0], axis=1) / np.linalg.norm(got[0][0], axis=1)
    assert err.max() < 1e-10
