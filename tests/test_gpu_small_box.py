"""Boxes so small that separations the integer law takes by the box's measure
come under the reference's filters (|R|, |R+S| < 1e-8, octree.c:311,330)."""
import numpy as np
import pytest

from openvort_gb300 import abi, gpu, workloads as W

pytestmark = pytest.mark.gpu


def _tangle(D):
    return W.random_walk_tangle(4, 64, D=D, delta=0.01 * D, seed=2)


@pytest.mark.parametrize("D", [2e-7, 1e-6, 5e-6, 2.5e-5])
@pytest.mark.parametrize("prec", [abi.OV_PREC_FP64, abi.OV_PREC_DD])
def test_split_walk_keeps_the_filters(D, prec):
    got = []
    for precision, walk in ((abi.OV_PREC_FP64, abi.OV_WALK_FP64), (prec, abi.OV_WALK_SPLIT)):
        ht = _tangle(D)
        ctx = gpu.Context(0, params=W.config_params("rw"), precision=precision)
        ctx.set_walk(walk)
        ctx.upload(ht)
        ctx.update_tangle(0.0)
        ctx.download(ht)
        st = ctx.stats()
        ctx.close()
        got.append((ht.vs.copy(), st))
    (v64, s64), (v, s) = got
    assert s["visits"] == s64["visits"] and s["accepts"] == s64["accepts"]
    # FP64 parity, as between the walks of larger boxes
    per_node = np.linalg.norm(v - v64, axis=1) / np.linalg.norm(v64, axis=1)
    assert per_node.max() < 1e-10


@pytest.mark.parametrize("D", [1e-6, 2.5e-5])
def test_direct_sums_keep_the_filters(D):
    torch = pytest.importorskip("torch")
    from tests._util import node_rel_err
    from tests.test_zz_no_alloc import _Caller, _reference
    ht = _tangle(D)
    p = W.config_params("rw")
    ids = np.arange(0, ht.n, 5, dtype=np.int32)
    (ref,) = _reference(ht, p, [ids])
    got = _Caller(torch, ht, p).call(ids)
    assert node_rel_err(got[0], ref[0]) < 1e-10
    assert node_rel_err(got[1], ref[1]) < 1e-10
