"""More candidate pairs than an int counts (every node within rec_dist of every
other one): the reconnection is refused, and the context goes on."""
import pytest

from openvort_gb300 import gpu, workloads as W

pytestmark = pytest.mark.gpu

OV_ERR_ARG = 1


def test_two_billion_pairs_are_refused():
    ht = W.random_walk_tangle(257, 257, D=0.1, seed=1)   # 66,049 nodes: 2.18e9 pairs
    ctx = gpu.Context(0, params=W.config_params("rw", rec_dist=1.0))
    ctx.upload(ht)
    ctx.update_tangle(0.0)
    with pytest.raises(gpu.OVError) as e:
        ctx.reconnect(0.0)
    assert e.value.code == OV_ERR_ARG and "2181202176 pairs" in str(e.value)
    ctx.set_params(W.config_params("rw"))
    ctx.reconnect(0.0)
    ctx.update_tangle(0.0)
    ctx.close()
