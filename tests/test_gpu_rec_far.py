"""The candidates' direct sums by the far-segment series (k_rec_far): within
their own error bound of the FP64 sums for every grid of image shifts, at the
edges of candidate pairs, chunks and members, and with segments on both sides
of the distance from which the series holds."""
import numpy as np
import pytest

from openvort_gb300 import abi, gpu, workloads as W

pytestmark = pytest.mark.gpu


def _check(ctx, nodes):
    sm, bm, mm = ctx.direct_sums_bounded(nodes, abi.OV_PREC_MIXED)
    sf, bf, _ = ctx.direct_sums_bounded(nodes, abi.OV_PREC_FP64)
    err = np.abs(sm - sf).max(axis=1)
    assert (err <= bm + bf).all()
    # the bound itself: 97 eps32 of the terms' magnitudes (1.03 for what bounds those)
    assert (bm <= 1.1 * 97 * 2.0 ** -24 * mm + 4 * 2.0 ** -24 * np.abs(sm).sum(axis=1) + 1e-11 * mm).all()


@pytest.mark.parametrize("loops,per_loop,D,images,count", [
    (1, 9, 0.1, 26, 9),         # fewer segments than threads, odd candidate count
    (3, 100, 0.1, 18, 1),       # one candidate: a pair of itself
    (40, 256, 0.1, 6, 37),      # two chunks
    (33, 250, 0.05, 26, 64),    # dense: many near segments
    (20, 64, 0.1, 0, 11),       # no images
    (4, 64, 0.01, 26, 33),      # a box as small as the near sphere: no segment is far
])
def test_sums_within_bound(loops, per_loop, D, images, count):
    ht = W.random_walk_tangle(loops, per_loop, D=D, seed=loops + images, n_images=images)
    ctx = gpu.Context(0, params=W.config_params("rw"), precision=abi.OV_PREC_MIXED)
    ctx.upload(ht)
    _check(ctx, np.linspace(0, ht.n - 1, count).astype(np.int32))
    ctx.close()


def test_pairs_across_members():
    ms = [W.random_walk_tangle(n, 64, D=0.1, seed=50 + n) for n in (3, 1, 5)]
    ctx = gpu.Context(0, precision=abi.OV_PREC_MIXED)
    ctx.upload_ensemble(ms, [W.config_params("rw") for _ in ms], 1.0)
    starts = np.cumsum([0] + [m.n for m in ms])
    nodes = np.array([5, starts[1] - 1, starts[1], starts[2] - 1, starts[2] + 7, starts[3] - 1, 0], dtype=np.int32)
    _check(ctx, nodes)
    ctx.close()
