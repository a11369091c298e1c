"""Uploads and downloads through the caller's arrays in place (a device that
reads and writes pageable host memory through the host's page tables)
against the staged copies: the same device state and the same host arrays,
bit for bit, for whole-tangle and per-field transfers, in a single context
and in a context whose capacity exceeds the tangle (EMPTY slots past N)."""
from __future__ import annotations

import numpy as np
import pytest

from openvort_gb300 import abi, gpu, workloads as W

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vels", "vs", "tangents", "normals", "conn", "stat")


def _run(direct: bool):
    ht = W.random_walk_tangle(16, 64, D=0.1, seed=5)
    ctx = gpu.Context(0, params=W.config_params("rw"))
    ctx.set_host_access(direct)
    ctx.upload(ht)
    ctx.update_tangle(0.0)
    ctx.download(ht)
    first = {k: np.array(getattr(ht, k)) for k in FIELDS}
    # positions and topology only, then velocities only
    ht.pos[:] = ht.pos + 1e-6
    ctx.upload_fields(ht, abi.OV_F_POS | abi.OV_F_TOPOLOGY)
    ctx.update_tangle(0.0)
    ctx.download(ht, abi.OV_F_VELS)
    second = {k: np.array(getattr(ht, k)) for k in FIELDS}
    in_place = ctx.host_access_direct
    ctx.close()
    return first, second, in_place


def test_in_place_transfers_equal_staged_copies():
    staged = _run(False)
    direct = _run(True)
    assert not staged[2]
    for a, b in zip(staged[:2], direct[:2]):
        for k in FIELDS:
            assert np.array_equal(a[k], b[k]), k
    assert np.all(np.isfinite(direct[1]["vels"])) and np.abs(direct[1]["vels"]).max() > 0


def test_download_into_a_larger_host_tangle():
    """Host slots past the device's N become EMPTY with zero vectors on both paths."""
    outs = []
    for direct in (False, True):
        ht = W.random_walk_tangle(8, 64, D=0.1, seed=9)
        ctx = gpu.Context(0, params=W.config_params("rw"))
        ctx.set_host_access(direct)
        ctx.upload(ht)
        ctx.update_tangle(0.0)
        big = W.HostTangle(np.vstack([ht.pos, np.ones((7, 3))]), np.append(ht.conn[:, 0], [-1] * 7),
                           np.append(ht.conn[:, 1], [-1] * 7), ht.box_lo, ht.box_hi)
        big.vels[:] = 5.0
        ctx.download(big, abi.OV_F_VELS | abi.OV_F_TOPOLOGY)
        ctx.close()
        outs.append((np.array(big.vels), np.array(big.conn), np.array(big.stat)))
        assert np.all(big.vels[ht.n:] == 0) and np.all(big.stat[ht.n:, 0] == abi.OV_EMPTY)
    for a, b in zip(*outs):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n", [3, 255, 256, 257, 769])
@pytest.mark.parametrize("direct", [False, True])
def test_round_trip_at_block_edges(n, direct):
    """What is uploaded is what is downloaded, for the last slots of a block too;
    the slots behind the tangle's are left alone."""
    ht = W.random_walk_tangle(1, n, D=0.1, seed=6)
    rng = np.random.default_rng(n)
    for k in FIELDS[1:5]:
        getattr(ht, k)[:] = rng.standard_normal((n, 3))
    want = {k: np.array(getattr(ht, k)) for k in FIELDS}
    ctx = gpu.Context(0, params=W.config_params("rw"))
    ctx.set_host_access(direct)
    ctx.upload(ht)
    for k in FIELDS[:5]:
        getattr(ht, k)[:] = 0
    ctx.download(ht)
    ctx.close()
    for k in FIELDS:
        np.testing.assert_array_equal(getattr(ht, k), want[k], err_msg=k)


def test_ensemble_upload_in_place_equals_staged():
    """Members of different sizes, with headroom: positions, links and status of each
    member and the velocities of an evaluation, on both paths."""
    outs = []
    for direct in (False, True):
        members = [W.random_walk_tangle(m, 50 + m, D=0.1, seed=m) for m in (1, 6, 3)]
        ctx = gpu.Context(0, params=W.config_params("rw"))
        ctx.set_host_access(direct)
        ctx.upload_ensemble(members, [W.config_params("rw") for _ in members], 1.5)
        ctx.update_tangle(0.0)
        got = []
        for i, m in enumerate(members):
            want = np.array(m.pos), np.array(m.conn)
            m.pos[:] = 0
            h = ctx.download_member(i)
            np.testing.assert_array_equal(h.pos[:len(want[0])], want[0])
            np.testing.assert_array_equal(h.conn[:len(want[1])], want[1])
            assert np.all(h.stat[len(want[0]):, 0] == abi.OV_EMPTY)
            got.append(np.array(h.vels))
        ctx.close()
        outs.append(got)
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
