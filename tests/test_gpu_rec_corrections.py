"""The corrections of reconnection candidates after rewirings (k_corr_far for grids
of image shifts, k_corr for the other image sets): every candidate's sum over the
changed segments against extended precision, within its bound, with a full list
of 32 segments, and the bound itself."""
import ctypes as C

import numpy as np
import pytest

from openvort_gb300 import abi, gpu, workloads as W

pytestmark = pytest.mark.gpu

LD = np.longdouble if np.finfo(np.longdouble).nmant > 52 else np.float64
EPS32 = 2.0 ** -24


def _query(ht, box, j, p):
    """Image j's query points of p (j = -1: the nodes themselves), as the reference forms them."""
    if j < 0:
        return p
    shift, faces = box["images"][j]
    q = p - box["L"] * np.array(shift, LD)
    for face in faces:
        w = (box["hi"] if face & 1 else box["lo"])[face // 2]
        q[:, face // 2] = 2 * w - p[:, face // 2]
    return q


def _contributions(ht, cand, m, f, sign, kappa):
    """sum over the segments m -> f of sign times their velocity at the candidates, and of its magnitude bound."""
    imgs, walls = abi.image_set(ht.image_set)
    box = dict(lo=np.asarray(ht.box_lo, LD), hi=np.asarray(ht.box_hi, LD), images=imgs)
    L = box["L"] = box["hi"] - box["lo"]
    per = np.array([walls[2 * a] == abi.OV_WALL_PERIODIC for a in range(3)])
    pos = ht.pos.astype(LD)
    a, b = pos[m], pos[f].copy()
    d = b - a
    b += np.where(per & (d < -L / 2), L, 0) - np.where(per & (d > L / 2), L, 0)
    out, mag = np.zeros((len(cand), 3), LD), np.zeros(len(cand), LD)
    for j in range(-1, len(imgs)):
        q = _query(ht, box, j, pos[cand].copy())
        R, P = a[None] - q[:, None], b[None] - q[:, None]
        lr, lp, dot = np.sqrt((R ** 2).sum(-1)), np.sqrt((P ** 2).sum(-1)), (R * P).sum(-1)
        keep = (lr >= 1e-8) & (lp >= 1e-8)
        if j < 0:   # a node's own segments
            keep &= ~((m[None] == cand[:, None]) | (f[None] == cand[:, None]))
        lr, lp = np.where(keep, lr, 1), np.where(keep, lp, 1)
        keep &= dot / lr / lp >= 1e-8
        sc = np.where(keep, LD(kappa) / 4 / LD(np.pi) * (lr + lp) / np.where(keep, lr * lp * (lr * lp + dot), 1), 0)
        out += (np.cross(R, P) * sc[..., None] * sign[None, :, None]).sum(1)
        mag += (np.sqrt(((b - a) ** 2).sum(-1))[None] * lr * sc).sum(1)
    return out.astype(np.float64), mag.astype(np.float64)


def _functions():
    L, ip, dp = gpu.load(), C.POINTER(C.c_int), C.POINTER(C.c_double)
    begin, correct, fetch = (L[n] for n in ("_Z12ov_rec_beginP6ov_ctxPKiiPd", "_Z14ov_rec_correctP6ov_ctxiiPKiS2_PKdiS2_i",
                                            "_Z12ov_rec_fetchP6ov_ctxiiPd"))
    begin.argtypes = [C.c_void_p, ip, C.c_int, dp]
    correct.argtypes = [C.c_void_p, C.c_int, C.c_int, ip, ip, dp, C.c_int, ip, C.c_int]
    fetch.argtypes = [C.c_void_p, C.c_int, C.c_int, dp]
    i, d = (lambda a: a.ctypes.data_as(ip)), (lambda a: a.ctypes.data_as(dp))
    return begin, correct, fetch, i, d


@pytest.mark.parametrize("images,grid", [("periodic_26", True), ("periodic_18", True), ("periodic_6", True),
                                         ("open", True), ("wall_2_4", False), ("wall_1_26", False)])
@pytest.mark.parametrize("D,changes", [(0.1, 32), (0.03, 5)])
def test_corrections_within_their_bound(images, grid, D, changes):
    begin, correct, fetch, i, d = _functions()
    base = W.random_walk_tangle(12, 64, D=D, seed=changes)
    ht = W.HostTangle(base.pos.copy(), base.conn[:, 0], base.conn[:, 1], base.box_lo, base.box_hi, image_set=images)
    p = W.config_params("rw")
    ctx = gpu.Context(0, params=p, precision=abi.OV_PREC_MIXED)
    ctx.upload(ht)
    cand = np.arange(0, ht.n, 3, dtype=np.int32)
    out = np.zeros((len(cand), 5))
    assert begin(ctx.handle, i(cand), len(cand), d(out)) == 0
    rng = np.random.default_rng(changes)
    wraps = np.flatnonzero((np.abs(ht.pos[ht.conn[:, 0]] - ht.pos) > D / 2).any(1))
    before = np.zeros((len(cand), 4))
    for _ in range(12):
        # some of the segments cross the box's boundary, some are candidates' own
        m = rng.integers(0, ht.n, changes).astype(np.int32)
        m[:2] = rng.choice(wraps, 2)
        m[2] = cand[rng.integers(len(cand))]
        f = ht.conn[m, 0].astype(np.int32)
        sign = np.where(np.arange(changes) % 2, 1.0, -1.0)
        assert correct(ctx.handle, 0, len(cand), i(m), i(f), d(sign), changes, i(cand), 0) == 0
        got = np.zeros((len(cand), 4))
        assert fetch(ctx.handle, 0, len(cand), d(got)) == 0
        want, mag = _contributions(ht, cand, m, f, sign, p.kappa)
        step, before = got - before, got
        # (differences of running FP64 sums)
        slack = 4 * 2.0 ** -53 * np.abs(got[:, :3]).max(axis=1)
        assert (np.abs(step[:, :3] - want).max(axis=1) <= step[:, 3] + slack).all()
        if not grid:   # in closed form: 64 eps32 of the terms' magnitudes, which add up in FP64
            assert (step[:, 3] <= 64 * 1.012 * EPS32 * mag + 2e-12 * mag + 1e-14 * np.abs(got[:, :3]).sum(axis=1)).all()
    ctx.close()


@pytest.mark.parametrize("images", ["periodic_26", "periodic_6", "open", "wall_2_4"])
def test_changed_segments_add_up_in_fp64(images):
    """A segment, another and the first one again with the other sign: what is left is the
    second one's contribution to FP64 rounding, though the terms are FP32 ones."""
    begin, correct, fetch, i, d = _functions()
    base = W.random_walk_tangle(6, 64, D=0.1, seed=9)
    ht = W.HostTangle(base.pos.copy(), base.conn[:, 0], base.conn[:, 1], base.box_lo, base.box_hi, image_set=images)
    ctx = gpu.Context(0, params=W.config_params("rw"), precision=abi.OV_PREC_MIXED)
    ctx.upload(ht)
    cand = np.arange(0, ht.n, 5, dtype=np.int32)
    assert begin(ctx.handle, i(cand), len(cand), d(np.zeros((len(cand), 5)))) == 0
    last = np.zeros((len(cand), 4))

    def added(changes):
        """The corrections' change by {position in the list: (segment, sign)}; empty positions between."""
        nonlocal last
        m, sign = np.full(max(changes) + 1, -1, np.int32), np.zeros(max(changes) + 1)
        for at, (seg, sg) in changes.items():
            m[at], sign[at] = seg, sg
        f = np.where(m >= 0, ht.conn[m, 0], -1).astype(np.int32)
        assert correct(ctx.handle, 0, len(cand), i(m), i(f), d(sign), len(m), i(cand), 0) == 0
        got = np.zeros((len(cand), 4))
        assert fetch(ctx.handle, 0, len(cand), d(got)) == 0
        step, last = got - last, got
        return step[:, :3]

    for one, two in ((3, 200), (130, 77), (301, 9)):
        first, second = added({0: (one, 1.0)}), added({0: (two, 1.0)})
        both = added({0: (one, 1.0), 16: (two, 1.0), 1: (one, -1.0)})
        # three additions of the terms, and those of the running sums
        scale = np.abs(first) + np.abs(second) + np.abs(last[:, :3])
        assert (np.abs(both - second) <= 16 * 2.0 ** -53 * scale).all()
    ctx.close()
