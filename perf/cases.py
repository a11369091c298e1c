"""Performance cases of the velocity and time-step path.

Every case is one call (or one short run) as a host program makes it: the
tangle's arrays in host memory, uploaded into a context that the program
keeps, the path's entry points, and the results downloaded into host arrays
it keeps too.  The kinds:

  eval       update_tangle: tangents, normals and velocities of a tangle
  rk4        update_tangle + rk4_step: one RK4 step without topology passes
  step       the whole main-loop step (reconnection, remeshing, smoothing,
             RK4, periodic wrap) on one tangle
  ensemble   the same step on a batch of independent tangles, a few steps
             after the upload
  direct     the O(N) direct sums of a list of nodes, as the tree's error is
             measured against
  spherical  update_tangle of the spherical fork's section of a shell

`exact` evaluates the same Barnes-Hut sums, direct sums, finite differences
and RK4 combination in 64-bit torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from openvort_gb300 import abi, gpu, workloads as W

PREC = {"fp64": abi.OV_PREC_FP64, "mixed": abi.OV_PREC_MIXED, "dd": abi.OV_PREC_DD}
RESULTS = abi.OV_F_VELS | abi.OV_F_VS | abi.OV_F_TANGENTS | abi.OV_F_NORMALS


# ------------------------------------------------------------------- cases
def listed():
    return [
        # 8 rings, about 500 nodes: the smallest run people start from; one
        # evaluation through the drop-in's upload / compute / download
        dict(name="rings8_eval", kind="eval", tangle="rings", loops=8, per_loop=62, D=0.1, images="periodic_26",
             prec="fp64", theta=0.4),
        # the same run's whole time step: launches and host passes, not arithmetic
        dict(name="rings8_step", kind="step", tangle="rings", loops=8, per_loop=62, D=0.1, images="periodic_26",
             prec="fp64", theta=0.4, smooth=False, dt=5e-5),
        # a mid-size tangle of odd loop lengths, fewer images
        dict(name="walk4125_eval", kind="eval", tangle="walk", loops=33, per_loop=125, D=0.06, images="periodic_18",
             prec="fp64", theta=0.3),
        # the velocity evaluation that the benchmark quotes
        dict(name="walk65536_eval", kind="eval", tangle="walk", loops=256, per_loop=256, D=0.1, images="periodic_26",
             prec="fp64", theta=0.4),
        # the same tangle in double-single arithmetic
        dict(name="walk65536_dd", kind="eval", tangle="walk", loops=256, per_loop=256, D=0.1, images="periodic_26",
             prec="dd", theta=0.4),
        # mixed precision on a larger tangle at a tight opening angle
        dict(name="walk262144_mixed", kind="eval", tangle="walk", loops=1024, per_loop=256, D=0.1,
             images="periodic_26", prec="mixed", theta=0.3),
        # mirror walls: reflected query points and image sums
        dict(name="walls30009_eval", kind="eval", tangle="walk", loops=147, per_loop=204, D=0.1, images="wall_2_4",
             prec="fp64", theta=0.4),
        # one RK4 step of the benchmark's tangle in mixed precision
        dict(name="walk65536_rk4", kind="rk4", tangle="walk", loops=256, per_loop=256, D=0.1, images="periodic_26",
             prec="mixed", theta=0.4, dt=5e-5),
        # a batch of tangles of uneven size, two whole steps from the upload
        dict(name="ensemble12_step", kind="ensemble", members=12, min_nodes=2048, max_nodes=32768, per_loop=256,
             D=0.1, images="periodic_26", prec="mixed", theta=0.4, dt=5e-5, steps=2),
        # the largest single tangle: a whole step with smoothing
        dict(name="walk524288_step", kind="step", tangle="walk", loops=2048, per_loop=256, D=0.1587,
             images="periodic_26", prec="mixed", theta=0.4, smooth=True, dt=2e-5),
        # direct sums of a node subsample: how the tree's error is reported
        dict(name="direct2048_of_32768", kind="direct", tangle="walk", loops=128, per_loop=256, D=0.1,
             images="periodic_26", theta=0.4, nodes=2048),
        # the spherical fork's velocity path
        dict(name="spherical16000", kind="spherical", rings=640, prec="fp64", theta=0.4),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["eval", "eval", "eval", "rk4", "step", "ensemble", "direct", "spherical"])
    theta = round(rng.uniform(0.3, 0.5), 3)
    if kind == "spherical":
        return dict(kind=kind, rings=int(_log(rng, 12, 640)), prec=rng.choice(["fp64", "mixed"]), theta=theta)
    if kind == "ensemble":
        return dict(kind=kind, members=rng.randint(3, 16), min_nodes=1024, max_nodes=int(_log(rng, 4096, 40000)),
                    per_loop=rng.randint(100, 300), D=0.1, images="periodic_26", prec=rng.choice(["fp64", "mixed"]),
                    theta=theta, dt=5e-5, steps=rng.randint(1, 3))
    per_loop = rng.randint(64, 512)
    images = rng.choice(["periodic_26", "periodic_26", "periodic_18", "periodic_6", "wall_2_4", "wall_1_26"])
    c = dict(kind=kind, tangle="walk", per_loop=per_loop, images=images, theta=theta)
    if kind == "direct":
        n = _log(rng, 512, 40000)
        c["nodes"] = int(_log(rng, 64, 2048))
    else:
        c["prec"] = rng.choice(["fp64", "fp64", "mixed", "mixed", "dd"])
        n = _log(rng, 500, 262144 if kind == "eval" else 131072)
    c["loops"] = max(2, int(n / per_loop))
    # node density between a dilute tangle's and the benchmark's largest
    c["D"] = round((c["loops"] * per_loop / _log(rng, 1.3e7, 2.6e8)) ** (1 / 3), 4)
    if kind in ("rk4", "step"):
        c["images"] = "periodic_26"
        c["dt"] = round(_log(rng, 1e-5, 1e-4), 7)
    if kind == "step":
        c["smooth"] = rng.random() < 0.3
    return c


# ----------------------------------------------------------------- prepare
def _walk(loops, per_loop, D, seed, images):
    """Closed random-walk loops in the box, with its named image set; along an
    axis between mirror walls the loops are folded back into the box."""
    ht = W.random_walk_tangle(loops, per_loop, D=D, seed=seed)
    if images != "periodic_26":
        pos = ht.pos.reshape(loops, per_loop, 3)
        walls = abi.image_set(images)[1]
        for a in range(3):
            if abi.OV_WALL_MIRROR in walls[2 * a:2 * a + 2]:
                d = np.diff(pos[:, :, a], axis=1)
                z = pos[:, :1, a] + np.concatenate([np.zeros((loops, 1)), np.cumsum(d - D * np.round(d / D), 1)], 1)
                pos[:, :, a] = D - np.abs(np.mod(z, 2 * D) - D)
        ht = W.HostTangle(ht.pos, ht.conn[:, 0], ht.conn[:, 1], ht.box_lo, ht.box_hi, image_set=images)
    return ht


def _tangle(case, seed):
    if case["tangle"] == "rings":
        return W.ring_tangle(case["loops"], 0.02, D=case["D"], seed=seed)
    return _walk(case["loops"], case["per_loop"], case["D"], seed, case["images"])


def _sph_tangle(case, seed):
    return W.spherical_tangle(case["rings"], seed=seed, line=False, empty=0)


def _params(case):
    name = "rings8" if case.get("tangle") == "rings" else ("large" if case.get("smooth") else "rw")
    return W.config_params(name, bh_resolution=case["theta"])


def _room(ht, slots):
    """Host arrays to download into: `slots` slots, every page touched."""
    out = W.HostTangle(np.zeros((slots, 3)), np.full(slots, -1), np.full(slots, -1), ht.box_lo, ht.box_hi,
                       n_images=0, status=np.full(slots, abi.OV_EMPTY))
    for a in (out.pos, out.vels, out.vs, out.tangents, out.normals):
        a.fill(0.0)
    return out


def _ensemble(case, seed):
    u = np.random.default_rng(seed).uniform(size=(case["members"], 3))
    hosts, params = [], []
    for i, (b, c, d) in enumerate(u):
        # sizes spread evenly over the logarithm of the range (the case's, whatever the seed)
        n = case["min_nodes"] * (case["max_nodes"] / case["min_nodes"]) ** ((0.5 + 0.6180339887 * i) % 1.0)
        loops = max(1, int(round(n / case["per_loop"])))
        hosts.append(_walk(loops, case["per_loop"], case["D"], seed * 1000 + i, case["images"]))
        params.append(W.config_params("rw", bh_resolution=case["theta"], alpha=0.03 + 0.27 * b, alpha_p=0.02 * c,
                                      vn=(abi.OV_SIMPLE, 0.2 + 1.8 * d, (1, 0, 0))))
    return hosts, params


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, seed=seed)
    if kind == "spherical":
        p = gpu.sph_params_default()
        p.bh_resolution = case["theta"]
        p.use_temperature = 0
        s.update(ctx=gpu.Context(0, precision=PREC[case["prec"]]), host=_sph_tangle(case, seed), params=p)
        return s
    if kind == "ensemble":
        hosts, params = _ensemble(case, seed)
        s.update(ctx=gpu.Context(0, precision=PREC[case["prec"]]), host=hosts, params=params,
                 out=[_room(h, 2 * h.n) for h in hosts])
        return s
    ht = _tangle(case, seed)
    s.update(ctx=gpu.Context(0, params=_params(case), precision=PREC[case.get("prec", "fp64")]), host=ht)
    if kind == "direct":
        s["nodes"] = np.sort(np.random.default_rng(seed).permutation(ht.n)[:min(case["nodes"], ht.n)]).astype(np.int32)
    else:
        s["out"] = _room(ht, 2 * ht.n if kind == "step" else ht.n)
    return s


# --------------------------------------------------------------------- run
def run(s):
    case, ctx, host = s["case"], s["ctx"], s["host"]
    kind = case["kind"]
    if kind == "spherical":
        ctx.sph_update(host, s["params"], 0.0)
        return {"vels": host.vels, "vs": host.vs, "tangents": host.tangents, "normals": host.normals}
    if kind == "ensemble":
        ctx.upload_ensemble(host, s["params"])
        for i in range(case["steps"]):
            ctx.step(i * case["dt"], case["dt"])
        got = []
        for i, out in enumerate(s["out"]):
            m = ctx.download_member(i, out, abi.OV_F_POS | abi.OV_F_TOPOLOGY)
            got.append((m.pos, m.conn, m.stat))
        return got
    if kind == "step":
        ctx.upload(host)
        ctx.step(0.0, case["dt"])
        out = ctx.download_resized(s["out"])
        return {"pos": out.pos, "vels": out.vels, "conn": out.conn, "stat": out.stat}
    ctx.upload_fields(host, abi.OV_F_POS | abi.OV_F_TOPOLOGY)
    if kind == "direct":
        ctx.update_tangents_normals()
        vels, vs = ctx.direct_velocities(s["nodes"], 0.0)
        return {"vels": vels, "vs": vs}
    ctx.update_tangle(0.0)
    if kind == "rk4":
        ctx.rk4_step(0.0, case["dt"])
        out = ctx.download(s["out"], abi.OV_F_POS | abi.OV_F_VELS)
        return {"pos": out.pos, "vels": out.vels}
    out = ctx.download(s["out"], RESULTS)
    return {"vels": out.vels, "vs": out.vs, "tangents": out.tangents, "normals": out.normals}


# -------------------------------------------------------------------- work
def _accepts(n, theta):
    """Accepted cells per query point: 68 for 65,536 nodes at theta 0.4 (the
    tree's own counts), growing as theta^-2.6 and log(n)^2.6."""
    return min(n, 68.0 * (0.4 / theta) ** 2.6 * (math.log2(max(n, 2)) / 16.0) ** 2.6)


def work(case):
    """Positions and links in, results out; 42 flops an accepted segment."""
    kind = case["kind"]
    if kind == "spherical":
        n = 25 * case["rings"]
        return dict(bytes=n * (40.0 + 96.0), flops=42.0 * n * 18 * _accepts(n, case["theta"]))
    q = 1 + len(abi.image_set(case["images"])[0])
    if kind == "ensemble":
        lo, hi = case["min_nodes"], max(case["max_nodes"], case["min_nodes"] + 1)
        each = (hi - lo) / math.log(hi / lo)
        n, steps = case["members"] * each, case["steps"]
        return dict(bytes=n * 80.0, flops=42.0 * 4 * steps * n * q * _accepts(each, case["theta"]))
    n = case["loops"] * case["per_loop"]
    if kind == "direct":
        return dict(bytes=n * 40.0 + case["nodes"] * 48.0, flops=42.0 * min(case["nodes"], n) * n * q)
    evals = 1 if kind == "eval" else 4
    out = 96.0 if kind == "eval" else (48.0 if kind == "rk4" else 64.0)
    return dict(bytes=n * (40.0 + out), flops=42.0 * evals * n * q * _accepts(n, case["theta"]))


# ------------------------------------------------------------------- exact
def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _wrap(r1, r2, box):
    """r2 moved to the periodic copy nearest r1 (axes that are periodic)."""
    L, per = box["L"], box["per"]
    d = r2 - r1
    return r2 - torch.where(per & (d > L / 2), L, 0.0) + torch.where(per & (d < -L / 2), L, 0.0)


def _tangents(x, f, b, near):
    """Tangents and normals from the two neighbours on either side;
    near(r1, r2): r2's copy nearest r1."""
    s1, s2, m1, m2 = x[f], x[f[f]], x[b], x[b[b]]
    dist = lambda p, q: (near(p, q) - p).norm(dim=1)  # noqa: E731
    w = [near(x, p) - x for p in (s2, s1, m1, m2)]
    d1, e1 = w[1].norm(dim=1), w[2].norm(dim=1)
    d2, e2 = d1 + dist(s1, s2), e1 + dist(m1, m2)
    den = [d2 * (d2 - d1) * (e1 + d2) * (e2 + d2), d1 * (d2 - d1) * (e1 + d1) * (e2 + d1),
           e1 * (e1 + d1) * (e1 + d2) * (e2 - e1), e2 * (e2 + d1) * (e2 + d2) * (e2 - e1)]
    c1 = [-d1 * e1 * e2, d2 * e1 * e2, -d1 * d2 * e2, d1 * d2 * e1]
    c2 = [2 * ((e1 - d1) * e2 - d1 * e1), -2 * ((e1 - d2) * e2 - d2 * e1),
          2 * ((d2 + d1) * e2 - d1 * d2), -2 * ((d2 + d1) * e1 - d1 * d2)]
    tg = sum((c1[i] / den[i])[:, None] * w[i] for i in range(4))
    nm = sum((c2[i] / den[i])[:, None] * w[i] for i in range(4))
    return tg, nm


class _Tree:
    """Octree over coordinates `u` (Cartesian, or radius and angles), one node
    a leaf; monopoles of `pos` and `circ`.  `size(lo, hi)` gives a cell's Lm."""

    def __init__(self, u, lo, hi, pos, circ, size):
        dev = u.device
        self.com, self.circ, self.lm, self.n, self.first, self.kids = [], [], [], [], [], []
        node = torch.arange(len(u), device=dev)
        cell = torch.zeros(len(u), dtype=torch.long, device=dev)
        lo, hi = lo[None].clone(), hi[None].clone()
        base, level = 0, 0
        while True:
            nc = len(lo)
            cnt = torch.zeros(nc, device=dev, dtype=torch.float64).index_add_(0, cell, torch.ones_like(cell, dtype=torch.float64))
            com = torch.zeros(nc, 3, device=dev, dtype=torch.float64).index_add_(0, cell, pos[node]) / cnt[:, None]
            q = torch.zeros(nc, 3, device=dev, dtype=torch.float64).index_add_(0, cell, circ[node])
            self.com.append(com); self.circ.append(q); self.lm.append(size(lo, hi)); self.n.append(cnt)
            go = cnt[cell] > 1
            if level == 0:
                go &= ((u[node] >= lo) & (u[node] <= hi)).all(dim=1)
            node, par = node[go], cell[go]
            if len(node) == 0 or level > 60:
                self.first.append(torch.zeros(nc, dtype=torch.long, device=dev))
                self.kids.append(torch.zeros(nc, dtype=torch.long, device=dev))
                break
            mid = (lo + hi) / 2
            up = u[node] >= mid[par]
            digit = up[:, 0].long() + 2 * up[:, 1].long() + 4 * up[:, 2].long()
            keys, cell = torch.unique(par * 8 + digit, return_inverse=True)
            kp, kd = keys // 8, keys % 8
            kids = torch.zeros(nc, dtype=torch.long, device=dev).index_add_(0, kp, torch.ones_like(kp))
            self.kids.append(kids)
            base += nc
            self.first.append(base + torch.cumsum(kids, 0) - kids)
            bit = torch.stack([kd & 1, (kd >> 1) & 1, (kd >> 2) & 1], dim=1).bool()
            lo, hi = torch.where(bit, mid[kp], lo[kp]), torch.where(bit, hi[kp], mid[kp])
            level += 1
        for k in ("com", "circ", "lm", "n", "first", "kids"):
            setattr(self, k, torch.cat(getattr(self, k)))

    def sums(self, q, theta, f):
        """Barnes-Hut velocities of the segment monopoles at the points q."""
        out = torch.zeros_like(q)
        for at in range(0, len(q), 65536):
            p = q[at:at + 65536]
            t = torch.arange(len(p), device=q.device)
            c = torch.zeros_like(t)
            v = torch.zeros_like(p)
            while len(t):
                R = self.com[c] - p[t]
                d = R.norm(dim=1)
                seen = d >= 1e-8
                leaf = self.kids[c] == 0
                acc = seen & (leaf | (self.lm[c] / d < theta))
                v.index_add_(0, t[acc], _law(R[acc], self.circ[c[acc]], f))
                op = seen & ~acc
                t, c = t[op], c[op]
                k = self.kids[c]
                t = torch.repeat_interleave(t, k)
                start = torch.repeat_interleave(self.first[c] - (torch.cumsum(k, 0) - k), k)
                c = start + torch.arange(len(t), device=q.device)
            out[at:at + 65536] = v
        return out


def _law(R, S, f):
    """Biot-Savart velocity of straight segments from R to R + S."""
    P = R + S
    a, b, dot = R.norm(dim=-1), P.norm(dim=-1), (R * P).sum(-1)
    ok = (a >= 1e-8) & (b >= 1e-8) & (dot / a / b >= 1e-8)
    sc = torch.where(ok, f * (a + b) / (a * b * (a * b + dot)), 0.0)
    return _cross(R, S) * torch.nan_to_num(sc)[..., None]


def _reflected(box, j, p):
    """Image j's query points of p."""
    q = p - box["L"] * torch.tensor(box["images"][j][0], device=p.device, dtype=torch.float64)
    for face in box["images"][j][1]:
        ax = face // 2
        q[:, ax] = 2 * (box["hi"] if face & 1 else box["lo"])[ax] - p[:, ax]
    return q


def _back(box, j, v):
    for face in box["images"][j][1]:
        v[:, face // 2] = -v[:, face // 2]
    return v


def _friction(tg, vs, vn, alpha, alpha_p):
    c1 = _cross(tg, vn - vs)
    return vs + alpha * c1 - alpha_p * _cross(tg, c1)


def _lia(x, f, b, tg, nm, near, kappa, a0, clamp=None):
    l1, l2 = (near(x, x[f]) - x).norm(dim=1), (near(x[b], x) - x[b]).norm(dim=1)
    if clamp:
        l1, l2 = l1.clamp(*clamp), l2.clamp(*clamp)
    return _cross(tg, nm) * (kappa * torch.log(2 * torch.sqrt(l1 * l2) / math.sqrt(math.e) / a0) / 4 / math.pi)[:, None]


def _box(ht, images, dev):
    imgs, walls = abi.image_set(images)
    t = lambda v: torch.tensor(np.asarray(v), device=dev, dtype=torch.float64)  # noqa: E731
    lo, hi = t(ht.box_lo), t(ht.box_hi)
    per = torch.tensor([walls[2 * a] == abi.OV_WALL_PERIODIC for a in range(3)], device=dev)
    return dict(lo=lo, hi=hi, L=hi - lo, per=per, images=imgs)


def _eval(x, f, b, box, p, vn, nodes=None):
    """tangents, normals, vs and vels of every node (of `nodes` by direct sums)."""
    near = lambda r1, r2: _wrap(r1, r2, box)  # noqa: E731
    tg, nm = _tangents(x, f, b, near)
    vs = _lia(x, f, b, tg, nm, near, p.kappa, p.vortex_width)
    circ = near(x, x[f]) - x
    f4 = p.kappa / 4 / math.pi
    if nodes is None:
        tree = _Tree(x, box["lo"], box["hi"], x, circ, lambda lo, hi: (hi - lo).amax(dim=1))
        vs = vs + tree.sums(x, p.bh_resolution, f4)
        for j in range(len(box["images"])):
            vs = vs + _back(box, j, tree.sums(_reflected(box, j, x), p.bh_resolution, f4))
    else:
        tg, vs, y = tg[nodes], vs[nodes], x[nodes]
        for j in range(-1, len(box["images"])):
            # the node's own two segments are left out of its primary sum; the
            # direct sum adds mirror images unreflected
            q = y if j < 0 else _reflected(box, j, y)
            sums = []
            for i in range(0, len(q), 64):
                w = _law(x[None] - q[i:i + 64, None], circ[None], f4)
                if j < 0:
                    at, me = torch.arange(len(w), device=x.device), nodes[i:i + 64].long()
                    w[at, me] = 0.0
                    w[at, b[me]] = 0.0
                sums.append(w.sum(1))
            vs = vs + torch.cat(sums)
    vel = _friction(tg, vs, vn, p.alpha, p.alpha_p) if p.use_mutual_friction else vs
    return tg, nm, vs, vel


def _sph_angles(x):
    return torch.stack([x.norm(dim=1), torch.atan2(x[:, 2], x[:, :2].norm(dim=1)), torch.atan2(x[:, 1], x[:, 0])], 1)


def _sph_point(u):
    r, az, pl = u.unbind(1)
    return torch.stack([r * torch.cos(az) * torch.cos(pl), r * torch.cos(az) * torch.sin(pl), r * torch.sin(az)], 1)


def _exact_spherical(case, seed, dev):
    """Rings in a section of a shell: the section's tree, the tree of the
    tangle inverted through the inner surface, 8 rotated copies of both."""
    ht = _sph_tangle(case, seed)
    p = gpu.sph_params_default()
    ri, ro, A, P = ht.domain
    t = lambda v: torch.tensor(np.asarray(v), device=dev)  # noqa: E731
    row = lambda *v: torch.tensor(v, device=dev, dtype=torch.float64)  # noqa: E731
    x, f, b = t(ht.pos), t(ht.conn[:, 0]).long(), t(ht.conn[:, 1]).long()

    def near(r1, r2):
        w = _sph_angles(r2)
        d = w - _sph_angles(r1)
        return _sph_point(torch.stack([w[:, 0]] + [
            w[:, k] - torch.where(d[:, k].abs() > h, torch.round(d[:, k] / (2 * h)) * 2 * h, 0.0)
            for k, h in ((1, A), (2, P))], 1))

    def size(lo, hi):
        chord = lambda w: 2 * torch.sin(w / 2).abs()  # noqa: E731
        az = hi[:, 0] * chord(hi[:, 1] - lo[:, 1])
        pl = hi[:, 0] * chord(hi[:, 2] - lo[:, 2]) * torch.cos((hi[:, 1] + lo[:, 1]) / 2).abs()
        return torch.stack([hi[:, 0] - lo[:, 0], az, pl], 1).amax(1)

    def tree_of(pts, r0, r1):
        ds = near(pts, pts[f]) - pts
        circ = torch.where(ds.norm(dim=1, keepdim=True) > 5 * p.dl_max, 0.0, ds)
        return _Tree(_sph_angles(pts), row(r0, -A, -P), row(r1, A, P), pts, circ, size)

    u = _sph_angles(x)
    image = _sph_point(torch.stack([ri * ri / u[:, 0], u[:, 1], u[:, 2]], 1))
    tg, nm = _tangents(x, f, b, near)
    vs = _lia(x, f, b, tg, nm, near, p.kappa, p.vortex_width, (p.dl_min / 4, 4 * p.dl_max))
    for tree, sign in ((tree_of(x, ri, ro), 1.0), (tree_of(image, ri * ri / ro, ri), -1.0)):
        for sa, sp in ((0, 0), (1, 0), (-1, 0), (0, 1), (0, -1), (1, 1), (-1, 1), (1, -1), (-1, -1)):
            rot = row(0.0, 2 * A * sa, 2 * P * sp)
            v = tree.sums(_sph_point(u + rot) if sa or sp else x, case["theta"], p.kappa / 4 / math.pi)
            vs = vs + sign * (_sph_point(_sph_angles(v) - rot) if sa or sp else v)
    vel = _friction(tg, vs, torch.zeros_like(vs), p.alpha, p.alpha_p) if p.use_mutual_friction else vs
    return {"vels": vel, "vs": vs, "tangents": tg, "normals": nm}


def exact(case, seed):
    kind = case["kind"]
    dev = "cuda"
    if kind in ("step", "ensemble"):
        return None   # the topology passes decide on sums; no plain 64-bit counterpart
    if kind == "spherical":
        return _exact_spherical(case, seed, dev)
    ht = _tangle(case, seed)
    p = _params(case)
    box = _box(ht, case["images"], dev)
    t = lambda v: torch.tensor(np.asarray(v), device=dev)  # noqa: E731
    x, f, b = t(ht.pos), t(ht.conn[:, 0]).long(), t(ht.conn[:, 1]).long()
    vn = torch.tensor([p.vn.strength, 0.0, 0.0], device=dev, dtype=torch.float64)
    if kind == "direct":
        nodes = np.sort(np.random.default_rng(seed).permutation(ht.n)[:min(case["nodes"], ht.n)])
        _, _, vs, vel = _eval(x, f, b, box, p, vn, t(nodes))
        return {"vels": vel, "vs": vs}
    tg, nm, vs, vel = _eval(x, f, b, box, p, vn)
    if kind == "eval":
        return {"vels": vel, "vs": vs, "tangents": tg, "normals": nm}
    # RK4 with every stage displaced by dt/2 from the start
    dt, ks = case["dt"], [vel]
    for _ in range(3):
        ks.append(_eval(x + ks[-1] * (dt / 2), f, b, box, p, vn)[3])
    return {"pos": x + ks[0] * (dt / 6) + ks[1] * (dt / 3) + ks[2] * (dt / 3) + ks[3] * (dt / 6), "vels": vel}
