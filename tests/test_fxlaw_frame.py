"""The integer law's coordinates (fx_frame in csrc/ov_fxlaw.cuh) in boxes off the
origin: counted from the box, so that what the law takes does not depend on
where the box lies.  CPU: the header's host build.  GPU: the split walk
against the all-FP64 walk."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from openvort_gb300 import abi, workloads as W

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "openvort_gb300", "csrc")

HARNESS = r"""
#include <cstdio>
#include <cmath>
#include <cstdlib>
#include "ov_fxlaw.cuh"
typedef long double LD;
static unsigned long long s = 88172645463325252ull;
static double un() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return (double)(s >> 11) * 0x1p-53; }
int main(int argc, char **argv)
{
    double lo[3], hi[3], L = 0;
    for (int a = 0; a < 3; ++a) { lo[a] = atof(argv[1 + a]); hi[a] = atof(argv[4 + a]); L = fmax(L, hi[a] - lo[a]); }
    const FxFrame f = fx_frame(lo, hi);
    long refused = 0, inexact = 0, large = 0;
    for (int it = 0; it < 100000; ++it) {
        // a point of the box, and one at a distance (largest component) of a 160th of the box
        // or more, up to the next period
        double p[3], c[3], far = 0;
        int64_t q[3], x[3];
        const double r = L / 150 * pow(150.0, un());
        double dir[3], n = 0;
        for (int a = 0; a < 3; ++a) { dir[a] = un() - 0.5; n += dir[a] * dir[a]; }
        for (int a = 0; a < 3; ++a) {
            p[a] = lo[a] + un() * (hi[a] - lo[a]);
            c[a] = p[a] + r * dir[a] / sqrt(n);
            far = fmax(far, fabs(c[a] - p[a]));
            const double u = fma(p[a], f.inv, f.at[a]), v = fma(c[a], f.inv, f.at[a]);
            large += fabs(u) >= kFxLimit || fabs(v) >= kFxLimit;
            q[a] = (int64_t)rint(u);
            x[a] = (int64_t)rint(v);
            // differences of coordinates: as of the numbers themselves, to one unit's rounding
            inexact += fabsl((LD)(x[a] - q[a]) - ((LD)c[a] - (LD)p[a]) * f.inv) > 1.0L;
        }
        if (far < L / 160) continue;
        int64_t S[3];
        for (int a = 0; a < 3; ++a) S[a] = (int64_t)((un() - 0.5) * r * f.inv * 0.5);
        const CellFX cell = fx_cell(x, S, true);
        fx_sum w[3] = {{0, 0}, {0, 0}, {0, 0}};
        refused += !fx_law(cell, q, true, w, kFxMaxShift);
    }
    printf("%ld %ld %ld %d\n", refused, inexact, large, ilogb(f.inv * f.u));
}
"""


# The law below 2^51 units, where both sides are whole numbers of units, and the
# test of that.
NEAR = r"""
#include <cstdio>
#include <cmath>
#include "ov_fxlaw.cuh"
typedef long double LD;
static unsigned long long s = 88172645463325252ull;
static unsigned long long rnd() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static double un() { return (double)(rnd() >> 11) * 0x1p-53; }
int main()
{
    long taken = 0, bad = 0, flags = 0, early = 0;
    for (long it = 0; it < 400000; ++it) {
        const double d = 0x1p47 * pow(16.0, un()), mag = pow(1e-4, un());
        int64_t q[3], R[3], S[3], at[3], top = 0;
        for (int i = 0; i < 3; ++i) {
            q[i] = (int64_t)((un() - 0.5) * 0x1p60);
            R[i] = (int64_t)((2 * un() - 1) * d);
            S[i] = (int64_t)((2 * un() - 1) * d * mag);
            at[i] = q[i] + R[i];
            top = R[i] > top ? R[i] : (-R[i] > top ? -R[i] : top);
        }
        fx_sum w[3] = {{0, 0}, {0, 0}, {0, 0}};
        // rounded coordinates on either side: not below 2^51 units
        if (top < (1ll << 51) - 1) {
            early += fx_law(fx_cell(at, S, true), q, true, w, kFxWholeShift);
            early += fx_law(fx_cell(at, S, true, kFxWholeShift), q, true, w);
            for (int i = 0; i < 3; ++i) early += w[i].h != 0 || w[i].l != 0;
        }
        const CellFX c = fx_cell(at, S, true, kFxWholeShift);
        if (c.e < 0 || !fx_law(c, q, true, w, kFxWholeShift)) continue;
        ++taken;
        LD a = 0, b = 0, t = 0, n = 0;
        for (int i = 0; i < 3; ++i) {
            const LD P = (LD)R[i] + S[i];
            a += (LD)R[i] * R[i]; b += P * P; t += R[i] * P; n += (LD)S[i] * S[i];
        }
        a = sqrtl(a); b = sqrtl(b);
        const LD sc = (a + b) / (a * b * (a * b + t));
        const LD x[3] = {((LD)R[1] * S[2] - (LD)R[2] * S[1]) * sc, ((LD)R[2] * S[0] - (LD)R[0] * S[2]) * sc,
                         ((LD)R[0] * S[1] - (LD)R[1] * S[0]) * sc};
        for (int i = 0; i < 3; ++i) {
            const LD g = ldexpl((LD)w[i].h + ldexpl((LD)w[i].l, -32), kFxUnit);
            // as for the larger separations: 2^-49 of |R||S| sc, and 2 units
            bad += fabsl(g - x[i]) > 0x1p-49L * a * sqrtl(n) * sc + ldexpl(2, kFxUnit);
        }
    }
    for (long it = 0; it < 400000; ++it) {
        const double x = ldexp(2 * un() - 1, (int)(un() * 70)) , y = it & 1 ? rint(x) : x;
        flags += fx_whole(y) != (y == rint(y));
    }
    // counted from 4: exact where 4 takes no bits from a number, known to be rounded elsewhere
    FxFrame f = fx_unit(-58);
    f.at[0] = -4 * f.inv;
    for (long it = 0; it < 400000; ++it) {
        const double x = ldexp(2 * un() - 1, (int)(un() * 70) - 66), r = fma(x, f.inv, f.at[0]);
        const bool exact = (LD)r == (LD)x * f.inv + f.at[0];
        const int t = fx_shift(r, x, f);
        flags += t >= 0 && t != kFxRoundShift && (!exact || (t == f.whole) != (r == rint(r)));
        flags += t == kFxRoundShift && fabs(r) <= fabs(x * f.inv) / 2;
        flags += fx_shift(x * f.inv, x, f) == kFxRoundShift;
        flags += (t < 0) != (fabs(r) >= kFxLimit);
    }
    flags += fx_shift(NAN, NAN, f) >= 0 || fx_shift(INFINITY, INFINITY, f) >= 0;
    flags += !fx_whole(0.0) + !fx_whole(-0.0) + !fx_whole(1.0) + fx_whole(0.5) + fx_whole(-1.5);
    printf("%d %ld %ld %ld\n", taken > 100000, bad, early, flags);
}
"""


def _built(tmp_path_factory, source):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("fxframe")
    (d / "t.cpp").write_text(source)
    subprocess.run([cxx, "-O2", "-std=c++17", f"-I{CSRC}", "-o", str(d / "t"), str(d / "t.cpp")], check=True)
    return str(d / "t")


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    return _built(tmp_path_factory, HARNESS)


def test_near_separations_of_whole_coordinates(tmp_path_factory):
    exe = _built(tmp_path_factory, NEAR)
    got = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()
    assert list(map(int, got)) == [1, 0, 0, 0]


@pytest.mark.parametrize("lo,side", [
    ((0, 0, 0), (0.1, 0.1, 0.1)),
    ((10, 10, 10), (0.1, 0.1, 0.1)),
    ((50, 50, 50), (0.1, 0.1, 0.1)),
    ((-50.1, -50.1, -50.1), (0.1, 0.1, 0.1)),
    ((-0.05, -0.05, -0.05), (0.1, 0.1, 0.1)),
    ((0.17, -3.3, -0.02), (0.1, 0.1, 0.1)),      # beyond, before and around the origin
    ((0.07, 0.01, -0.19), (0.1, 0.1, 0.1)),      # within a length of it
    ((1000.0, 0, -1), (1.0, 1.0, 1.0)),
])
def test_law_takes_the_same_distances_wherever_the_box_lies(harness, lo, side):
    hi = [a + b for a, b in zip(lo, side)]
    got = subprocess.run([harness, *map(repr, map(float, lo)), *map(repr, hi)], capture_output=True, text=True,
                         check=True).stdout.split()
    assert list(map(int, got)) == [0, 0, 0, 0]


def _moved(ht, off, images="periodic_26"):
    off = np.asarray(off, dtype=np.float64)
    return W.HostTangle(ht.pos + off, ht.conn[:, 0], ht.conn[:, 1], ht.box_lo + off, ht.box_hi + off,
                        image_set=images)


def _small(loops, per_loop, size, box, at=0.37):
    """A tangle that is small against its open box: many or all interactions are left
    to the FP64 law, more than a late list holds at each query point."""
    ht = W.random_walk_tangle(loops, per_loop, D=size, delta=size * 0.006, seed=3)
    return W.HostTangle(ht.pos + at * box, ht.conn[:, 0], ht.conn[:, 1], np.zeros(3), np.full(3, box),
                        image_set="open")


@pytest.mark.gpu
@pytest.mark.parametrize("make", [
    lambda: _moved(W.random_walk_tangle(33, 64, D=0.1, seed=5), [10, 10, 10]),
    lambda: _moved(W.random_walk_tangle(33, 64, D=0.1, seed=5), [-50.1, -50.1, -50.1]),
    lambda: _moved(W.random_walk_tangle(33, 64, D=0.1, seed=5), [10, -0.05, -50]),
    lambda: _moved(W.random_walk_tangle(33, 64, D=0.1, seed=5), [50, 50, 50], "wall_2_4"),
    lambda: _small(16, 67, 0.0005, 0.1),
    lambda: _small(3, 33, 0.0001, 0.1),
    lambda: _small(16, 67, 0.0005, 0.1, at=0.0),     # beside the planes from which coordinates are counted
    lambda: _small(16, 67, 1e-5, 0.1),               # nothing else than the FP64 law's
])
def test_split_walk_equals_fp64_walk_off_the_origin(make):
    from openvort_gb300 import gpu
    got = []
    for walk in (abi.OV_WALK_FP64, abi.OV_WALK_SPLIT):
        ht = make()
        ctx = gpu.Context(0, params=W.config_params("rw"))
        ctx.set_walk(walk)
        ctx.upload(ht)
        ctx.update_tangle(0.0)
        ctx.download(ht)
        st = ctx.stats()
        ctx.close()
        got.append((ht.vs.copy(), st))
    (v64, s64), (v, s) = got
    assert s["visits"] == s64["visits"] and s["accepts"] == s64["accepts"]
    assert s["error_word"] == s64["error_word"] and s["error_word"] in (0, 1)   # (1: nodes sharing a deepest cell)
    # the all-FP64 law rounds R x Rp1 relative to |R||Rp1|, up to 10^4 |R||S| here
    per_node = np.linalg.norm(v - v64, axis=1) / np.linalg.norm(v64, axis=1)
    assert per_node.max() < 1e-10
    assert np.linalg.norm(v - v64) < 1e-12 * np.linalg.norm(v64)
