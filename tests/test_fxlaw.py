"""The integer-mantissa segment law of the FP64 path (csrc/ov_fxlaw.cuh).

CPU: the header's host build against the law in long double over the
geometries it accepts, with the words where its carries and signs can go
wrong.  GPU: the split walk that uses it against the all-FP64 walk at the
edges of its tiles, lists and fallbacks.
"""
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
static unsigned long long s;
static unsigned long long rnd() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static double un() { return (double)(rnd() >> 11) * 0x1p-53; }
int main(int argc, char **argv)
{
    const double span = atof(argv[1]), smax = atof(argv[2]);   // distance range, largest |S| / |R|
    const int zeros = atoi(argv[3]);                          // low zero bits of every coordinate
    s = 88172645463325252ull;
    long taken = 0, bad = 0;
    for (long it = 0; it < 400000; ++it) {
        const double d = 0x1p51 * pow(span, un()), mag = smax * pow(1e-4, un());
        int64_t q[3], R[3], S[3], at[3];
        for (int i = 0; i < 3; ++i) {
            const int64_t mask = ~((1ll << zeros) - 1);
            q[i] = (int64_t)((un() - 0.5) * 0x1p60) & mask;
            R[i] = (int64_t)((2 * un() - 1) * d) & mask;
            S[i] = (int64_t)((2 * un() - 1) * d * mag) & mask;
            at[i] = q[i] + R[i];
        }
        const CellFX c = fx_cell(at, S, true);
        if (c.e < 0) continue;
        fx_sum w[3] = {{0, 0}, {0, 0}, {0, 0}};
        if (!fx_law(c, q, true, w)) {
            for (int i = 0; i < 3; ++i) bad += w[i].h != 0 || w[i].l != 0;   // left untouched
            continue;
        }
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
            // 2^-49 of |R||S| sc (squared lengths are off by a few units of 2^52 at
            // least), and 2 units for the aligned quotient's last bit
            if (fabsl(g - x[i]) > 0x1p-49L * a * sqrtl(n) * sc + ldexpl(2, kFxUnit)) ++bad;
        }
    }
    printf("%ld %ld\n", taken, bad);
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("fxlaw")
    (d / "t.cpp").write_text(HARNESS)
    subprocess.run([cxx, "-O2", "-std=c++17", f"-I{CSRC}", "-o", str(d / "t"), str(d / "t.cpp")], check=True)
    return str(d / "t")


@pytest.mark.parametrize("span,smax,zeros", [
    (4.0, 1.0, 0),       # the nearest it takes
    (512.0, 0.5, 0),     # every distance, short segments
    (512.0, 8.0, 0),     # segments longer than the distance
    (512.0, 0.5, 20),    # coordinates of coarse numbers: low words of exactly 2^31
    (512.0, 1e-6, 6),    # circulations that nearly cancel
])
def test_law_against_long_double(harness, span, smax, zeros):
    taken, bad = map(int, subprocess.run([harness, repr(span), repr(smax), str(zeros)], capture_output=True,
                                         text=True, check=True).stdout.split())
    assert taken > 20000
    assert bad == 0


def _close(n, D, gap, seed):
    """n nodes on small rings whose neighbours are a few grid steps apart: more
    cells than a lane's list of FP64 terms holds."""
    ht = W.random_walk_tangle(max(1, n // 32), 32, D=D, delta=gap, seed=seed)
    ht.pos[:] = 0.4 * D + 0.02 * ht.pos
    return ht


@pytest.mark.gpu
@pytest.mark.parametrize("make,theta", [
    (lambda: W.random_walk_tangle(1, 31, D=0.1, seed=3), 0.4),        # less than one tile
    (lambda: W.random_walk_tangle(3, 11, D=0.1, seed=4), 0.4),        # one lane of a second tile
    (lambda: W.random_walk_tangle(65, 64, D=0.05, seed=5), 0.12),     # lists flushed many times a walk
    (lambda: _close(2048, 0.1, 1e-5, 6), 0.4),                         # most cells left to the FP64 law
    (lambda: W.random_walk_tangle(40, 256, D=4.0, seed=7), 0.4),      # coarse grid: near cells in FP64
    (lambda: W.random_walk_tangle(300, 30, D=0.1, seed=8, n_images=6), 0.4),
])
def test_split_walk_equals_fp64_walk(make, theta):
    from openvort_gb300 import gpu
    got = []
    for walk in (abi.OV_WALK_FP64, abi.OV_WALK_SPLIT):
        ht = make()
        ctx = gpu.Context(0, params=W.config_params("rw", bh_resolution=theta))
        ctx.set_walk(walk)
        ctx.upload(ht)
        ctx.update_tangle(0.0)
        ctx.download(ht)
        st = ctx.stats()
        ctx.close()
        got.append((ht.vs.copy(), st))
    (v64, s64), (v, s) = got
    assert s["visits"] == s64["visits"] and s["accepts"] == s64["accepts"]
    # the all-FP64 law rounds R x Rp1 relative to |R||Rp1|, up to 10^4 |R||S| here
    per_node = np.linalg.norm(v - v64, axis=1) / np.linalg.norm(v64, axis=1)
    assert per_node.max() < 1e-10
    assert np.linalg.norm(v - v64) < 1e-12 * np.linalg.norm(v64)


@pytest.mark.gpu
@pytest.mark.parametrize("make,nodes", [
    (lambda: W.random_walk_tangle(1, 7, D=0.1, seed=3), 7),              # fewer segments than threads
    (lambda: W.random_walk_tangle(3, 257, D=0.1, seed=4), 1),            # one node: shortest chunks
    (lambda: W.random_walk_tangle(70, 250, D=0.1, seed=5, n_images=6), 130),   # a ragged last chunk
    (lambda: _close(600, 0.1, 1e-5, 6), 50),                              # nearly every segment left to FP64
])
def test_direct_sums_equal_fp64_terms(make, nodes):
    """The direct sums' integer law against the allocation-free entry point,
    which evaluates every term in FP64, at the FP64 parity tolerance."""
    torch = pytest.importorskip("torch")
    from tests._util import node_rel_err
    from tests.test_zz_no_alloc import _Caller, _reference
    ht = make()
    p = W.config_params("rw")
    ids = np.linspace(0, ht.n - 1, nodes).astype(np.int32)
    (ref,) = _reference(ht, p, [ids])
    got = _Caller(torch, ht, p).call(ids)
    assert node_rel_err(got[0], ref[0]) < 1e-10
    assert node_rel_err(got[1], ref[1]) < 1e-10
