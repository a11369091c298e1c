"""The integer law with its FP32 seeds at the ends of their documented error
(rsqrt.approx 2^-22.9, rcp.approx 1 ulp): the header's host build with the two
host seeds off by that much, against the law in long double as
tests/test_fxlaw.py has it for correctly rounded ones, to the same bound."""
import os
import shutil
import subprocess

import pytest

from tests.test_fxlaw import CSRC, HARNESS

SQRT = r"""
#include <cstdio>
#include <cmath>
#include "ov_fxlaw.cuh"
int main()
{
    unsigned long long s = 88172645463325252ull;
    long bad = 0;
    for (long it = 0; it < 3000000; ++it) {
        s ^= s << 13; s ^= s >> 7; s ^= s << 17;
        const int64_t a = (int64_t)((s >> 2 | 1ull << 61) >> (it % 12));   // 2^50 .. 2^62
        // one unit each for the truncated residual, the rounded last digit and what the
        // seed's error leaves of it, and one for the square left out
        bad += fabsl((long double)fx_sqrt(a) - sqrtl((long double)a) * 0x1p32L) > 4.0L;
    }
    printf("%ld\n", bad);
}
"""

RSQRT = "{ return 1.0f / sqrtf(x); }"
RCP = "{ return 1.0f / x; }"


@pytest.fixture(scope="module")
def build(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    header = open(os.path.join(CSRC, "ov_fxlaw.cuh")).read()
    assert header.count(RSQRT) == 1 and header.count(RCP) == 1

    def make(root, reciprocal, source=HARNESS):
        d = tmp_path_factory.mktemp("seeds")
        (d / "ov_fxlaw.cuh").write_text(
            header.replace(RSQRT, f"{{ return (float)((1.0 / sqrt((double)x)) * (1.0 + {root!r})); }}")
            .replace(RCP, f"{{ return (float)((1.0 / (double)x) * (1.0 + {reciprocal!r})); }}"))
        (d / "t.cpp").write_text(source)
        subprocess.run([cxx, "-O2", "-std=c++17", f"-I{d}", "-o", str(d / "t"), str(d / "t.cpp")], check=True)
        return str(d / "t")

    return make


@pytest.mark.parametrize("root", [-2.0 ** -22.9, 2.0 ** -22.9])
@pytest.mark.parametrize("reciprocal", [-2.0 ** -23, 2.0 ** -23])
def test_law_with_seeds_at_the_ends_of_their_error(build, root, reciprocal):
    exe = build(root, reciprocal)
    for span, smax, zeros in ((4.0, 1.0, 0), (512.0, 0.5, 0), (512.0, 8.0, 0), (512.0, 0.5, 20), (512.0, 1e-6, 6)):
        taken, bad = map(int, subprocess.run([exe, repr(span), repr(smax), str(zeros)], capture_output=True, text=True,
                                             check=True).stdout.split())
        assert taken > 20000
        assert bad == 0, (span, smax, zeros)


@pytest.mark.parametrize("root", [-2.0 ** -22.9, 0.0, 2.0 ** -22.9])
def test_root_to_its_last_units(build, root):
    exe = build(root, 0.0, SQRT)
    assert subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split() == ["0"]
