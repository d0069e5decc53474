"""Quick phases of fq_sin and fq_log (csrc/fq_math.h) where their errors are largest beside the result: sin close to
the multiples of pi, on both sides of the distance 2^-20 below which it leaves them to the full evaluation, and log of
arguments of all exponents and close to 1.  In every set nearly all points have to be compared."""

import shutil
import subprocess

import pytest
from test_math_quick import CSRC

SOURCE = r"""
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include "fq_math.h"
static uint64_t s = 0x9E3779B97F4A7C15ULL;
static uint64_t r64(void)
{
    s = s * 6364136223846793005ULL + 1442695040888963407ULL;
    return s ^ (s >> 29);
}
static double u01(void) { return (double)(r64() >> 11) * 0x1p-53; }
int main(int argc, char** argv)
{
    const int which = atoi(argv[1]);
    const long n = atol(argv[2]);
    long bad = 0, full = 0;
    for (long i = 0; i < n; ++i) {
        double x, y;
        if (which <= 2) {
            /* offsets from k pi, log-uniform: 2^-20 .. 2^-6 (0), 2^-20 .. 2^-18 (1), 2^-24 .. 2^-20 (2) */
            const double lo = which == 2 ? -24.0 : -20.0, hi = which == 0 ? -6.0 : which == 1 ? -18.0 : -20.0;
            const double t = exp2(lo + (hi - lo) * u01());
            x = (double)(i % 7 - 3) * 3.14159265358979312 + ((r64() >> 40) & 1 ? t : -t);
        }
        else if (which == 3) {
            x = ldexp(1.0 + (double)(r64() >> 32) * 0x1p-32, (int)(r64() >> 40) % 2000 - 1000);
        }
        else {
            x = 1.0 + ((r64() >> 40) & 1 ? -1.0 : 1.0) * floor(exp2(30.0 * u01())) * 0x1p-32;
        }
        if (which <= 2 ? !fq_sin_quick(x, &y) : !fq_log_quick(x, &y)) {
            ++full;
            continue;
        }
        const double z = which <= 2 ? fq_sin_full(x) : fq_log_full(x);
        bad += fq_bits(y) != fq_bits(z);
    }
    printf("%ld %ld\n", bad, full);
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs gcc")
@pytest.mark.parametrize("which", range(5))
def test_quick_equals_full(tmp_path, which):
    (tmp_path / "q.c").write_text(SOURCE)
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", f"-I{CSRC}", str(tmp_path / "q.c"), "-o", str(tmp_path / "q"),
                    "-lm"], check=True, capture_output=True)
    n = 2000000
    r = subprocess.run([str(tmp_path / "q"), str(which), str(n)], check=True, capture_output=True, text=True)
    bad, full = map(int, r.stdout.split())
    assert bad == 0
    if which == 2:
        assert full > 0.99 * n  # below the cutoff
    else:
        assert full < 0.02 * n
