"""Quick phases of fq_log and fq_sin (csrc/fq_math.h): where they round, they round to the double of the full
evaluation -- over the yield distances' arguments 1 - u32 2^-32 (both ends and a stride through the rest), and
over the phases of the Smooth potential with the surroundings of the multiples of pi."""

import pathlib
import shutil
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "frictionqpotspringblock_gb300" / "csrc"

SOURCE = r"""
#include <stdio.h>
#include <stdlib.h>
#include "fq_math.h"
int main(int argc, char** argv)
{
    const int which = atoi(argv[1]);
    const long n = atol(argv[2]);
    long bad = 0, full = 0;
    for (long i = 0; i < n; ++i) {
        double x, y;
        if (which == 0) {
            const uint32_t k = i < 100000 ? (uint32_t)i : i < 200000 ? (uint32_t)(100000 - i) : (uint32_t)(i * 2654435761u);
            x = 1.0 - k * 0x1p-32;
        }
        else {
            const double t = (double)(uint32_t)(i * 2654435761u) * 0x1p-32 - 0.5;
            x = which == 1 ? t * 6.5 : which == 2 ? t * 25.0 : (double)(i % 9 - 4) * 3.14159265358979312 + t * 1e-7;
        }
        if (which == 0 ? !fq_log_quick(x, &y) : !fq_sin_quick(x, &y)) {
            ++full;
            continue;
        }
        const double z = which == 0 ? fq_log_full(x) : fq_sin_full(x);
        bad += fq_bits(y) != fq_bits(z);
    }
    printf("%ld %ld\n", bad, full);
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs gcc")
@pytest.mark.parametrize("which", [0, 1, 2, 3])
def test_quick_equals_full(tmp_path, which):
    (tmp_path / "q.c").write_text(SOURCE)
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", f"-I{CSRC}", str(tmp_path / "q.c"), "-o", str(tmp_path / "q"),
                    "-lm"], check=True, capture_output=True)
    n = 2000000
    r = subprocess.run([str(tmp_path / "q"), str(which), str(n)], check=True, capture_output=True, text=True)
    bad, full = map(int, r.stdout.split())
    assert bad == 0
    if which < 3:
        assert full < n / 200  # about 2^-10 of the arguments are evaluated in full


def test_table_is_its_generators_output():
    pytest.importorskip("mpmath")
    r = subprocess.run(["python3", str(CSRC / "gen_log_table.py")], check=True, capture_output=True, text=True)
    assert r.stdout == (CSRC / "fq_log_table.h").read_text()
