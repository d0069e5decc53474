"""Integer-pipe product by a prepared factor (fq_soft64.h, fq_smulc): bit-identical to the IEEE product."""

import pathlib
import shutil
import subprocess

import pytest

HERE = pathlib.Path(__file__).resolve().parent
CSRC = HERE.parent / "frictionqpotspringblock_gb300" / "csrc"


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
@pytest.mark.parametrize("family", [0, 1, 2, 3])
def test_factor_host_bit_exact(tmp_path, family):
    exe = tmp_path / "check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{CSRC}",
                    str(HERE / "soft64" / "soft64_factor_check.cpp"), "-o", str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe), str(family), "100000"], capture_output=True, text=True)
    ops, bad, slow = map(int, r.stdout.split())
    assert r.returncode == 0 and bad == 0
    if family == 0:
        # the parameters of a step: the fast path carries the operands around 1 (half of the cases)
        assert slow < 0.2 * ops
