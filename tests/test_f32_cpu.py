"""The FP32 form's arguments without FP64 (da-gtm_gb300/csrc/f32pair.cuh), compiled for the
host from the same header: the bits of the FP64 expressions (tests/f32_check.cc)."""
import os
import subprocess

from conftest import ROOT


def test_arguments_have_the_bits_of_the_fp64_expressions(tmp_path):
    exe = str(tmp_path / "f32_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                           os.path.join(ROOT, "tests", "f32_check.cc"), "-lm"])
    bad1, bad2, badw, slow = subprocess.run([exe], capture_output=True, text=True, timeout=300,
                                            check=True).stdout.split()
    assert int(bad1) == 0 and int(bad2) == 0 and int(badw) == 0
    # the inputs are built to lie at rounding boundaries; most still need no FP64
    assert float(slow) < 0.25
