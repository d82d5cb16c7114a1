"""The fixed-point pieces of the digit-slice products
(da-gtm_gb300/csrc/ozfix.cuh), compiled for the host from the same header and
checked against long-double references (tests/oz_check.cc): digits rebuild the
56-bit integer and the integer the value to half a unit; exp2_neg within 2^-57
and its double within one FP64 rounding (2^-53); the fixed-point product within
one unit (2^-53) below 2000, at scales of 2^-60 to 1."""
import os
import subprocess

from conftest import ROOT


def test_fixed_point_pieces(tmp_path):
    exe = str(tmp_path / "oz_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                           os.path.join(ROOT, "tests", "oz_check.cc"), "-lm"])
    bad, exp2, dbl, prod = subprocess.run([exe], capture_output=True, text=True, timeout=300,
                                          check=True).stdout.split()
    assert float(bad) == 0
    assert float(exp2) <= 2.0 ** -57
    assert float(dbl) <= 2.0 ** -53 + 2.0 ** -57
    assert float(prod) <= 1.0


def test_exponents_over_the_whole_range(tmp_path):
    """Every power that FP64 can hold (to 2^-1074) has an exponent, whatever the
    mantissa of kappa and the unit (tests/oz_range_check.cc); within two units."""
    exe = str(tmp_path / "oz_range_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                           os.path.join(ROOT, "tests", "oz_range_check.cc"), "-lm"])
    dropped, beyond, worst = subprocess.run([exe], capture_output=True, text=True, timeout=300,
                                            check=True).stdout.split()
    assert int(dropped) == 0 and int(beyond) == 0
    assert float(worst) <= 2.0


def test_units_of_the_distances(tmp_path):
    """v = t.y - |y|^2 / 2 on each point's own unit, for sizes over 400 powers of two
    (tests/oz_unit_check.cc): within what an FP64 sum may lose, nothing within the
    reference's cut taken for far away, and no overflow."""
    exe = str(tmp_path / "oz_unit_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                           os.path.join(ROOT, "tests", "oz_unit_check.cc"), "-lm"])
    worst, far, over = subprocess.run([exe], capture_output=True, text=True, timeout=300,
                                      check=True).stdout.split()
    assert float(worst) <= 1.0
    assert int(far) == 0 and int(over) == 0


def test_exact_sums(tmp_path):
    """96-bit sums and their doubles (tests/oz_sum_check.cc) against 128-bit integers: the
    sums equal, the doubles within half a unit in the last place."""
    exe = str(tmp_path / "oz_sum_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                           os.path.join(ROOT, "tests", "oz_sum_check.cc"), "-lm"])
    wrong, worst = subprocess.run([exe], capture_output=True, text=True, timeout=300,
                                  check=True).stdout.split()
    assert int(wrong) == 0 and float(worst) <= 1.0
