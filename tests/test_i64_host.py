"""The integer-arithmetic FP64 forms (tp_i64.cuh, tp_bispec64.cuh) on the CPU:
every function against long double at random arguments and at the edges of its
tables, and a bispectrum node against the literal formula in long double."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "threepoint_gb300", "csrc")


@pytest.fixture(scope="module")
def report(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("i64") / "i64_check")
    r = subprocess.run(["g++", "-std=gnu++17", "-O2", "-w", "-I" + CSRC, os.path.join(HERE, "i64_check.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return {k: float(v) for k, v in (line.split() for line in r.stdout.splitlines())}


# (name, bound): relative errors except log2 and the fixed-point conversions
# (absolute). sincos: the argument's Q60 rounding and its product with 1/(2 pi),
# two units of 2^-60 turns = 2^-57.6 radian; exp2: truncated products of 2^-64 and the sixth-order term
# (2^-8 ln2)^6/720 = 2^-60.6, together below 2^-57.5; log2: (2^-8)^7/(7 ln2) =
# 2^-58.3 and the Q31 coefficients, below 2^-57; products lose three units of a
# 62-bit result; a sum keeps at least 58 bits.
@pytest.mark.parametrize("name,bound", [("sincos", 2.0 ** -57.5), ("exp2", 2.0 ** -57.5), ("log2", 2.0 ** -57), ("mul", 2.0 ** -60),
                                        ("add", 2.0 ** -55), ("rcp", 2.0 ** -60), ("to_double", 2.0 ** -52.9),
                                        ("from_double", 0.0), ("fix", 2.0 ** -52.9)])
def test_functions(report, name, bound):
    assert report[name] <= bound, (name, report[name])


def test_plin_table_is_no_less_accurate_than_the_double_formula(report):
    assert report["plin_int_max"] <= report["plin_dbl_max"]
    assert report["plin_int_rms"] <= report["plin_dbl_rms"]


def test_node_is_no_less_accurate_than_the_double_formula(report):
    assert report["nodes"] > 15000
    for q in ("median", "p99", "max"):
        assert report["node_int_" + q] <= report["node_dbl_" + q], q


def test_power_spectrum_term_is_no_less_accurate_than_the_double_formula(report):
    assert report["pells"] > 15000
    for q in ("median", "p99", "max"):
        assert report["pell_int_" + q] <= report["pell_dbl_" + q], q
