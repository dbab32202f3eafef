"""The integer-arithmetic FP64 forms over the whole range of rows that they
accept, on the CPU: a row whose exponents or logarithms do not fit the
fixed-point fields is refused (and keeps the FP64 instructions), every other
one agrees with long double."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "threepoint_gb300", "csrc")


@pytest.fixture(scope="module")
def report(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("i64d") / "check")
    r = subprocess.run(["g++", "-std=gnu++17", "-O2", "-w", "-I" + CSRC, "-I" + HERE,
                        os.path.join(HERE, "i64_domain_check.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return {k: int(v) for k, v in (line.split() for line in r.stdout.splitlines())}


@pytest.mark.parametrize("kind", [0, 1])
def test_every_accepted_bispectrum_row(report, kind):
    assert report[f"nodes{kind}"] > 40000
    assert report[f"over{kind}"] == 0


def test_every_accepted_plin_table(report):
    # the cells' polynomials hold where their coefficients fit: 1e-12
    assert report["tables"] > 150
    assert report["plin_err"] <= 1000


def test_every_accepted_power_spectrum_row(report):
    assert report["pells"] > 40000
    assert report["pell_over"] == 0
