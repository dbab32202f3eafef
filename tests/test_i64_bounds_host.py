"""The error bounds that the integer arithmetic's header states, on the CPU."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "threepoint_gb300", "csrc")


@pytest.fixture(scope="module")
def report(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("i64b") / "check")
    r = subprocess.run(["g++", "-std=gnu++17", "-O2", "-w", "-I" + CSRC, os.path.join(HERE, "i64_bounds_check.cpp"), "-o",
                        exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return {k: float(v) for k, v in (line.split() for line in r.stdout.splitlines())}


# a sum: under two units of a result of 2^58 or more; sincos: two units of 2^-60
# turns and the products' units; a reciprocal: e^3 (2^-62 for starts 2 ulp and
# half a step of the argument off), the step's truncations, 2^-60 together
@pytest.mark.parametrize("name,bound", [("add", 2.0 ** -57), ("sincos", 2.0 ** -57.6), ("rcp", 2.0 ** -60)])
def test_bounds(report, name, bound):
    assert report[name] <= bound, (name, report[name])


def test_rounding_claims(report):
    assert report["alike"] > 100000
    assert report["unlike"] == 0
