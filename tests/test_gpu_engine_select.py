"""The cubature's selection of the regions to split against a sort: more
candidates than its list, more regions than its staged keys, cuts below its
octave bins, ties, zeros, the region cap, errors that are not finite."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_selection(tmp_path):
    from threepoint_gb300 import build as B

    exe = str(tmp_path / "select")
    r = subprocess.run([B._nvcc(), *B.ARCH, "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "include"), "-I" + B.CSRC,
                        os.path.join(HERE, "engine_select_check.cu"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    bad = [line for line in r.stdout.splitlines() if not line.endswith(" ok")]
    assert r.returncode == 0 and not bad and len(r.stdout.splitlines()) > 100, (bad[:20], r.stderr)
