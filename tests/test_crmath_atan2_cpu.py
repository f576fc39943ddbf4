"""atan2 of the correctly rounded functions where its float-float series are
longest (ratios of 1/16 to 1/8, and up to 1/8 either side of every table
point), on the host against atan2l rounded once: bit-identical, in the normal
build and in the one whose float-float stage meets every argument it covers."""
import os
import re
import subprocess

import pytest

from test_crmath_cpu import HERE, _nvcc


@pytest.mark.parametrize("build", [[], ["-DAVBD_CRMATH_TEST_FF"]], ids=["normal", "float-float"])
def test_atan2_bands_against_long_double(tmp_path, build):
    exe = str(tmp_path / "atan2_bands")
    src = os.path.join(HERE, "crmath", "atan2_bands.cu")
    r = subprocess.run([_nvcc(), "-std=c++17", "-O2", "-x", "cu", "-Xcompiler", "-ffp-contract=off"] + build +
                       [src, "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    out = subprocess.run([exe, "4000000"], capture_output=True, text=True, timeout=600)
    m = re.search(r"^atan2 (\d+) (\d+)$", out.stdout, re.M)
    assert m, out.stdout + out.stderr
    assert int(m.group(1)) == 7 * 4000000 + 2
    assert int(m.group(2)) == 0, out.stdout
