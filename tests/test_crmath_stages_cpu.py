"""The float-float stage of the correctly rounded functions and the
reciprocal-based divisions of the 6x6 solve, on the host (no GPU).

The float-float stage: the sweep of test_crmath_cpu.py in a build whose float
stage rejects everything, so that every argument the pairs cover meets them
first; bit-identical to the long-double references.  The divisions: quotients
bit-identical to the IEEE ones over random operands of the stated range (a
quotient the range test sends back is not compared, and few are), solutions
bit-identical to the dividing solve, breakdowns included."""
import os
import re
import subprocess

import pytest

from test_crmath_cpu import HERE, _nvcc, _sweep


def test_float_float_stage_against_long_double(tmp_path):
    res, log = _sweep(tmp_path, ["-DAVBD_CRMATH_TEST_FF"], [40961, 100000])
    for name, (n, bad) in res.items():
        assert n > 100000, (name, n)
        assert bad == 0, log


def test_divisions_by_reciprocal_equal_ieee(tmp_path):
    exe = str(tmp_path / "div_sweep")
    src = os.path.join(HERE, "crmath", "div_sweep.cu")
    r = subprocess.run([_nvcc(), "-std=c++17", "-O2", "-x", "cu", "-Xcompiler", "-ffp-contract=off", src, "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    out = subprocess.run([exe, "20000000"], capture_output=True, text=True, timeout=600)
    got = {m.group(1): tuple(int(m.group(k)) for k in (2, 3, 4))
           for m in re.finditer(r"^(\w+) (\d+) (\d+) (\d+)$", out.stdout, re.M)}
    assert set(got) == {"div_by", "solve"}, out.stdout + out.stderr
    n, back, bad = got["div_by"]
    assert bad == 0 and back < n // 4, out.stdout
    n, fail, bad = got["solve"]
    assert bad == 0 and fail > 0, out.stdout
