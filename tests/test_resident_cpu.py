"""The per-device cache behind the cooperative launches, on the host: a device
never takes another's count, and concurrent first calls do not race."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_resident_counts_per_device_and_thread(tmp_path):
    exe = str(tmp_path / "resident")
    src = os.path.join(HERE, "host", "resident.cpp")
    base = ["g++", "-std=c++17", "-O1", "-pthread", src, "-o", exe]
    r = subprocess.run(base + ["-fsanitize=thread"], capture_output=True, text=True)
    if r.returncode != 0:  # no sanitiser here
        r = subprocess.run(base, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and "bad 0" in out.stdout, out.stdout + out.stderr
