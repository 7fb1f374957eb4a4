"""The search kernels' grid barrier, on the host: a search of more levels than
32 bits of arrivals count (15 million, a path) still waits at every barrier."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_barrier_counts_past_32_bits(tmp_path):
    out = os.path.join(str(tmp_path), "barrier_check")
    subprocess.run(["g++", "-std=c++17", "-O1",
                    os.path.join(ROOT, "tests", "cpp", "barrier_check.cpp"), "-o", out], check=True)
    r = subprocess.run([out], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "barrier ok" in r.stdout, r.stdout
