"""Parts of the CUDA sources that the host can check by itself.

The search kernels' grid barrier: a search of more levels than 32 bits of
arrivals count (15 million, a path) still waits at every barrier.  The words
that every traversal uses: an allocation that fails leaves none of them.  The
chunks of triangles at listed vertices: their sum fits its type.  The PageRank
kernels' inline loads: volatile, or nothing keeps them after the wait for the
kernel whose results they read."""
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("name,says", [("barrier_check", "barrier ok"),
                                       ("travwords_check", "words ok"),
                                       ("tcvrule_check", "rule ok")])
def test_part(tmp_path, name, says):
    out = os.path.join(str(tmp_path), name)
    subprocess.run(["g++", "-std=c++17", "-O1", os.path.join(ROOT, "tests", "cpp", name + ".cpp"),
                    "-o", out], check=True)
    r = subprocess.run([out], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and says in r.stdout, (r.returncode, r.stdout)


def test_pagerank_loads_are_ordered():
    src = open(os.path.join(ROOT, "sstgraph_gb300", "csrc", "prfixed.cuh")).read()
    loads = re.findall(r"asm( volatile)?\s*\(\s*\"(ld\.[^ ]*)", src)
    assert len(loads) >= 2
    assert all(v for v, _ in loads), loads
    # contributions: written by the kernel before
    assert [op for _, op in loads if "evict_last" in op] == ["ld.global.L1::evict_last.b64"]
