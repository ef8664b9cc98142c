"""Grid-stride walks over up to 2^32 - 2 entries (csrc/index_walk.h), on the host: at the largest grid
and the steps of the user features' kernels a walk ends after its own entries."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_walks_near_the_end_of_32_bits(tmp_path):
    exe = tmp_path / "index_walk_check"
    src = os.path.join(HERE, "native", "index_walk_check.cpp")
    cc = subprocess.run(["g++", "-O2", "-std=c++17", "-o", str(exe), src], capture_output=True, text=True)
    assert cc.returncode == 0, cc.stderr
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr + res.stdout
    assert "bad 0" in res.stdout
