"""A call's stream (csrc/train_common.h) is waited for before it is destroyed, so that no copy from the
caller's memory outlives the call; on the host, with a CUDA runtime of the test's own."""
import os
import subprocess

from conftest import ROOT

HERE = os.path.dirname(os.path.abspath(__file__))


def test_stream_is_waited_for(tmp_path):
    from cumf_sgd_gb300 import build
    exe = tmp_path / "stream_check"
    src = os.path.join(HERE, "native", "stream_check.cpp")
    inc = [os.path.join(build._cuda_home(), "include"), os.path.join(ROOT, "include"),
           os.path.join(ROOT, "cumf_sgd_gb300", "csrc")]
    cc = subprocess.run(["g++", "-O2", "-std=c++17", *[f"-I{d}" for d in inc], "-o", str(exe), src], capture_output=True,
                        text=True)
    assert cc.returncode == 0, cc.stderr
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stdout + res.stderr
    assert "bad 0" in res.stdout
