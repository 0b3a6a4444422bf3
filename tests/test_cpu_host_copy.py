"""The copy team that stages host buffers: slices done once, in their limits."""
import os
import subprocess

import pytest


HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("copy") / "probe")
    csrc = os.path.join(ROOT, "gahhg_b200", "csrc")
    subprocess.check_call(["nvcc", "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                           "-I", csrc, "-I", os.path.join(ROOT, "include"),
                           os.path.join(HERE, "native", "copy_team_probe.cpp"), os.path.join(csrc, "host_copy.cpp"),
                           "-o", exe, "-lpthread"])
    return exe


@pytest.mark.parametrize("workers", [1, 3, 8])
def test_jobs(probe, workers):
    r = subprocess.run([probe, str(workers), "400"], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "0", r.stdout + r.stderr
