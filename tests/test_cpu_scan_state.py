"""A scan state after an allocation that failed (gahhg_b200/csrc/scan_state.cpp,
built for the host with an allocator that fails when told to): the next call
makes a whole one, with a cleared counter and cleared status words, and
nothing is lost."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("scan") / "libscan_probe.so")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic",
                           "-I", os.path.join(os.path.dirname(HERE), "include"), "-I", "/usr/local/cuda/include",
                           "-o", out, os.path.join(HERE, "native", "scan_state_probe.cpp")])
    return ctypes.CDLL(out)


@pytest.mark.parametrize("n1,n2", [(1, 1), (100, 10_000_000), (1 << 22, 1 << 20), (2048, 4097)])
def test_after_a_failure(probe, n1, n2):
    what = ctypes.c_int()
    failures = []
    for fail in range(0, 9):  # 0: none
        r = probe.reserve_with_failure(ctypes.c_long(n1), ctypes.c_long(n2), fail, ctypes.byref(what))
        assert r >= 0, (fail, what.value)
        failures.append(r)
    assert failures[0] == 0 and failures[1:5] == [1, 1, 1, 1]
