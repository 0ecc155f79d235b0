"""The planner's two passes are compiled apart and have to find the same units,
so the box tests they share must round alike whatever the compiler contracts:
one source compiled with and without contraction into fused operations, every
result's bits the same."""
import os
import platform
import subprocess

import pytest

import build_engine

HERE = os.path.dirname(os.path.abspath(__file__))


def test_the_same_bits_with_and_without_contraction(tmp_path):
    if platform.machine() == "x86_64":  # (fused operations are not in its baseline)
        if " fma " not in open("/proc/cpuinfo").read():
            pytest.skip("no fused operations to contract into")
        fused = ["-mfma"]
    else:
        fused = []
    out = []
    for contract in ("off", "fast"):
        exe = str(tmp_path / contract)
        subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=" + contract] + fused +
                       ["-I" + os.path.join(build_engine.CUDA, "include"), os.path.join(HERE, "plan_bounds_check.cc"), "-o", exe],
                       check=True)
        out.append(subprocess.run([exe], capture_output=True, text=True, check=True).stdout)
    assert out[0] == out[1] and len(out[0].strip()) == 16
