"""The limiter's frozen branch (csrc/lim_coef.cuh, superbee's by comparisons),
built for the host, against the oracle's, which divides."""
import pathlib
import shutil
import subprocess

import pytest

HERE = pathlib.Path(__file__).resolve().parent


def test_branches_match_the_oracle(tmp_path, oracle_mod):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ is not available")
    lib = oracle_mod.LIB
    exe = tmp_path / "lim_coef_host"
    subprocess.check_call([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-o", str(exe),
                           str(HERE / "lim_coef_host.cpp"), str(lib), f"-Wl,-rpath,{lib.parent}"])
    out = subprocess.run([str(exe), "200000"], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout[-2000:]
    assert out.stdout.count("mismatches 0") == 42
