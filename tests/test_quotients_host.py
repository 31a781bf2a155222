"""The quotients that carry a proof instead of a certificate (quot_rn and
div_rn_3 of csrc/exact_div.cuh), built for the host and compared with IEEE
division bit for bit: general operands, divisors just below a power of two and
within a few ulps of one, short mantissas (exact quotients) and tails down to
the subnormals.  Refused operands are the callers' to divide, and the sign of
a zero quotient is not kept."""
import pathlib
import shutil
import subprocess

import pytest

HERE = pathlib.Path(__file__).resolve().parent


def test_quotients_are_ieee(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ is not available")
    exe = tmp_path / "quotients_host"
    subprocess.check_call([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-o", str(exe),
                           str(HERE / "quotients_host.cpp")])
    out = subprocess.run([str(exe), "400000", "3"], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout[-2000:]
    refused = {tuple(f[:2]): int(f[7]) / int(f[3]) for f in (line.split() for line in out.stdout.splitlines())}
    assert len(refused) == 10
    # nearly every ordinary operand is taken (10 in 420 of the limiter's divisors lie outside its range)
    assert refused["quot_rn", "any"] < 0.06 and refused["div_rn_3", "any"] < 1.0e-4
