"""The replica engine divides the bead updates by kept divisors through their
reciprocals (rmpcdmd_b200/csrc/quotient.cuh): the quotients are the division's, bit for
bit, over random, extreme and special operands."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_quotients_are_those_of_the_division(tmp_path):
    exe = tmp_path / "quotient"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "rmpcdmd_b200" / "csrc"),
                    str(ROOT / "tests" / "c" / "quotient.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert int(r.stdout) > 4000000
