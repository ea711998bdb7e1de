"""The reciprocal and the quotient of csrc/fp_recip.h, compiled here as plain C++, against IEEE
division: the reciprocal within one unit in the last place, the quotient too and equal in all but
one of a thousand cases (it is rounded once, from an exact remainder), without its correction within
two, infinities, NaN, zeros and numbers without a representable reciprocal included."""
import subprocess
from pathlib import Path

REPO = Path(__file__).resolve().parent.parent


def test_quotient_and_reciprocal_against_ieee(tmp_path):
    out = tmp_path / "fp_recip_check"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-Wall", "-Werror", "-I",
                        str(REPO / "tnl-mhfem_gb300" / "csrc"), str(REPO / "tests" / "fp_recip_check.cpp"), "-o", str(out)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(out)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:]
