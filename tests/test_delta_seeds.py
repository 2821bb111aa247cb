"""CPU check of the seeds of the Wigner rows at beta = pi/2 for every pair of orders up to the last bandwidth, 512
(tests/cpp/delta_seeds.cpp), against the exact binomials: seed^2 4^a = binomial(2a, a - b).

Tolerance: a - b <= 511 products and quotients and a square root in double-double, each within 8 2^-104: 2^-92
relative, twice that of the square."""
import os
import shutil
import subprocess
from fractions import Fraction

from test_tables import CSRC, ROOT, _cuda_include


def test_seeds_are_exact_to_double_double(tmp_path):
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    exe = str(tmp_path / "delta_seeds")
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Wextra", "-Werror", "-I", CSRC, "-I", _cuda_include(),
                    os.path.join(ROOT, "tests", "cpp", "delta_seeds.cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)
    lines = iter(subprocess.run([exe], capture_output=True, text=True, timeout=300, check=True).stdout.splitlines())
    for a in range(512):
        binom = [1]   # binomial(2a, q), q = 0 .. a
        for q in range(a):
            binom.append(binom[-1] * (2 * a - q) // (q + 1))
        for b in range(a + 1):
            h, l = next(lines).split()
            assert "n" not in h + l, (a, b, h, l)   # inf or nan
            s = Fraction(float.fromhex(h)) + Fraction(float.fromhex(l))
            exact = binom[a - b]
            # |s^2 4^a - exact| <= 2^-91 exact, in integers
            v = s * s * 4 ** a
            assert abs(v.numerator - exact * v.denominator) << 91 <= exact * v.denominator, (a, b)
