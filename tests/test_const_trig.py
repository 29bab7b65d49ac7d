"""The literal coefficients of the odd register DFTs
(agdeblend_b200/csrc/const_trig.hpp), compiled for the host: against 50-digit
values, no further off (root mean square) than the C library's functions of
the rounded angle 2 pi m / n, from which the tables of the other lengths are
made."""
import math
import os
import shutil
import subprocess
from decimal import Decimal, getcontext

import pytest

from conftest import ROOT

LENGTHS = (3, 5, 7, 9, 11, 13, 17, 19, 23, 25, 27)
SOURCE = """
#include <cstdio>
#include <initializer_list>
#include "const_trig.hpp"
int main() {
  for (int n : {%s})
    for (int m = 0; m <= n; ++m)
      std::printf("%%d %%d %%a %%a\\n", n, m, agd::const_cos(m, n), agd::const_sin(m, n));
}
""" % ", ".join(map(str, LENGTHS))


def _exact(m, n):
    """cos and sin of 2 pi m / n by their series."""
    getcontext().prec = 50
    x = 2 * Decimal("3.14159265358979323846264338327950288419716939937510582") * m / n
    c = s = Decimal(0)
    term = Decimal(1)
    for k in range(80):
        if k % 2 == 0:
            c += term if k % 4 == 0 else -term
        else:
            s += term if k % 4 == 1 else -term
        term *= x / (k + 1)
    return c, s


def test_literal_coefficients(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    src, exe = tmp_path / "trig.cpp", tmp_path / "trig"
    src.write_text(SOURCE)
    subprocess.run([cxx, "-std=c++17", "-I", os.path.join(ROOT, "agdeblend_b200", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    own, lib = [0.0, 0.0], [0.0, 0.0]
    for line in subprocess.run([str(exe)], check=True, capture_output=True,
                               text=True).stdout.splitlines():
        n, m, c, s = line.split()
        n, m = int(n), int(m)
        angle = 2.0 * math.pi * m / n
        for i, (exact, mine, theirs) in enumerate(zip(
                _exact(m, n), (float.fromhex(c), float.fromhex(s)),
                (math.cos(angle), math.sin(angle)))):
            assert abs(Decimal(mine) - exact) <= Decimal(4e-16)
            own[i] += float(Decimal(mine) - exact) ** 2
            lib[i] += float(Decimal(theirs) - exact) ** 2
    assert own[0] <= lib[0] and own[1] <= lib[1]
