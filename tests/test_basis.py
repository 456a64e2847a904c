"""The transform's basis as this host's math library gives it: the symmetries
that the decoder's paired sums rely on hold to the last bit, and the check that
every context makes sees a change of one unit in the last place anywhere."""

import shutil
import subprocess

import pytest

from rivet_prores_b200.build import CSRC

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include "codec_tables.h"
int main() {
    float T[64];
    prores::dct_basis(T);
    int missed = 0;
    for (int i = 0; i < 64; i++) {
        const float t = T[i];
        T[i] = std::nextafter(t, 1.0f);
        missed += prores::dct_basis_mirrors(T);
        T[i] = t;
    }
    std::printf("%d %d\n", (int)prores::dct_basis_mirrors(T), missed);
}
"""


def test_the_basis_has_the_cosines_symmetries(tmp_path):
    compiler = shutil.which("g++") or pytest.skip("no g++")
    (tmp_path / "basis.cpp").write_text(PROGRAM)
    subprocess.run([compiler, "-std=c++17", "-I", CSRC, str(tmp_path / "basis.cpp"), "-o", str(tmp_path / "basis")],
                   check=True)
    assert subprocess.run([str(tmp_path / "basis")], capture_output=True, text=True).stdout == "1 0\n"
