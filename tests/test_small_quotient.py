"""The quotient the fused adjoint splits its work items with (csrc/sg_divide.h): r / k by one
multiplication, compiled for the host and compared with the division for every divisor a tile
can have (its axis-0 control points, 1 to 512) and every item of up to 32 channels, and at the
ends of the range that the header states."""
import os
import subprocess

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include "sg_divide.h"
static int check(uint32_t r, uint32_t k) {
    const uint32_t q = sg::small_quotient(r, sg::small_reciprocal(k));
    if (q == r / k) return 0;
    std::printf("%u / %u: %u, not %u\n", r, k, q, r / k);
    return 1;
}
int main() {
    int bad = 0;
    for (uint32_t k = 1; k <= 512 && bad < 10; ++k)
        for (uint32_t r = 0; r < 32 * k; ++r) bad += check(r, k);
    for (uint32_t k = 1; k <= 65535 && bad < 10; ++k)
        for (uint32_t q = 0; q < 65535 / k; q += 1 + q / 7)
            bad += check(q * k, k) + check(q * k + k - 1, k);
    return bad != 0;
}
"""


def test_quotient_is_the_division(tmp_path):
    src, exe = tmp_path / "quotient.cpp", tmp_path / "quotient"
    src.write_text(PROGRAM)
    csrc = os.path.join(ROOT, "splinegrids.jl_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", csrc, "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
