"""Fitting the Ewald polynomials is part of making every FP64 context: it must
stay well under the milliseconds that the rest takes (0.04 ms; a cosine per
product made it 1 ms)."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "md_b200", "csrc")
SOURCE = r"""
#include <chrono>
#include <cstdio>
#include "ewald_poly.hpp"
int main()
{
    double best = 1e9, s = 0;
    for (int rep = 0; rep < 7; ++rep) {
        const auto t = std::chrono::steady_clock::now();
        for (int i = 0; i < 50; ++i) s += mdf::make_ewald_poly(0.32 + 1e-4 * i, 10.0).p[3];
        best = std::fmin(best, std::chrono::duration<double>(std::chrono::steady_clock::now() - t).count() / 50);
    }
    printf("%g %g\n", best, s);
}
"""


def test_fit_takes_a_fraction_of_a_millisecond(tmp_path):
    src, exe = tmp_path / "t.cpp", str(tmp_path / "t")
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + CSRC, str(src), "-o", exe], check=True)
    best = float(subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()[0])
    assert best < 0.3e-3
