"""CPU: the visible-slope root search returns the plain bisection's result bit for bit.

csrc/visible_slope.cuh skips the bisection midpoints whose comparison is decided by a root estimate and an
error radius. Built here for the host with the host's exp, erfc and log, it is compared with the CPU
restatement's sampler (every midpoint evaluated, CLARITAS/CLARITAS.py:1965-2038), which the same host
functions drive: the two must agree in every bit and every failure code, over both branches (ordinary and
tail), next to their border at -1, next to the change of formula at 5, and for draws at both ends of (0, 1).
"""
from __future__ import annotations

import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#include "claritas_oracle.c"
int plain_sample11(double si, double u1, double u2, double* x, double* y, int* f) {
    return o_sample11(si, u1, u2, x, y, f);
}
"""

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include "visible_slope.cuh"
extern "C" int plain_sample11(double, double, double, double*, double*, int*);
int main(int argc, char** argv) {
    std::mt19937_64 g(atoi(argv[1]));
    const int range = atoi(argv[2]);
    const long n = atol(argv[3]);
    std::uniform_real_distribution<double> U(0, 1);
    long bad = 0, searched = 0;
    for (long i = 0; i < n; ++i) {
        const double t = U(g);
        double si;
        switch (range) {
            case 0: si = 2 * t - 1; break;                      // ordinary, the cancelling end included
            case 1: si = 1 + 10 * t; break;
            case 2: si = exp(9.2 * t); break;                   // towards normal incidence
            case 3: si = -1 - 4.5 * t; break;                   // tail, below and across the formulas' border
            case 4: si = -1 - exp(12 * t) * 1e-2; break;        // tail, towards grazing
            case 5: si = -1 + (t - 0.5) * 1e-6; break;          // the branches' border
            default: si = -5 + (t - 0.5) * 0.2; break;
        }
        unsigned r = (unsigned)g();
        if (i % 17 == 0) r = g() % 64;
        if (i % 19 == 0) r = 0xffffffffu - g() % 64;
        const double u1 = ((double)r + 0.5) * 2.3283064365386962890625e-10;
        double x0 = 0, y0 = 0, x1 = 0;
        int f0 = 0, f1 = 0;
        const int a = plain_sample11(si, u1, 0.3, &x0, &y0, &f0), b = clr::o_visible_slope_x(si, u1, &x1, &f1);
        if (a != b || f0 != f1 || (a && memcmp(&x0, &x1, 8))) {
            if (bad++ < 5) printf("differs: slope %.17g u %.17g: %d %.17g (%d), %d %.17g (%d)\n", si, u1, a, x0, f0, b, x1, f1);
        }
        double root, radius;
        if (si < -1) clr::o_tail_root(-si, clr::o_tail_B(-si), log(u1), fmax(-1 / si, 1e-12), &root, &radius);
        else clr::o_visible_root(si, clr::o_visible_q(si), u1, &root, &radius);
        searched += radius == HUGE_VAL;
    }
    printf("%ld differ, %ld without an estimate of %ld\n", bad, searched, n);
    return bad != 0 || searched > n / 4;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("slope")
    (d / "shim.c").write_text(SHIM)
    (d / "main.cpp").write_text(MAIN)
    inc = ["-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "oracle"), "-ffp-contract=off", "-O2"]
    subprocess.run(["gcc", "-std=c11", "-fopenmp", *inc, "-c", str(d / "shim.c"), "-o", str(d / "shim.o")], check=True)
    subprocess.run(["g++", "-std=c++17", *inc, "-I", os.path.join(ROOT, "tardiis_and_claritas_gb300", "csrc"),
                    str(d / "main.cpp"), str(d / "shim.o"), "-fopenmp", "-lm", "-o", str(d / "m")], check=True)
    return str(d / "m")


@pytest.mark.parametrize("where", range(7))
def test_same_bits_as_the_plain_bisection(program, where):
    r = subprocess.run([program, str(100 + where), str(where), "150000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
