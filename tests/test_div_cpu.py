"""Division by a tabulated reciprocal (kf_div.hpp) against the division, bit for
bit, and NaN where the kernel is to divide, compiled for the host: the same fma
steps as on the device."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kielflow_b200", "csrc")

PROGRAM = r"""
#include "kf_div.hpp"
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
using namespace kf;
static long bad = 0, n = 0;
static void check(double num, double den) {
    const double q = div_by(num, den, div_reciprocal(den)), w = num / den;
    ++n;
    bool ok;
    if (!(den >= 0x1p-60 && den <= 0x1p60) || !(std::fabs(num) <= 1e308 && std::fabs(w) <= 1e308))
        ok = q != q || q == w;  // the caller divides
    else if (std::fabs(w) < 0x1p-900)
        ok = std::fabs(q - w) <= 0x1p-950;
    else
        ok = !std::memcmp(&q, &w, sizeof q);
    if (!ok && ++bad < 10) std::printf("%a / %a: %a, not %a\n", num, den, q, w);
}
int main() {
    std::mt19937_64 g(7);
    std::uniform_real_distribution<double> u(1., 2.);
    auto any = [&](int lo, int hi) { return (g() & 1 ? -1. : 1.) * std::ldexp(u(g), lo + (int)(g() % (unsigned)(hi - lo + 1))); };
    auto den = [&](int k) {  // cell widths squared, the table's whole range, mantissas near its ends
        if (k == 0) { const double h = 25.132741228718345 / (double)(2 + g() % 255); return h * (h + h * u(g)); }
        if (k == 1) return std::fabs(any(-60, 59));
        if (k == 2) return std::ldexp(2. - std::ldexp((double)(1 + g() % 9), -52), (int)(g() % 20) - 10);
        return std::ldexp(1. + std::ldexp((double)(g() % 9), -52), (int)(g() % 20) - 10);
    };
    for (long i = 0; i < 4000000; ++i) {
        const double d = den(i & 3);
        check(any(-30, 10), d);                             // potentials
        check(any(-1040, 1010), d);                         // everything
        check(d * std::ldexp(u(g), 3) , d);
        check(std::nextafter(d * (double)(g() % 1000), 9e9), d);  // next to exact quotients
    }
    const double inf = std::numeric_limits<double>::infinity(), tiny = std::numeric_limits<double>::denorm_min();
    for (double x : {0., -0., inf, -inf, std::nan(""), tiny, -tiny, 1e-300, 1e-320, 1e300, 1.7e308, -1.7e308})
        for (double d : {1., 3., 0.1, 1e-18, 1e18, 1e-30, 1e30, 1e-310, 0x1p-60, 0x1p60}) check(x, d);
    std::printf("%ld of %ld differ\n", bad, n);
    return bad != 0;
}
"""


def test_div_by_is_the_division(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    (tmp_path / "d.cpp").write_text(PROGRAM)
    exe = str(tmp_path / "d")
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I" + CSRC, "-o", exe, str(tmp_path / "d.cpp")],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
