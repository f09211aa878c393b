"""ieee::twice_product and is_finite (ieee_bits.h) against the compiler's IEEE
double operations, on the host."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tissue-ablation-mc_gb300", "csrc")
DRIVER = r"""
#include "ieee_bits.h"
#include <cmath>
#include <cstdio>
#include <random>
using namespace tam::ieee;
static long bad = 0;
static void one(double g, double t)
{
    const volatile double p = g * t, g2 = 2.0 * g, want = g2 * t;
    if (std::isfinite(g) && !std::isfinite((double)g2)) return;  // the function takes a g whose double is finite
    const double got = twice_product(p, g, t);
    if (bits(got) != bits(want) && !(std::isnan(got) && std::isnan(want)) && bad++ < 5) std::printf("%a %a: %a %a\n", g, t, got, (double)want);
    if (is_finite(t) != (bool)std::isfinite(t)) ++bad;
}
int main()
{
    const double sp[] = {0.0, -0.0, 1.0, 5e-324, 2.2250738585072014e-308, 1.7976931348623157e308, INFINITY, NAN, 300.0, 1e4};
    for (double a : sp) for (double b : sp) { one(a, b); one(-a, b); }
    std::mt19937_64 r(7);
    for (int n = 0; n < 2000000; ++n) {
        const uint64_t a = r(), b = r();
        // results around the subnormals and the overflow, ordinary ones, any
        const uint64_t ea = n % 4 == 0 ? 2 + a % 60 : (n % 4 == 1 ? 2040 - a % 30 : (n % 4 == 2 ? 1000 + a % 40 : a % 2048));
        const uint64_t eb = n % 4 == 0 ? 960 + b % 64 : (n % 4 == 1 ? 1010 + b % 40 : (n % 4 == 2 ? 1000 + b % 40 : b % 2048));
        one(from_bits((a & 0x800FFFFFFFFFFFFFull) | ea << 52), from_bits((b & 0x800FFFFFFFFFFFFFull) | eb << 52));
    }
    std::printf("mismatches %ld\n", bad);
    return bad != 0;
}
"""


def test_twice_product(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(DRIVER)
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "mismatches 0" in r.stdout, r.stdout
