"""csrc/quotient.h: the division of a bin's gradient columns by its weight from
one rounded reciprocal, bit for bit the REAL division (a product with the
reciprocal alone is not), zeros and infinities included; below 1e-30, where the
remainder is no longer exact, within the last place."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "radtrancode_b200", "csrc")
MAIN = r"""
#include <cstdio>
#include <cmath>
#include <cstring>
#include <limits>
#include <random>
#include "quotient.h"
int main() {
    std::mt19937_64 g(7);
    std::uniform_real_distribution<double> ub(0.0, 1.5), ue(-30.0, 30.0), us(-45.0, -30.0);
    long bad = 0, product = 0, small = 0;
    auto same = [](float x, float y) { return std::memcmp(&x, &y, 4) == 0; };
    const float inf = std::numeric_limits<float>::infinity();
    for (int i = 0; i < 4000000; ++i) {
        const float b = i < 64 ? std::ldexp(1.0f, -(i % 32)) : (float)(ub(g) + 0x1p-28), r = 1.0f / b;
        const float a = (float)((i & 1 ? -1.0 : 1.0) * std::pow(10.0, ue(g)));
        bad += !same(rtb::quotient(a, b, r), a / b);
        product += !same(a * r, a / b);
        const float s = (float)std::pow(10.0, us(g)), q = s / b;
        small += std::fabs((double)rtb::quotient(s, b, r) - q) > (double)std::nextafter(q, inf) - q;
        if (i < 64) {
            bad += !same(rtb::quotient(0.0f, b, r), 0.0f) || !same(rtb::quotient(inf, b, r), inf);
            bad += !same(rtb::quotient(-inf, b, r), -inf) || !std::isnan(rtb::quotient(std::nanf(""), b, r));
        }
    }
    std::printf("%ld %ld %ld\n", bad, product, small);
}
"""


def test_quotient_is_the_rounded_division(tmp_path):
    src, exe = tmp_path / "q.cpp", tmp_path / "q"
    src.write_text(MAIN)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    bad, product, small = map(int, subprocess.run([str(exe)], capture_output=True, check=True, text=True).stdout.split())
    assert bad == 0 and small == 0
    assert product > 0
