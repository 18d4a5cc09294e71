"""divide.hpp (compiled here) against the division: random operands over the
exponents it takes and past them, the divisors that its argument leaves to a
comparison, quotients next to a tie, and values at its bounds."""
import os
import shutil
import subprocess

import pytest

from helpers import ROOT

SOURCE = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include "divide.hpp"
static uint64_t s = 88172645463325252ull;
static uint32_t rnd() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return (uint32_t)(s >> 11); }
static float number(uint32_t mantissa, int e) { return std::ldexp(1.f + (mantissa & 0x7fffff) * 0x1p-23f, e); }
static long bad = 0;
static void check(float a, float b)
{
	const float y = 1.f / b, w = a / b, g = bm4dof::divide_by(a, b, y);
	if (w != w && g != g) return;
	if (std::memcmp(&w, &g, 4) && bad++ < 5) std::printf("%a / %a: %a, not %a\n", a, b, g, w);
}
int main()
{
	for (long i = 0; i < 20000000; i++) {
		const float a = number(rnd(), (int)(rnd() % 200) - 130), b = number(rnd(), rnd() % 64);
		check(rnd() & 1 ? a : -a, b);
	}
	// the mantissas of b that the argument leaves open, and one more: every a
	for (uint32_t k = 1; k <= 3; k++)
		for (uint32_t m = 0; m < (1u << 23); m++) check(number(m, 0), number(0x800000 - k, 0));
	// quotients next to a tie: normal and subnormal ones
	for (long i = 0; i < 3000000; i++) {
		const float b = number(rnd(), 0), c = number(rnd(), 40 + rnd() % 20);
		const float a = (float)((double)b * (1.0 + (2 * (rnd() & 0x7fffff) + 1) * 0x1p-24));
		const float d = (float)((double)c * ((2 * (rnd() & 0xfffff) + 1) * 0x1p-150));
		check(a, b);
		check(std::nextafter(a, 0.f), b);
		check(std::nextafter(a, 9.f), b);
		check(d, c);
		check(std::nextafter(d, 0.f), c);
		check(std::nextafter(d, 9.f), c);
	}
	check(0x1.fd0d9ep-89f, 0x1.c9a8p+51f);
	check(0x1.9f1baep-96f, 0x1.5e24p+45f);
	check(0x1.eaed08p-91f, 0x1.ep+41f);
	for (float a : {0.f, 1e-45f, -1e-40f, NAN, 3e38f, -3e38f, 0x1p-100f, -0x1.fffffep-101f, 0x1p80f})
		for (float b : {1.f, 3.f, 0x1p20f, 0x1.000002p20f, 0x1.8p20f, 0x1p60f, 3e38f, INFINITY, NAN, 0.f, 0x1p-120f, -3.f}) check(a, b);
	return bad != 0;
}
"""


def test_divide_by_is_the_division(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "t.cpp").write_text(SOURCE)
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "bm4d-of_gb300", "csrc"),
                    str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
