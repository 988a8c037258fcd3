"""The helium right-hand side's division by three (csrc/psg_div3.h) against
the C compiler's, bit for bit: random doubles of every exponent, the numbers
beside multiples of three, subnormals, zeros, infinities and NaN."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <stdint.h>
#include <stdio.h>
#include <string.h>
#include "psg_div3.h"
static uint64_t bits(double x) { uint64_t u; memcpy(&u, &x, 8); return u; }
static double dbl(uint64_t u) { double x; memcpy(&x, &u, 8); return x; }
static int bad = 0;
static void one(double x) {
	volatile double three = 3.0;
	const double want = x / three, got = psg_div3(x);
	if ((want != want) ? !(got != got) : bits(want) != bits(got)) {
		if (bad++ < 10) printf("%a: %a, not %a\n", x, got, want);
	}
}
int main(void) {
	uint64_t s = 1;
	for (int e = 0; e < 2048; e++)
		for (int i = 0; i < 3000; i++) {
			s = s * 6364136223846793005ull + 1442695040888963407ull;
			const uint64_t m = (s >> 12) ^ (s << 20);
			const uint64_t u = (uint64_t)e << 52 | (m & 0xfffffffffffffull);
			one(dbl(u));
			one(dbl(u | 1ull << 63));
			one(dbl(m & 0x3ffffffffull));      /* the quotient's high word around zero */
			const double q = dbl((uint64_t)(e > 2 ? e - 2 : 0) << 52 | (m & 0xfffffffffffffull));
			for (int k = -2; k <= 2; k++) one(dbl(bits(3.0 * q) + k));
		}
	for (uint64_t u = 0; u < 100000; u++) {      /* zeros and the smallest subnormals */
		one(dbl(u));
		one(dbl(u | 1ull << 63));
	}
	one(dbl(0x7ff0000000000000ull));
	one(dbl(0xfff0000000000000ull));
	one(dbl(0x7fefffffffffffffull));
	return bad != 0;
}
"""


def test_div3_is_the_division(tmp_path):
    cc = shutil.which("gcc") or shutil.which("cc")
    if cc is None:
        pytest.skip("no C compiler")
    src, exe = tmp_path / "div3.c", tmp_path / "div3"
    src.write_text(SRC)
    subprocess.run([cc, "-std=gnu11", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "psphray_b200", "csrc"),
                    str(src), "-o", str(exe), "-lm"], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
