"""Exponent arithmetic of the digit products (fixed.cuh) on the host: no signed overflow
(under the undefined-behaviour sanitizer) and the right exponent over the whole range of
exponent fields that the digits take."""
import subprocess

from macaw_gb300 import build

SOURCE = r"""
#include <math.h>
#include <stdio.h>
#include <string.h>
#include "fixed.cuh"
int main() {
  // operands cut with the fields ea and eb are below 2^(ea - 1022), 2^(eb - 1022); the
  // integer v stands for v 2^(ea - 1022 + eb - 1022 - 12 - bits)
  for (unsigned bits = 43; bits <= 47; ++bits)
    for (unsigned ea = FX_EMIN; ea <= FX_EMAX; ea += 5)
      for (unsigned eb = FX_EMIN; eb <= FX_EMAX; eb += 7) {
        const double v = ldexp(3.0, 50), want = ldexp(v, (int)(ea + eb - 2044 - 12) - (int)bits);
        unsigned long long w;
        memcpy(&w, &v, 8);
        const unsigned es = fx_exp(ea << 20, eb << 20, bits);
        w = ((unsigned long long)fx_add_exp((unsigned)(w >> 32), es) << 32) | (unsigned)w;
        double got;
        memcpy(&got, &w, 8);
        if (got != want) return printf("%u %u %u\n", ea, eb, bits), 1;
        if (fx_add_exp(0u, es) != 0u) return 2;
      }
  return 0;
}
"""


def test_exponent_words(tmp_path):
    src, exe = tmp_path / "exponents.cu", tmp_path / "exponents"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-I", build.CSRC, "-Xcompiler",
                    "-fsanitize=undefined,-fno-sanitize-recover=all", str(src), "-o", str(exe), "-lubsan"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
