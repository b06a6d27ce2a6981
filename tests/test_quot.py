"""fh_quot (fh_quot.cuh): the quotient from a kept reciprocal has the bits of the
division, for operands from the smallest subnormal to the largest number, where the
remainders that correct it would leave the normal range, and for zeros, infinities
and NaN.  Host code of the header, on the CPU."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include "fh_quot.cuh"
#include <stdint.h>
#include <stdio.h>
#include <string.h>
static uint64_t st = 88172645463325252ull;
static uint32_t rnd() { st ^= st << 13; st ^= st >> 7; st ^= st << 17; return (uint32_t)(st >> 16); }
static float of(uint32_t b) { float f; memcpy(&f, &b, 4); return f; }
static uint32_t bits(float f) { uint32_t b; memcpy(&b, &f, 4); return b; }
static long bad = 0, n = 0;
static void one(float a, float b) {
  volatile float bv = b;
  const float r = 1.0f / bv, w = a / bv, q = fh_quot(a, b, r);
  ++n;
  if (isnan(w) ? !isnan(q) : bits(w) != bits(q))
    if (bad++ < 10) printf("%a / %a = %a, not %a\n", a, b, w, q);
}
int main() {
  const float sp[] = {0.f, -0.f, of(1), of(0x7fffff), of(0x800000), 1.f, -1.f, of(0x7f7fffff), INFINITY, -INFINITY, NAN};
  for (float a : sp)
    for (float b : sp) one(a, b);
  for (int i = 0; i < 2000000; ++i) one(of(rnd()), of(rnd()));                 // any operands
  for (int e = 0; e < 255; ++e)                                                // every size of a, b = 1 - al in (0, 2)
    for (int i = 0; i < 20000; ++i) {
      const uint32_t m = rnd();
      one(of((uint32_t)e << 23 | (m & 0x807fffffu)), of((rnd() % 60 + 68) << 23 | (rnd() & 0x7fffffu)));
      one(of((uint32_t)e << 23 | (m & 0x7fffffu)), of(0x3f800000u - (rnd() & 0xffffu)));  // mantissas of ones
    }
  printf("%ld of %ld differ\n", bad, n);
  return bad != 0;
}
"""


def test_quotient_has_the_divisions_bits(tmp_path):
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not available")
    src, exe = tmp_path / "quot.cu", tmp_path / "quot"
    src.write_text(SRC)
    r = subprocess.run(["nvcc", "-O2", "-std=c++17", "-Xcompiler", "-ffp-contract=off", "-I",
                        os.path.join(REPO, "theses_code_gb300", "csrc"), str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
