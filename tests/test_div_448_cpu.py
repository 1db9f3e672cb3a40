"""CPU: the quotient x / 448 of the fp8 scales (csrc/det_math.h), compiled here, against the host's IEEE division: every
significand of a binade, and a sample of every binade from 2^-93 to the largest, whose steps are the same but for the exponent."""
import ctypes as ct
import subprocess

from conftest import PKG_DIR

SOURCE = r"""
#include "det_math.h"
#include <stdio.h>
static uint32_t bits_of(float f) { uint32_t b; memcpy(&b, &f, 4); return b; }
static long compare(int exponent, uint32_t step) {
  long wrong = 0;
  for (uint32_t m = 0; m < (1u << 23); m += step) {
    const uint32_t b = ((uint32_t)(exponent + 127) << 23) | m;
    float x;
    memcpy(&x, &b, 4);
    volatile float want = x / 448.0f;
    wrong += bits_of(dm_div_448(x)) != bits_of(want);
  }
  return wrong;
}
extern "C" long wrong_quotients() {
  long wrong = compare(0, 1) + compare(127, 1);
  for (int e = -93; e <= 127; ++e) wrong += compare(e, 127);
  return wrong + (dm_div_448(0.0f) != 0.0f) + (dm_div_448(INFINITY) != INFINITY);
}
"""


def test_every_significand_gives_the_rounded_quotient(tmp_path):
    (tmp_path / "q.cpp").write_text(SOURCE)
    lib = tmp_path / "q.so"
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", str(PKG_DIR / "csrc"), str(tmp_path / "q.cpp"),
                    "-o", str(lib)], check=True)
    f = ct.CDLL(str(lib)).wrong_quotients
    f.restype = ct.c_long
    assert f() == 0
