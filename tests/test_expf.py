"""clue_expf_normal (include/clue_expf.h), the exponential of runs whose exponents all
lie in [-80, 0], against clue_expf over that range: the same bits (no GPU)."""

import ctypes as C
import os
import subprocess

from tests.conftest import ROOT

SOURCE = r"""
#include "clue_expf.h"
/* Floats -x for the bit patterns first, first + step, ... up to -80: how many differ. */
long differing(uint32_t first, uint32_t step) {
  long bad = 0;
  for (uint64_t b = first; b <= 0xc2a00000u; b += step) {
    const uint32_t bits = (uint32_t)b;
    float x, y, z;
    memcpy(&x, &bits, 4);
    y = clue_expf(x);
    z = clue_expf_normal(x);
    bad += memcmp(&y, &z, 4) != 0;
  }
  return bad;
}
"""


def test_clue_expf_normal_has_the_bits_of_clue_expf(tmp_path):
    src, lib = tmp_path / "expf.c", tmp_path / "expf.so"
    src.write_text(SOURCE)
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "include"),
                    str(src), "-o", str(lib), "-lm"], check=True)
    differing = C.CDLL(str(lib)).differing
    differing.argtypes, differing.restype = [C.c_uint32, C.c_uint32], C.c_long
    assert differing(0x80000000, 4001) == 0      # -0 to -80, every 4,001st float
    assert differing(0xc2a00000 - 300000, 1) == 0  # every float near -80
    assert differing(0xbf317218 - 200000, 501) == 0  # around -ln 2 and on
