"""The double-word split on the integer pipe (split_words, meshfreetrixi.jl_gb300/csrc/
mft_fpbits.h), compiled for the host: h = RN32(x) and l = (float)rem * 2^k equal the two
roundings RN32(x) and RN32(x - RN32(x)) bit for bit over every exponent it takes, random
significands, exact ties and carries, both signs; it declines outside its range."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

SRC = r"""
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>
#include "mft_fpbits.h"
static uint64_t rng = 0x9E3779B97F4A7C15ull;
static uint64_t next() { rng ^= rng >> 12; rng ^= rng << 25; rng ^= rng >> 27; return rng * 2685821657736338717ull; }
static uint32_t fb(float x) { uint32_t b; memcpy(&b, &x, 4); return b; }
int main() {
  const uint64_t half = 1ull << 28, tails[] = {0, 1, half - 1, half, half + 1, (1ull << 29) - 1};
  long bad = 0, took = 0;
  for (uint64_t e = 0; e < 2048; ++e)
    for (uint64_t s = 0; s < 2; ++s)
      for (int t = 0; t < 3000; ++t) {
        uint64_t m = next() & ((1ull << 52) - 1);
        if (t < 12) m = (m >> 30 << 30) | ((uint64_t)(t & 1) << 29) | tails[t / 2];
        else if (t < 18) m = ((1ull << 52) - (1ull << 29)) | tails[t - 12];
        const uint64_t b = (s << 63) | (e << 52) | m;
        double x;
        memcpy(&x, &b, 8);
        uint32_t h, scale;
        int32_t rem;
        const bool ok = mft::fpbits::split_words((uint32_t)(b >> 32), (uint32_t)b, &h, &rem, &scale);
        const bool inside = fabs(x) >= ldexp(1.0, -74) && fabs(x) < ldexp(1.0, 127);
        if (ok != inside) { ++bad; continue; }
        if (!ok) continue;
        ++took;
        float sc;
        memcpy(&sc, &scale, 4);
        const float hf = (float)x, lf = (float)(x - (double)hf), l = (float)rem * sc;
        if (h != fb(hf) || fb(l) != fb(lf)) ++bad;
      }
  printf("%ld bad of %ld\n", bad, took);
  return bad != 0 || took != 201l * 2 * 3000;
}
"""


def test_split_matches_two_roundings(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "split.cpp", tmp_path / "split"
    src.write_text(SRC)
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    str(ROOT / "meshfreetrixi.jl_gb300" / "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout
